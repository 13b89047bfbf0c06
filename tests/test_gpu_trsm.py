"""Several right-hand sides at once (fp_trsm.cu): every group size and its edges,
partial blocks, against the oracle's LAPACK solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one partial 128-row block; one whole; two blocks, the second of 4 rows; three, the
# last of 16; nine
@pytest.mark.parametrize("nc,ns", [(10, 6), (16, 8), (22, 6), (34, 8), (40, 28)])
@pytest.mark.parametrize("k", [2, 3, 5, 8, 9, 17, 24, 25, 33, 40])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_right_hand_sides(fp, O, nc, ns, k, precision):
    w = fp.meshes.swept_wing("0012", nc, ns)
    body = fp.RigidWakeBody(w)
    normals = fp.calc_normals(body)
    cps = fp.calc_controlpoints(body, normals)
    a = np.deg2rad(4.2)
    D = np.tile([np.cos(a), 0.0, np.sin(a)], (w.nsheddings, 1))
    U = np.random.default_rng(k).standard_normal((k, w.npanels, 3))
    c = fp._capi.Context(0)
    try:
        c.set_geometry(w.nodes, w.panel_offsets, w.panel_nodes, cps, normals)
        c.set_wake(w.shedding, D, D)
        x, st = c.solve_body(fp._capi.FP_ELEMENT_VORTEXRING, U, opts=fp._capi.make_opts("ludiv", precision))
    finally:
        c.close()
    Gr = O.assemble_vortexring(w, cps, normals, D, D)
    lu = O.lu_factor(Gr)
    xr = np.stack([O.lu_solve(lu, O.rhs_noflowthrough(u, normals)) for u in U])
    assert np.abs(x - xr).max() / np.abs(xr).max() < 1e-10
    assert np.linalg.norm(x - xr) / np.linalg.norm(xr) < 1e-10
