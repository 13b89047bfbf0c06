"""Two and four right-hand sides on either side of the sizes at which lu_solve
changes its sweeps, against the oracle's LAPACK solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 1,020 and 1,032: 2 right-hand sides by one sweep or two; 4 take the group's sweep in
# FP64 and k_trsm in FP32; 132: two blocks of 64 rows and 4
@pytest.mark.parametrize("nc,ns", [(22, 6), (34, 30), (86, 12)])
@pytest.mark.parametrize("k", [2, 4])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sweeps_by_size(fp, O, nc, ns, k, precision):
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
    lu = O.lu_factor(O.assemble_vortexring(w, cps, normals, D, D))
    xr = np.stack([O.lu_solve(lu, O.rhs_noflowthrough(u, normals)) for u in U])
    # as the tests of the sweeps over several right-hand sides
    assert np.linalg.norm(x - xr) / np.linalg.norm(xr) < 1e-10
