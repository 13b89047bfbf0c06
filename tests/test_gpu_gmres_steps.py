"""GMRES at the edges of its kernels' tiles (fp_gmres.cu): rows and columns that do
not fill a tile, more basis vectors than one staged group and than the storage
hint, against the oracle's LAPACK solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 16 unknowns (one partial tile of rows, column ranges of one); 128 and 132; 516
# (steps past 128 staged vectors); 4,140 (past 4,096 staged rows)
@pytest.mark.parametrize("nc,ns", [(4, 4), (16, 8), (22, 6), (86, 6), (46, 90)])
@pytest.mark.parametrize("memory", [3, 50])
def test_gmres_tile_edges(fp, O, nc, ns, memory):
    w = fp.meshes.swept_wing("0012", nc, ns)
    body = fp.RigidWakeBody(w)
    normals = fp.calc_normals(body)
    cps = fp.calc_controlpoints(body, normals)
    a = np.deg2rad(4.2)
    V = np.array([np.cos(a), 0.0, np.sin(a)])
    D = np.tile(V, (w.nsheddings, 1))
    U = np.tile(V, (w.npanels, 1))
    c = fp._capi.Context(0)
    try:
        c.set_geometry(w.nodes, w.panel_offsets, w.panel_nodes, cps, normals)
        c.set_wake(w.shedding, D, D)
        opts = fp._capi.make_opts("gmres", "fp64", gmres_memory=memory, gmres_atol=1e-10, gmres_rtol=1e-10)
        x, st = c.solve_body(fp._capi.FP_ELEMENT_VORTEXRING, np.stack([U, -2 * U]), opts=opts)
    finally:
        c.close()
    Gr = O.assemble_vortexring(w, cps, normals, D, D)
    rhs = O.rhs_noflowthrough(U, normals)
    # the stopping rule itself: ||b - A x|| <= atol + rtol ||b||, of the estimate the process stops by
    tol = 2 * (1e-10 + 1e-10 * np.linalg.norm(rhs))
    assert np.linalg.norm(Gr @ x[0] - rhs) < tol
    assert np.linalg.norm(Gr @ x[1] + 2 * rhs) < 2 * tol
    assert st.gmres_iters > 0
