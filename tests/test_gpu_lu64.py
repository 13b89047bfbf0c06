"""The FP64 factorisation (fp_lu64.cu) at the edges of its blocks and panels,
against the oracle's LAPACK solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one partial block; one whole; a block and 4 columns; a panel less 4, whole, and
# with 4 columns in the next; two panels and 4; a last panel of 3 blocks and a part
@pytest.mark.parametrize("nc,ns", [(10, 6), (8, 8), (34, 2), (42, 6), (16, 16), (26, 10), (86, 6), (18, 26)])
@pytest.mark.parametrize("shuffle", [False, True])
def test_fp64_lu_block_edges(fp, O, nc, ns, shuffle):
    """With the rows of the AIC shuffled the pivots come from all over each
    block (and the factorisation may be uncertified: then the solve refines)."""
    w = fp.meshes.swept_wing("0012", nc, ns)
    if shuffle:   # new panel i = old panel perm[i], within blocks of 64
        rng = np.random.default_rng(nc)
        perm = np.concatenate([k + rng.permutation(min(64, w.npanels - k)) for k in range(0, w.npanels, 64)])
        cells = [w.panel(i) for i in perm]
        w.panel_nodes = np.concatenate(cells).astype(np.int32)
        inv = np.argsort(perm)
        w.shedding = w.shedding.copy()
        w.shedding[:, 0], w.shedding[:, 3] = inv[w.shedding[:, 0]], inv[w.shedding[:, 3]]
    body = fp.RigidWakeBody(w)
    normals = fp.calc_normals(body)
    cps = fp.calc_controlpoints(body, normals)
    if shuffle:   # and the control points in another order: rows no longer on their diagonal
        rows = np.concatenate([k + rng.permutation(min(64, w.npanels - k)) for k in range(0, w.npanels, 64)])
        cps, normals = cps[rows], normals[rows]
    a = np.deg2rad(4.2)
    V = np.array([np.cos(a), 0.0, np.sin(a)])
    D = np.tile(V, (w.nsheddings, 1))
    U = np.tile(V, (w.npanels, 1))
    c = fp._capi.Context(0)
    try:
        c.set_geometry(w.nodes, w.panel_offsets, w.panel_nodes, cps, normals)
        c.set_wake(w.shedding, D, D)
        x, st = c.solve_body(fp._capi.FP_ELEMENT_VORTEXRING, U, opts=fp._capi.make_opts("ludiv", "fp64"))
    finally:
        c.close()
    Gr = O.assemble_vortexring(w, cps, normals, D, D)
    rhs = O.rhs_noflowthrough(U, normals)
    xr = O.solve_ludiv(Gr, rhs)
    assert np.linalg.norm(x - xr) / np.linalg.norm(xr) < 1e-10
    if st.gepp_certified:
        assert np.linalg.norm(Gr @ x - rhs) / (np.linalg.norm(Gr) * np.linalg.norm(x)) < 1e-15
