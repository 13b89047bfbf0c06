"""The static-order factorisation by groups of four panels (lu_static_groups in
fp_lu_static.cu): groups cut short after each panel, ragged last
panels, against the one by single panels and the residual in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 7,192 and 7,200: 24 and 32 columns in a 57th panel; 57 to 60 whole panels; then
# one panel or less, the second begun, one to two groups
@pytest.mark.parametrize("nc,ns", [(58, 124), (90, 80), (96, 76), (116, 64), (118, 64), (96, 80),
                                   (10, 10), (16, 8), (12, 12), (16, 16), (20, 14), (32, 16), (34, 16), (40, 24)])
def test_groups_against_single_panels(fp, nc, ns):
    m = fp.meshes.swept_wing("0012", nc, ns)
    cap = fp._capi
    V = np.array([np.cos(0.07), 0.0, np.sin(0.07)])
    D = np.tile(V, (m.nsheddings, 1))
    U = np.tile(V, (m.npanels, 1))
    x, st = [], []
    c = cap.Context(0)
    try:
        c.set_geometry(m.nodes, m.panel_offsets, m.panel_nodes)
        c.set_wake(m.shedding, D, D)
        for split in (1, 0):
            c.set_tuning(cap.FP_TUNE_LU_SPLIT, split)
            a, b = c.solve_body(cap.FP_ELEMENT_VORTEXRING, U, opts=cap.make_opts("ludiv", "mixed"))
            x.append(np.asarray(a).ravel())
            st.append(b)
    finally:
        c.close()
    assert np.isfinite(x[0]).all()
    # both refined to FP64 working accuracy: the condition number (1e5) times 1e-16 apart
    assert np.linalg.norm(x[0] - x[1]) < 1e-10 * np.linalg.norm(x[1])
    assert st[0].ir_iters <= st[1].ir_iters + 1   # as good a factorisation
