"""The FP64 factorisation's trailing update on the INT8 tensor cores (fp_i8.cu),
against the oracle's LAPACK solve and the update on the FP64 tensor path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# rows below the first 256-column panel: 2,048 (the least that takes the digits,
# whole tiles), 2,124 and 4,332 (partial tiles of rows and columns, several
# panels with digits), 2,044 (none)
@pytest.mark.parametrize("nc,ns", [(48, 48), (34, 70), (62, 74), (50, 46)])
def test_i8_update_matches_oracle(fp, O, nc, ns):
    w = fp.meshes.swept_wing("0012", nc, ns)
    body = fp.RigidWakeBody(w)
    normals = fp.calc_normals(body)
    cps = fp.calc_controlpoints(body, normals)
    a = np.deg2rad(4.2)
    V = np.array([np.cos(a), 0.0, np.sin(a)])
    D = np.tile(V, (w.nsheddings, 1))
    U = np.tile(V, (w.npanels, 1))
    xs = []
    for mode in (6, 5):   # the default, and the FP64 tensor path for every panel
        c = fp._capi.Context(0)
        try:
            c.set_tuning(fp._capi.FP_TUNE_FP64_DMMA, mode)
            c.set_geometry(w.nodes, w.panel_offsets, w.panel_nodes, cps, normals)
            c.set_wake(w.shedding, D, D)
            xs.append(c.solve_body(fp._capi.FP_ELEMENT_VORTEXRING, U, opts=fp._capi.make_opts("ludiv", "fp64")))
        finally:
            c.close()
    Gr = O.assemble_vortexring(w, cps, normals, D, D)
    rhs = O.rhs_noflowthrough(U, normals)
    xr = O.solve_ludiv(Gr, rhs)
    x, st = xs[0]
    assert st.gepp_certified == xs[1][1].gepp_certified and st.max_abs_L == pytest.approx(xs[1][1].max_abs_L, rel=1e-12)
    assert np.linalg.norm(x - xr) / np.linalg.norm(xr) < 1e-10
    assert np.linalg.norm(x - xs[1][0]) / np.linalg.norm(x) < 1e-12
    # backward error of the raw solve at the level of an FP64 factorisation's
    assert np.linalg.norm(Gr @ x - rhs) / (np.linalg.norm(Gr) * np.linalg.norm(x)) < 1e-15
