"""The Krylov basis of GMRES (fp_gmres.cu): one there is no room for is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(fp, nc, ns):
    w = fp.meshes.swept_wing("0012", nc, ns)
    body = fp.RigidWakeBody(w)
    normals = fp.calc_normals(body)
    D = np.tile([1.0, 0.0, 0.0], (w.nsheddings, 1))
    c = fp._capi.Context(0)
    c.set_geometry(w.nodes, w.panel_offsets, w.panel_nodes, fp.calc_controlpoints(body, normals), normals)
    c.set_wake(w.shedding, D, D)
    a = np.deg2rad(4.2)
    return c, np.tile([np.cos(a), 0.0, np.sin(a)], (w.npanels, 1))


def _solve(fp, c, U, memory, itmax=0):
    opts = fp._capi.make_opts("gmres", "fp64", gmres_memory=memory, gmres_atol=1e-10, gmres_rtol=1e-10, gmres_itmax=itmax)
    return c.solve_body(fp._capi.FP_ELEMENT_VORTEXRING, U, opts=opts)


def test_basis_without_room(fp):
    """A storage hint of 4e7 vectors of 4,160 doubles (1.3 TB): an error of the
    device, and the context solves on."""
    c, U = _setup(fp, 46, 90)
    with pytest.raises(fp._capi.FlowPanelError, match="GMRES basis"):
        _solve(fp, c, U, 40_000_000, 40_000_000)
    x, st = _solve(fp, c, U, 50)
    assert st.gmres_iters > 0 and np.isfinite(x).all()
    c.close()
