"""The Krylov basis of GMRES (fp_gmres.cu): it grows for a step that is taken, not for
one launched ahead, and a basis there is no room for is refused."""
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


def test_basis_does_not_grow_for_steps_ahead(fp):
    """Device memory of a solve of `steps` steps with room for exactly those and with
    room for the two launched ahead: a basis that doubled would hold 5 MB or more on top."""
    torch = pytest.importorskip("torch")
    used, xs = [], []
    c, U = _setup(fp, 46, 90)
    x, st = _solve(fp, c, U, 1000)
    c.close()
    steps = st.gmres_iters
    assert 150 < steps < 998   # doubling the basis: steps x 33 KB, 5 MB or more
    for memory in (steps + 2, steps):
        free0 = torch.cuda.mem_get_info()[0]
        c, U = _setup(fp, 46, 90)
        y, st = _solve(fp, c, U, memory)
        used.append(free0 - torch.cuda.mem_get_info()[0])
        c.close()
        assert st.gmres_iters == steps and (y == x).all()
    assert abs(used[1] - used[0]) <= 4 << 20   # the allocator's granularity, 2 MB a buffer


def test_basis_without_room(fp):
    """A storage hint of 4e7 vectors of 4,160 doubles (1.3 TB): an error of the
    device, and the context solves on."""
    c, U = _setup(fp, 46, 90)
    with pytest.raises(fp._capi.FlowPanelError, match="GMRES basis"):
        _solve(fp, c, U, 40_000_000, 40_000_000)
    x, st = _solve(fp, c, U, 50)
    assert st.gmres_iters > 0 and np.isfinite(x).all()
    c.close()


def test_breakdown_with_steps_ahead(fp):
    """A tolerance of zero on 16 unknowns: the Krylov space is exhausted while later
    steps are under way. The process ends unconverged, and the context's next solve
    is that of a new one."""
    c, U = _setup(fp, 4, 4)
    with pytest.raises(fp._capi.FlowPanelError, match="did not reach its tolerance"):
        c.solve_body(fp._capi.FP_ELEMENT_VORTEXRING, U,
                     opts=fp._capi.make_opts("gmres", "fp64", gmres_memory=3, gmres_atol=0.0, gmres_rtol=0.0))
    x, st = _solve(fp, c, U, 50)
    c.close()
    c, U = _setup(fp, 4, 4)
    y, sy = _solve(fp, c, U, 50)
    c.close()
    assert (x == y).all() and st.gmres_iters == sy.gmres_iters
