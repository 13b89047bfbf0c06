"""FP64 vortex rings at the limits of the short roots and reciprocals
(short_forms in fp_elements.cuh): targets that no edge counts, coordinates and
offsets out of their range, meshes with a panel of no extent."""
import numpy as np
import pytest

from conftest import freestream

pytestmark = pytest.mark.gpu

NONE = np.zeros((0, 3))


def _sphere(fp, scale=1.0, split=False):
    m = fp.meshes.sphere(1.0, 12, 11)   # quadrilaterals, triangles at the poles
    m = fp.meshes.triangulate(m) if split else m
    m.nodes = scale * m.nodes
    return m


def test_targets_without_a_velocity(fp, ctx):
    """NaN and infinite targets lie within every edge's cutoff, and far enough
    away the factor underflows: the value already in `out` stays."""
    m = _sphere(fp)
    g = np.random.default_rng(5).standard_normal(m.npanels)
    X = np.array([[np.nan, 0, 0], [0, np.nan, 1], [np.inf, 0, 0], [0, -np.inf, 1], [np.inf, np.nan, 0],
                  [1e80, 0, 0], [1e100, 1e100, 1], [1e155, 0, 0]])
    ctx.set_geometry(m.nodes, m.panel_offsets, m.panel_nodes)
    for count in (1, 200):   # one block, and targets spread over several
        out = ctx.uind(fp._capi.FP_ELEMENT_VORTEXRING, g, np.tile(X, (count, 1)), np.full((count * len(X), 3), 7.0))
        assert (out == 7.0).all()


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("scale,offset,cutoff", [(1.0, -1e-8, 1e-14), (1.0, 0.0, 1e-14), (1.0, 1e-8, 0.0), (1.0, 0.0, 0.0),
                                                 (2.0 ** 61, 1e-8, 1e-14), (2.0 ** 59, 1e-8, 1e-14), (2.0 ** -200, 0.0, 0.0)])
def test_out_of_range_matches_oracle(fp, O, ctx, split, scale, offset, cutoff):
    m = _sphere(fp, scale, split)
    body = fp.RigidWakeBody(m, CPoffset=0.0)
    normals = fp.calc_normals(body)
    cps = fp.calc_controlpoints(body, normals)
    rng = np.random.default_rng(6)
    g = rng.standard_normal(m.npanels)
    X = np.concatenate([cps + 0.03 * scale * normals, 3 * scale * rng.standard_normal((67, 3)),
                        m.nodes[:9] + 1e-9 * scale * rng.standard_normal((9, 3))])
    ctx.set_geometry(m.nodes, m.panel_offsets, m.panel_nodes, cps, normals)
    ctx.assemble(fp._capi.FP_ELEMENT_VORTEXRING, offset, cutoff)
    G = ctx.get_aic()
    u = ctx.uind(fp._capi.FP_ELEMENT_VORTEXRING, g, X, None, fp._capi.FP_PREC_FP64, offset, cutoff)
    Gr = O.assemble_vortexring(m, cps, normals, NONE, NONE, offset, cutoff)
    ur = O.uind_vortexring(m, g, NONE, NONE, X, offset, cutoff)
    # the bounds of the shared-edge tests; beside a node the edges' cross products cancel to 1e-9 of
    # their terms, so that both sides hold about 1e-7 of the field there
    assert np.abs(G - Gr).max() < 1e-12 * np.abs(Gr).max()
    assert np.abs(u[:-9] - ur[:-9]).max() < 1e-12 * np.abs(ur[:-9]).max()
    assert np.abs(u[-9:] - ur[-9:]).max() < 1e-5 * np.abs(ur[-9:]).max()


@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_gepp"])
@pytest.mark.parametrize("kind", ["no first edge", "no area"])
def test_degenerate_panel_is_refused(fp, kind, precision):
    """A panel without a frame has no control point: its row of the AIC is zero
    and the solve is refused, not answered with NaN."""
    m = fp.meshes.swept_wing("0012", 8, 8)
    p = m.panel(20)
    if kind == "no first edge":
        m.nodes[p[1]] = m.nodes[p[0]]
    else:
        m.nodes[p[2]] = 2 * m.nodes[p[1]] - m.nodes[p[0]]
    body = fp.RigidWakeBody(m)
    V = freestream(4.2)
    D = np.tile(V, (m.nsheddings, 1))
    solver = fp.B200Solver("ludiv", precision)
    with pytest.raises(fp._capi.FlowPanelError, match="zero pivot"):
        fp.solve(body, np.tile(V, (m.npanels, 1)), D, D, solver=solver)
    solver.close()


def _vjp(ctx, m, g, X, W, offset=1e-8):
    ctx.set_geometry(m.nodes, m.panel_offsets, m.panel_nodes)
    ctx.assemble(1, offset)
    return ctx.uind_vjp(g, X, W, m.nnodes)


def test_reverse_mode_of_far_targets(fp, ctx):
    """Targets whose cross products overflow or are not numbers add nothing to
    the gradient of an ordinary one."""
    m = _sphere(fp)
    rng = np.random.default_rng(8)
    g, W = rng.standard_normal(m.npanels), rng.standard_normal((4, 3))
    X = np.array([[1.7, 0.4, -0.3], [1e90, 1e90, 1e90], [np.nan, 0, 0], [-1e95, 2e95, 1e94]])
    one, all_ = _vjp(ctx, m, g, X[:1], W[:1]), _vjp(ctx, m, g, X, W)
    assert (all_["dtargets"][1:] == 0.0).all()
    for k in ("dnodes", "dstrengths"):   # the same terms, added in another order
        assert np.abs(all_[k] - one[k]).max() < 1e-14 * np.abs(one[k]).max()
    assert np.abs(all_["dtargets"][0] - one["dtargets"][0]).max() < 1e-14 * np.abs(one["dtargets"]).max()


@pytest.mark.parametrize("offset,scale", [(-1e-8, 1.0), (0.0, 1.0), (1e-8, 2.0 ** 61), (1e-8, 2.0 ** 59)])
def test_reverse_mode_out_of_range(fp, O, ctx, offset, scale):
    """Against the oracle's Dual numbers, to the bound of test_gpu_adjoint.py."""
    m = _sphere(fp, scale)
    rng = np.random.default_rng(9)
    g = rng.standard_normal(m.npanels)
    X = scale * np.concatenate([1.1 * rng.standard_normal((40, 3)), m.nodes[:4] / scale + 1e-3 * rng.standard_normal((4, 3))])
    W = rng.standard_normal(X.shape)
    got = _vjp(ctx, m, g, X, W, offset)
    for key in ("dnodes", "dtargets", "dstrengths"):
        v = rng.standard_normal(got[key].shape)
        _, dF = O.uind_jvp(m, g, NONE, NONE, X, W, offset=offset, **{key: v})
        assert abs(np.sum(got[key] * v) - dF) <= 1e-9 * np.sum(np.abs(got[key] * v))
