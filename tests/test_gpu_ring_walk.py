"""Consecutive panels that share an edge (ring_walk in fp_elements.cuh): every way
the shared edge can lie, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _relabel(fp, m, turn):
    """Each panel's nodes turned by `turn(panel)` places: another edge becomes edge 0."""
    cells = [np.roll(m.panel(i), -turn(i)) for i in range(m.npanels)]
    out = fp.meshes.Mesh(m.nodes.copy(), m.panel_offsets.copy(), np.concatenate(cells).astype(np.int32))
    out.bodies = m.bodies
    return out


# turns that make edge 0 the shared one, or none of a run, or each edge of the
# previous panel in turn; 130 quadrilaterals or 258 triangles: tiles of 32 and 64 with a rest
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("turn", [lambda i: 0, lambda i: 1, lambda i: 2, lambda i: i, lambda i: (i * i + i // 3)])
def test_shared_edges(fp, O, split, turn):
    s = fp.meshes.sphere(1.0, 12, 11)   # quadrilaterals, and triangles at the poles
    m = fp.meshes.triangulate(s) if split else s
    nn = np.diff(m.panel_offsets)
    m = _relabel(fp, m, lambda i: turn(i) % nn[i])
    body = fp.RigidWakeBody(m)
    normals = fp.calc_normals(body)
    cps = fp.calc_controlpoints(body, normals)
    rng = np.random.default_rng(5)
    g = rng.standard_normal(m.npanels)
    X = np.concatenate([cps + 0.03 * normals, 3 * rng.standard_normal((67, 3)), m.nodes[:5]])   # and at nodes
    c = fp._capi.Context(0)
    try:
        c.set_geometry(m.nodes, m.panel_offsets, m.panel_nodes, cps, normals)
        c.assemble(fp._capi.FP_ELEMENT_VORTEXRING)
        G = c.get_aic()
        u64 = c.uind(fp._capi.FP_ELEMENT_VORTEXRING, g, X)
        u32 = c.uind(fp._capi.FP_ELEMENT_VORTEXRING, g, X[:-5], None, fp._capi.FP_PREC_MIXED)
    finally:
        c.close()
    none = np.zeros((0, 3))
    Gr = O.assemble_vortexring(m, cps, normals, none, none)
    assert np.abs(G - Gr).max() < 1e-12 * np.abs(Gr).max()
    ur = O.uind_vortexring(m, g, none, none, X)
    assert np.abs(u64 - ur).max() < 1e-12 * np.abs(ur).max()
    # FP32: coordinates to 6e-8 of 1, distances from 0.03 on, sums of 130 to 258 panels
    assert np.abs(u32 - ur[:-5]).max() < 1e-4 * np.abs(ur[:-5]).max()


# FP32 targets at nodes (the square root's short form has no value there) and
# coordinates beyond its range, among ordinary ones; one target to a few blocks
@pytest.mark.parametrize("scale", [1.0, 2.0 ** 21])
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("m_t", [1, 129, 300])
def test_fp32_beyond_the_short_forms(fp, O, scale, split, m_t):
    s = fp.meshes.sphere(1.0, 12, 11)
    m = fp.meshes.triangulate(s) if split else s
    m.nodes[:] = scale * m.nodes.astype(np.float32)
    rng = np.random.default_rng(7)
    g = rng.standard_normal(m.npanels)
    X = scale * (3 * rng.standard_normal((m_t, 3))).astype(np.float32).astype(float)
    X[::7] = m.nodes[rng.integers(0, len(m.nodes), len(X[::7]))]
    c = fp._capi.Context(0)
    try:
        c.set_geometry(m.nodes, m.panel_offsets, m.panel_nodes)
        u32 = c.uind(fp._capi.FP_ELEMENT_VORTEXRING, g, X, None, fp._capi.FP_PREC_MIXED)
    finally:
        c.close()
    none = np.zeros((0, 3))
    ur = O.uind_vortexring(m, g, none, none, X)
    # as above, the nodes an edge length (0.2) or more from the edges that count
    assert np.abs(u32 - ur).max() < 1e-4 * np.abs(ur).max()
