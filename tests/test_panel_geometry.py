"""Normals, areas and control points on the host (bodies.py): meshes of one panel
shape take whole arrays at once, with the values of the panel-by-panel indexing."""
import numpy as np
import pytest


def _polygons(fp, corners, n=5):
    """n flat polygons of `corners` nodes each, in planes of their own."""
    a = 2 * np.pi * np.arange(corners) / corners
    ring = np.stack([np.cos(a), np.sin(a), np.zeros(corners)], axis=1)
    rng = np.random.default_rng(corners)
    nodes = np.concatenate([ring @ np.linalg.qr(rng.standard_normal((3, 3)))[0] + 3.0 * i for i in range(n)])
    return fp.meshes.Mesh(nodes, np.arange(0, corners * n + 1, corners, dtype=np.int32),
                          np.arange(corners * n, dtype=np.int32), bodies=[fp.meshes.Body("p", "vortexring", n, 0)])


# the frame and the first triangle's area of a pentagon are those of its first three nodes
@pytest.mark.parametrize("corners", [3, 4, 5, 6])
def test_uniform_meshes(fp, corners):
    m = _polygons(fp, corners)
    body = fp.RigidWakeBody(m)
    P = m.nodes.reshape(-1, corners, 3)
    c = np.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
    area = 0.5 * np.linalg.norm(c, axis=1)
    assert np.allclose(fp.calc_normals(body), c / np.linalg.norm(c, axis=1)[:, None], rtol=0, atol=1e-14)
    if corners == 4:
        area = area + 0.5 * np.linalg.norm(np.cross(P[:, 2] - P[:, 0], P[:, 3] - P[:, 0]), axis=1)
    assert np.allclose(fp.bodies.calc_areas(body), area, rtol=1e-14)
    if corners <= 4:
        assert np.allclose(fp.calc_controlpoints(body), P.mean(axis=1), rtol=0, atol=1e-12)
