"""The device's panel records (fp_geometry.cu) against the host's geometry: the
AIC with formed and with given control points and normals."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["quads", "triangles", "mixed", "source", "one"])
@pytest.mark.parametrize("offset", [1e-14, 0.013])
def test_geometry_matches_host(fp, O, shape, offset):
    if shape in ("mixed", "source"):   # triangles at the poles, quads between; 129 panels: a partial block of threads
        m = fp.meshes.sphere(1.0, 3, 43)
    else:
        m = fp.meshes.swept_wing("2412", 4, 2 if shape == "one" else 34, sweep=30.0, twist_tip=-2.0)
        m = fp.meshes.triangulate(m) if shape == "triangles" else m
    source = shape == "source"
    body = (fp.NonLiftingBody if source else fp.RigidWakeBody)(m, CPoffset=offset)
    normals = fp.calc_normals(body)
    cps = fp.calc_controlpoints(body, normals)
    a = np.deg2rad(4.2)
    D = np.tile([np.cos(a), 0.0, np.sin(a)], (m.nsheddings, 1))
    solver = fp.B200Solver()
    c = solver.ctx
    G = []
    for given in (False, True):
        solver.load(body, *((normals, cps) if given else ()))
        if m.nsheddings:
            c.set_wake(m.shedding, D, D)
        c.assemble(body.element)
        G.append(c.get_aic())
    solver.close()
    Gr = O.assemble_source(m, cps, normals) if source else O.assemble_vortexring(m, cps, normals, D, D)
    scale = np.abs(Gr).max()
    assert np.abs(G[1] - Gr).max() < 1e-12 * scale
    # formed control points differ by the order of a sum: an ulp of their coordinates, seen by the nearest
    # edge at a distance of at least 1/100 of them
    assert np.abs(G[0] - G[1]).max() < 1e-12 * scale
