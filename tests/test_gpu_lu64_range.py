"""Entries of very different size in one matrix: the FP64 factors hold the small
ones to FP64 too. Two spheres of sources, one 100 or 1,000 times smaller and 10
away, their panels in one random order; the freestream is on the small one only, so
the strengths of the large one are its response, 1e-9 of the small one's."""
import numpy as np
import pytest
import scipy.linalg as sla

pytestmark = pytest.mark.gpu


# 2,592 panels: 10 panels of 256 columns, 9 trailing updates; 722: two
@pytest.mark.parametrize("ns", [36, 19])
@pytest.mark.parametrize("size", [1e-2, 1e-3])
def test_response_of_the_large_body(fp, ns, size):
    large, small = fp.meshes.sphere(1.0, ns, ns), fp.meshes.sphere(size, ns, ns)
    small.nodes = small.nodes + np.array([0.0, 10.0, 1.0])
    m = fp.meshes.concat([large, small])
    perm = np.random.default_rng(1).permutation(m.npanels)
    cells = [m.panel(i) for i in perm]
    m = fp.meshes.Mesh(m.nodes, np.cumsum([0] + [len(c) for c in cells]).astype(np.int32),
                       np.concatenate(cells).astype(np.int32), m.shedding, m.bodies)
    far = perm < large.npanels
    body = fp.NonLiftingBody(m)
    normals = fp.calc_normals(body)
    U = np.where(far[:, None], 0.0, np.array([1.0, 0.0, 0.0]))
    solver = fp.B200Solver()
    solver.load(body, normals, fp.calc_controlpoints(body, normals))
    x, st = solver.ctx.solve_body(body.element, U, opts=solver.opts)
    G = solver.ctx.get_aic()
    solver.close()
    assert st.gepp_certified and st.ir_iters == 0   # the factors' own accuracy
    b = -np.einsum("ij,ij->i", U, normals)
    lu = sla.lu_factor(G)
    t = sla.lu_solve(lu, b).astype(np.longdouble)
    for _ in range(4):   # refined with residuals in extended precision
        t = t + sla.lu_solve(lu, (b.astype(np.longdouble) - G.astype(np.longdouble) @ t).astype(float))
    t = t.astype(float)
    # n eps = 6e-13 at most, of a system that is nearly its diagonal
    for part in (far, ~far):
        assert np.linalg.norm(x[part] - t[part]) < 1e-12 * np.linalg.norm(t[part])
