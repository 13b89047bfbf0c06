"""The static-order FP32 factors hold an FP32 factorisation's accuracy: the residual
of one solve with them, before any refinement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_residual_of_the_first_solve(fp, ctx):
    """Spheres of sources (dominant diagonals, |L| about 0.01) of one to two diagonal
    blocks. The residual is roundings of A, of x and of the two sweeps, some ten of
    6e-8 / sqrt(3) each: 1.1e-7, and what the factorisation adds. Elimination by
    blocks adds a few roundings of an entry's size (1.6e-7 in all, with either
    kernel); 128 subtractions from the entry, one after another, 2.1e-7."""
    got = []
    for nt, np_ in ((8, 12), (10, 12), (16, 8), (16, 16)):
        m = fp.meshes.sphere(1.0, nt, np_)
        body = fp.NonLiftingBody(m)
        normals = fp.calc_normals(body)
        ctx.set_geometry(m.nodes, m.panel_offsets, m.panel_nodes, fp.calc_controlpoints(body, normals), normals)
        for seed in range(6):
            U = np.random.default_rng(seed).standard_normal((m.npanels, 3))
            _, st = ctx.solve_body(body.element, U, opts=fp._capi.make_opts("ludiv", "mixed", ir_tol=1e-3))
            assert st.ir_iters == 1
            got.append(st.rel_residual)
    assert np.sqrt(np.mean(np.square(got))) < 1.85e-7
