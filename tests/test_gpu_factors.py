"""The FP64 factors themselves, entry by entry: |PA - LU| against |L||U| in the rows
below each 64-column block (L21 = A21 U11^-1), also where a block-local pivot is small
and the solve would refine."""
import ctypes as C
import importlib.util
import os
import subprocess

import numpy as np
import pytest

from conftest import freestream

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def factors(tmp_path_factory):
    spec = importlib.util.spec_from_file_location("fp_build", os.path.join(ROOT, "flowpanel.jl_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    if not os.path.exists(build.NVCC):
        pytest.skip("no nvcc")
    out = str(tmp_path_factory.mktemp("factors") / "libfactors.so")
    subprocess.run([build.NVCC, *build.FLAGS, "-shared", "-I" + build.CSRC, os.path.join(ROOT, "tests", "factors.cu"),
                    "-o", out], check=True, capture_output=True, timeout=300)
    return C.CDLL(out).factors


# 480 unknowns: two panels, the second of 3 1/2 blocks; 264: a block of 8 columns last.
# spread: rows scaled by powers of two up to it (the normals are the caller's), so
# that the pivots of a block are not the column's
@pytest.mark.parametrize("nc,ns", [(20, 24), (22, 12)])
@pytest.mark.parametrize("spread", [0, 10, 20])
def test_entries_of_l21(fp, ctx, factors, nc, ns, spread):
    w = fp.meshes.swept_wing("0012", nc, ns)
    body = fp.RigidWakeBody(w)
    normals = fp.calc_normals(body)
    cps = fp.calc_controlpoints(body, normals)
    n = w.npanels
    scale = 2.0 ** np.random.default_rng(1).integers(0, spread + 1, n)
    D = np.tile(freestream(4.2), (w.nsheddings, 1))
    ctx.set_geometry(w.nodes, w.panel_offsets, w.panel_nodes, cps, normals * scale[:, None])
    ctx.set_wake(w.shedding, D, D)
    ctx.assemble(fp._capi.FP_ELEMENT_VORTEXRING)
    G = ctx.get_aic()
    ctx.factor(fp._capi.FP_PREC_FP64)
    lu, piv = np.empty((n, n), order="F"), np.empty(n, np.int32)
    assert factors(ctx.h, lu.ctypes.data_as(C.c_void_p), piv.ctypes.data_as(C.c_void_p)) == 0
    perm = np.arange(n)
    for i, q in enumerate(piv):
        perm[[i, q]] = perm[[q, i]]
    L = np.tril(lu, -1) + np.eye(n)
    U = np.triu(lu)
    R = np.abs(G[perm].astype(np.longdouble) - L.astype(np.longdouble) @ U.astype(np.longdouble)).astype(float)
    q = R / (np.abs(L) @ np.abs(U))
    below = np.arange(n)[:, None] // 64 > np.arange(n)[None, :] // 64
    # a sum of up to n products: sqrt(n) 2^-53 = 2.4e-15 of the largest partial sum, a few roundings more
    assert q[below].max() < 4e-15
