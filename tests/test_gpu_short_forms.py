"""The straight-line roots and reciprocals (fp_elements.cuh: the FP64 and FP32 ring
kernels, the multipliers of the FP64 LU) against CUDA's correctly rounded ones."""
import importlib.util
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def counts(tmp_path_factory):
    spec = importlib.util.spec_from_file_location("fp_build", os.path.join(ROOT, "flowpanel.jl_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    if not os.path.exists(build.NVCC):
        pytest.skip("no nvcc")
    exe = str(tmp_path_factory.mktemp("short_forms") / "short_forms")
    subprocess.run([build.NVCC, *build.FLAGS, "-I" + build.CSRC, os.path.join(ROOT, "tests", "short_forms.cu"), "-o", exe],
                   check=True, capture_output=True, timeout=300)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    return {k: int(v) for k, v in (line.split() for line in out.splitlines())}


def test_fp64_values(counts):
    """600 million random arguments of 2^-990 .. 2^990: correctly rounded. With
    mantissas at all ones (a chance of 2^-52 else) within an ulp."""
    for k in ("rcp64", "rcp64_negative", "inv64", "inv64_offset", "far64", "far64_ones"):
        assert counts[k] == 0, k


def test_fp32_values(counts):
    """All 1.7e9 arguments of the exponents -100 .. 99: correctly rounded."""
    assert counts["rcp32"] == 0 and counts["sqrt32"] == 0
