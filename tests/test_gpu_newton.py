"""The square roots and the reciprocal of M-SVD's and FSIM's kernels (iqm_b200/csrc/iqm_internal.cuh) on the GPU
against double precision.  sqrt_newton and rcp_newton refine an SFU value that is within 2^-23 or so: the step
leaves the square of that and the roundings of its last two operations, below an ulp of 2^-23.  sqrt_approx
is the SFU's own, within 2^-23 by the PTX manual; its 0 is exact."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("native") / "newton_check")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "iqm_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "newton_check.cu")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=120).stdout
    return {n: (float(a), float(b)) for n, a, b in map(str.split, out.splitlines())}


@pytest.mark.parametrize("name", ["sqrt_newton", "rcp_newton", "sqrt_approx"])
def test_helper_within_an_ulp(results, name):
    ours, cuda = results[name]
    print("%s: helper %.3e, CUDA %.3e" % (name, ours, cuda))
    assert ours <= 2.0 ** -23
