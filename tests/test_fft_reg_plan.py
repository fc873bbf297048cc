"""The register FFT engine's plans (iqm_b200/csrc/fft_reg.cu) on the CPU: every step's radix is compiled,
its lines cover the sequence's shared memory exactly once, and steps and tables compute the DFT.  The
tables are double values rounded to float (2^-25 relative each), a Bluestein point passes five of them, so
an output is within 1e-6 of the inputs' norm."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("native") / "fft_reg_check")
    csrc = os.path.join(ROOT, "iqm_b200", "csrc")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2",
                    "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include"), "-I", csrc, "-o", exe,
                    os.path.join(ROOT, "tests", "native", "fft_reg_check.cu"), os.path.join(csrc, "fft_reg.cu")], check=True)
    return exe


# every length of usual plane sides; around the longest Bluestein plan (m = 6000); the largest sides
@pytest.mark.parametrize("lo,hi", [(2, 520), (1020, 1035), (2995, 3005), (4090, 4096)])
def test_plans_compute_the_dft(checker, lo, hi):
    r = subprocess.run([checker, str(lo), str(hi)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[-200:]
    for line in r.stdout.splitlines():
        n, kind, err = line.split()
        assert float(err) <= 1e-6, line
        if int(n) <= 3000:
            assert kind != "none", line
