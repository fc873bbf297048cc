"""Compiled form of FSIM's transform kernels of the shared-memory engine: their transforms are inlined and every
kernel of up to 256 threads leaves room for a second CTA on an SM (65536 registers, allotted 8 a thread at a time)."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_transform_kernels_fit_twice():
    csrc = os.path.join(ROOT, "iqm_b200", "csrc")
    out = subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                          "--expt-relaxed-constexpr", "-Xptxas", "-v", "-I", os.path.join(ROOT, "include"), "-I", csrc, "-c",
                          "-o", os.devnull, os.path.join(csrc, "fsim.cu")], check=True, capture_output=True, text=True).stderr
    kernels = re.findall(r"Compiling entry function '\w*?(fsim_(?:fwd|inv)_(?:rows|cols)(?:_seq)?_kernel)\w*'.*?"
                         r"(\d+) bytes spill stores.*?Used (\d+) registers", out, re.S)
    assert len(kernels) == 6, out[-2000:]
    for name, spill, registers in kernels:
        assert int(spill) == 0 and 2 * 256 * ((int(registers) + 7) // 8 * 8) <= 65536, (name, spill, registers)
    assert "warp_stockham" not in out
