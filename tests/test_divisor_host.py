"""The divisor of the fused FP64 sweeps (adjoint.cuh, ReciprocalDivisor) against the division it
stands for: tests/cpp/test_divisor.cu, host code of the kernel's own template."""

import os
import subprocess

from mikroptim_b200 import build as mbuild

HERE = os.path.dirname(os.path.abspath(__file__))


def test_the_corrected_quotient_is_the_rounded_one():
    out = os.path.join(HERE, "cpp", "_build")
    os.makedirs(out, exist_ok=True)
    exe = os.path.join(out, "test_divisor")
    cmd = [mbuild.nvcc(), *mbuild.ARCH, "-O2", "-std=c++17", "--expt-relaxed-constexpr",
           "-Xcompiler", "-ffp-contract=off", "-cudart", "static",
           "-I", mbuild.CSRC, "-I", os.path.join(mbuild.ROOT, "include"),
           os.path.join(HERE, "cpp", "test_divisor.cu"), "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    res = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0 and "divisor checks passed" in res.stdout, res.stdout
