"""The roots, reciprocals and quotients of device.cuh (sqrt_rn, rcp_rn, quotient_rn) are the
correctly rounded ones: every float of [2^-100, 2^100) for the one-operand functions, every
numerator mantissa over the 64 largest and 64 smallest denominator mantissas and 8.6 billion
random pairs for the quotient, compared on the GPU with CUDA's own operators (no result may
differ)."""
import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_exact_math(cuda_device, tmp_path):
    exe = str(tmp_path / "exact_math")
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false",
                    "-std=c++17", "-I" + os.path.join(ROOT, "smallproject_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "exact_math.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.split() == ["0"] * 4, (r.returncode, r.stdout)
