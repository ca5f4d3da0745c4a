"""vebi_fp64.cuh's products, quotients and roots against the GPU's FP64 instructions, bit for bit, on 2^26
seeded operands of every class, with the GPU's own FP32 approximations as starts."""
import pathlib
import subprocess

import pytest

from vebisph_gb300 import build

pytestmark = pytest.mark.gpu

ROOT = pathlib.Path(__file__).resolve().parent.parent


def test_results_are_the_instructions(tmp_path):
    exe = tmp_path / "device"
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false", "-I", str(build.CSRC), "-o", str(exe),
                    str(ROOT / "tests" / "fp64" / "device.cu")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
