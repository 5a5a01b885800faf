"""The double-float operations of csrc/df64.cuh themselves, on the GPU: sums and
products-and-sums of known order and sums with a power-of-two weight have the
general operations' bits, comparisons the exact difference's sign."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NAMES = ("add_ordered", "add_ordered_float", "float_add_ordered", "add_scaled", "fma_large", "fma_small",
         "fma_small_const", "less")


def test_shortened_operations(tmp_path):
    from raptor_gb300 import build
    exe = str(tmp_path / "df64_check")
    subprocess.run([build.nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-I" + os.path.join(ROOT, "raptor_gb300", "csrc"), os.path.join(ROOT, "tests", "df64_check.cu"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()
    assert dict(zip(NAMES, map(int, out))) == {n: 0 for n in NAMES}
