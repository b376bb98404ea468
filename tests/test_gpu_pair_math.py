"""The square root and the exponential of the pair terms against CUDA's
functions, bit for bit, over every FP32 value of the ranges in which the
kernels use them: roots of [2.7e-20, 4e37], and 2^-x for x in [0, 126] (a pair
inside the kernel has x <= 0.19)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_pair_math_has_the_bits_of_the_cuda_functions(gpu, tmp_path):
    exe = os.path.join(str(tmp_path), "pair_math")
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    os.path.join(ROOT, "tests", "cpp", "pair_math_probe.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split("\n")
    rows = {r.split()[0]: [int(v) for v in r.split()[1:]] for r in out if r}
    assert rows["sqrt"][0] > 1_500_000_000 and rows["exp2"][0] > 1_100_000_000
    assert rows["sqrt"][1] == 0
    assert rows["exp2"][1] == 0
