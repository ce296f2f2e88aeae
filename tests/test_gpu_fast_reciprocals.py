"""The fast reciprocal and reciprocal root of common.cuh against FP64 division and
square root, over their stated range and its ends."""

import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

from dequantizer_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = """
#include "common.cuh"
__global__ void eval(const double *x, double *a, double *b, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  a[i] = dqz::fast_rsqrt(x[i]);
  b[i] = dqz::fast_rcp(x[i]);
}
extern "C" int run(const double *x, double *a, double *b, int n) {
  eval<<<(n + 255) / 256, 256>>>(x, a, b, n);
  return (int)cudaDeviceSynchronize();
}
"""


def test_within_two_ulp(tmp_path):
    """A seed of about 20 bits and a third-order step leave 2^-60, and the rounding
    of the step one ulp; the reference (division and root, half an ulp each) adds
    one: 2 ulp = 2^-51 relative."""
    src, lib = tmp_path / "eval.cu", tmp_path / "eval.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler",
                    "-fPIC", "--shared", "-I", build.CSRC, "-I", os.path.join(os.path.dirname(build.HERE), "include"),
                    str(src), "-o", str(lib)], check=True)
    rng = np.random.default_rng(1)
    one = np.array([1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0), 2.0, np.nextafter(4.0, 1.0)])
    x = np.concatenate([10.0 ** rng.uniform(-290, 290, 4_000_000), rng.uniform(1.0, 4.0, 12_000_000),
                        [1e-290, 1e290], np.ldexp(one[:, None], np.arange(-960, 960)[None, :]).ravel()])
    x = torch.from_numpy(x[(x >= 1e-290) & (x <= 1e290)]).cuda()
    a, b = torch.empty_like(x), torch.empty_like(x)
    run = ctypes.CDLL(str(lib)).run
    run.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int]
    torch.cuda.synchronize()
    assert run(x.data_ptr(), a.data_ptr(), b.data_ptr(), x.numel()) == 0
    for got, want in ((a, 1.0 / x.sqrt()), (b, 1.0 / x)):
        assert float(((got - want) / want).abs().max()) <= 2.0 ** -51
