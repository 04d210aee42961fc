"""The backprojectors' reciprocals (csrc/common.cuh) against 1 / x in float64: every mantissa of
one binade and random ones of every binade in [2^-126, 2^126], both signs."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from reconstruction_program_taichi_gb300 import _build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "common.cuh"

__global__ void reciprocals(int n, const float* x, float* one, float* two) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    one[i] = mct::reciprocal(x[i]);
    const float2 r = mct::reciprocal2(make_float2(x[i], x[n - 1 - i]));
    two[i] = r.x;
    two[n + n - 1 - i] = r.y;
}

extern "C" int run(int n, const float* x, float* one, float* two, void* stream) {
    reciprocals<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(n, x, one, two);
    return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def lib(cuda, tmp_path_factory):
    d = tmp_path_factory.mktemp("reciprocal")
    (d / "r.cu").write_text(SOURCE)
    out = str(d / "libr.so")
    subprocess.run([_build.nvcc_path(), *_build.ARCH, "-std=c++17", "-O3", "-shared", "-Xcompiler", "-fPIC", "-cudart", "shared",
                    "-I", _build.CSRC, "-I", os.path.join(ROOT, "include"), str(d / "r.cu"), "-o", out], check=True)
    return ctypes.CDLL(out)


def _values(which):
    if which == "binade":
        return np.arange(1 << 23, dtype=np.uint32) + np.uint32(127 << 23)
    rng = np.random.default_rng(3)
    bits = (np.repeat(np.arange(1, 253, dtype=np.uint32), 16384) << 23) | rng.integers(0, 1 << 23, 252 * 16384, dtype=np.uint32)
    return bits | (rng.integers(0, 2, bits.size, dtype=np.uint32) << 31)


@pytest.mark.parametrize("which", ["binade", "range"])
def test_reciprocals_are_within_their_bound(which, lib):
    """Half an ulp of the result and 2^-45 of it, as derived beside the function."""
    import torch
    x = _values(which).view(np.float32)
    n = x.size
    xt = torch.from_numpy(x.copy()).cuda()
    one, two = torch.empty(n, device="cuda"), torch.empty(2 * n, device="cuda")
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in (xt, one, two)]
    assert lib.run(n, *ptr, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    one, two = one.cpu().numpy(), two.cpu().numpy()
    exact = 1.0 / x.astype(np.float64)
    bound = 0.5 * np.spacing(np.abs(one)).astype(np.float64) + 2.0 ** -45 * np.abs(exact)
    assert (np.abs(one - exact) <= bound).all()
    assert np.array_equal(two[:n], one) and np.array_equal(two[n:], one)


def test_reciprocals_of_zero_and_infinity_are_no_numbers(lib):
    import torch
    xt = torch.tensor([0.0, -0.0, float("inf"), -float("inf"), float("nan"), 2.0], device="cuda")
    one, two = torch.empty(6, device="cuda"), torch.empty(12, device="cuda")
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in (xt, one, two)]
    assert lib.run(6, *ptr, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    assert torch.isnan(one[:5]).all() and one[5] == 0.5
    assert torch.isnan(two[:5]).all() and torch.isnan(two[6:11]).all()
