"""The blend's approximate exponential and reciprocal and its division by 3
(csrc/rm_approx.cuh) against the language's own, over the ranges that the blend
uses them in, from a test kernel compiled here."""
import ctypes
import os
import subprocess

import pytest
import torch

from radiance_meshes_b200 import build

pytestmark = pytest.mark.gpu

# Each kernel looks at the floats whose bit patterns are first, first + step, ...
# below last, and counts those that miss their bound.
SOURCE = r"""
#include <cstdint>
#include "rm_approx.cuh"

__device__ bool miss(int what, float x) {
    if (what == 0) {  // third(x): the same bits as the division
        const float a = rm::third(x), b = x / 3.0f;
        return __float_as_uint(a) != __float_as_uint(b) && !(a != a && b != b);
    }
    if (what == 1) {  // exp_approx(x), x in [-inf, 0]
        const double want = exp((double)x), got = rm::exp_approx(x);
        if (want < 0x1p-126) return !(got >= 0.0 && got <= 0x1p-125);
        return !(fabs(got - want) <= want * (0x1p-22 - (double)x * 0x1p-23));
    }
    const double want = 1.0 / (double)x, got = rm::rcp_approx(x);
    return !(fabs(got - want) <= fabs(want) * 0x1p-23);
}

__global__ void scan(int what, uint32_t first, uint32_t last, uint32_t step, unsigned long long* missed) {
    unsigned long long n = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x * step;
    for (uint64_t i = first + ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * step; i < last; i += stride)
        n += miss(what, __uint_as_float((uint32_t)i));
    if (n) atomicAdd(missed, n);
}

extern "C" __attribute__((visibility("default"))) int run(int what, uint32_t first, uint32_t last, uint32_t step,
                                                           void* missed, void* stream) {
    scan<<<148 * 8, 256, 0, (cudaStream_t)stream>>>(what, first, last, step, (unsigned long long*)missed);
    return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def missed(cuda, tmp_path_factory):
    d = tmp_path_factory.mktemp("approx")
    (d / "approx.cu").write_text(SOURCE)
    out = str(d / "approx.so")
    flags = [f for f in build.NVCC_FLAGS if f not in ("-Xptxas", "-warn-spills")]
    r = subprocess.run([build.nvcc(), *flags, "-I", build.CSRC, "-shared", "-o", out, str(d / "approx.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = ctypes.CDLL(out)

    def run(what, first, last, step=1):
        n = torch.zeros(1, dtype=torch.int64, device=cuda)
        stream = torch.cuda.current_stream().cuda_stream
        assert L.run(what, ctypes.c_uint32(first), ctypes.c_uint32(last), ctypes.c_uint32(step),
                     ctypes.c_void_p(n.data_ptr()), ctypes.c_void_p(stream)) == 0
        return int(n.item())

    return run


def _bits(x):
    return int(torch.tensor(x, dtype=torch.float32).view(torch.int32).item()) & 0xffffffff


def test_third_is_the_division_of_every_non_negative_float(missed):
    assert missed(0, 0, 0x80000000) == 0  # infinity and NaN among them


def test_exp_within_its_bound(missed):
    assert missed(1, 0, 1) == 0  # 0
    assert missed(1, 0x80000000, _bits(-float("inf")) + 1, 3) == 0


@pytest.mark.parametrize("sign", [0, 0x80000000])
def test_reciprocal_within_its_bound(missed, sign):
    assert missed(2, sign + _bits(1e-10), sign + _bits(2.0**126), 3) == 0
