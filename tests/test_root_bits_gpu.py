"""sqrt_pos against the IEEE square root on every float of its range, and what
RootRange lets through, in a kernel built from the engine's own header."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

from tracetransform_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "tt_common.cuh"
// differing roots of the floats with bits first + i, i < count
__global__ void compare(unsigned first, unsigned count, unsigned long long *bad) {
    unsigned mine = 0;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
         i < count; i += (unsigned long long)gridDim.x * blockDim.x) {
        const float v = __uint_as_float(first + (unsigned)i);
        mine += __float_as_uint(tt::sqrt_pos(v)) != __float_as_uint(__fsqrt_rn(v));
    }
    if (mine)
        atomicAdd(bad, (unsigned long long)mine);
}
__global__ void odd(const unsigned *bits, int count, int *out) {
    const int i = threadIdx.x;
    if (i < count) {
        tt::RootRange r;
        r.add(__uint_as_float(bits[i]));
        out[i] = r.odd();
    }
}
extern "C" int run_compare(unsigned first, unsigned count, void *bad) {
    compare<<<1024, 256>>>(first, count, (unsigned long long *)bad);
    return (int)cudaDeviceSynchronize();
}
extern "C" int run_odd(const void *bits, int count, void *out) {
    odd<<<1, 64>>>((const unsigned *)bits, count, (int *)out);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def kernels(tmp_path_factory):
    d = tmp_path_factory.mktemp("roots")
    src, lib = os.path.join(d, "roots.cu"), os.path.join(d, "libroots.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build.nvcc()] + build._flags() + ["-shared", src, "-o", lib], check=True)
    return ctypes.CDLL(lib)


LOW, HIGH = 0x0D800000, 0x7F7FFFFF  # 2^-100, the largest float


def test_sqrt_pos_is_the_ieee_root(kernels):
    bad = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    p = ctypes.c_void_p(bad.data_ptr())
    assert kernels.run_compare(ctypes.c_uint(0), ctypes.c_uint(1), p) == 0  # zero
    assert kernels.run_compare(ctypes.c_uint(LOW), ctypes.c_uint(HIGH - LOW + 1), p) == 0
    assert bad.item() == 0


def test_root_range(kernels):
    bits = [0, LOW, HIGH, 0x3F800000, 1, LOW - 1, HIGH + 1, 0x7FC00000, 0x7F800001, 0x80000000,
            0x80000001, 0xBF800000, 0xFF800000, 0xFFFFFFFF]
    d = torch.from_numpy(np.array(bits, np.uint32).view(np.int32)).cuda()
    out = torch.zeros(len(bits), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert kernels.run_odd(ctypes.c_void_p(d.data_ptr()), len(bits),
                           ctypes.c_void_p(out.data_ptr())) == 0
    assert out.tolist() == [0] * 4 + [1] * (len(bits) - 4)
