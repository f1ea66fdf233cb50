"""rcp_newton (device_common.cuh), the reciprocal of the packed pair terms, equals
__frcp_rn on every float of its range [2^-100, 2^100]: the bit-exact force mode
rests on it.  A small program compiled with the library's flags counts the differences."""
import subprocess

import pytest

from femmd_old_gb300 import build

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include <cuda_runtime.h>
#include "femmd_internal.h"
#include "device_common.cuh"

__global__ void compare(unsigned first, unsigned count, unsigned long long *differ) {
    unsigned long long n = 0;
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const float x = __uint_as_float(first + k);
        n += __float_as_uint(femmd::rcp_newton(x)) != __float_as_uint(__frcp_rn(x));
    }
    if (n) atomicAdd(differ, n);
}

int main() {
    // 2^-100 to 2^100: biased exponents 27 to 227
    const unsigned first = 27u << 23, last = 227u << 23;
    unsigned long long *d, h = 1;
    if (cudaMalloc(&d, sizeof h) || cudaMemset(d, 0, sizeof h)) return 1;
    compare<<<1216, 256>>>(first, last - first + 1, d);
    if (cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost)) return 1;
    printf("%u %llu\n", last - first + 1, h);
    return 0;
}
"""


def test_every_float_of_the_range(tmp_path):
    src, exe = tmp_path / "rcp.cu", tmp_path / "rcp"
    src.write_text(PROGRAM)
    subprocess.run([build._nvcc(), *build.FLAGS, str(src), "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True)
    assert r.stdout.split() == [str((200 << 23) + 1), "0"]
