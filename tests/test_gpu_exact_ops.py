"""The raymarch's reciprocal, square root, quotient, power and exponential
without special cases against CUDA's own, bit for bit, over whole binades
(GB300 only; compiles a small kernel around the library's header)."""
import ctypes as C
import subprocess

import pytest

from meteoros_gb300 import build

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SOURCE = r"""
#include "mt_device.cuh"
using namespace mt;
__device__ bool differ(float a, float b) { return __float_as_uint(a) != __float_as_uint(b); }
// every mantissa at one exponent: mismatches of {rcp(b), rcp(-b), sqrt, quotients, pow, exp}
__global__ void check(int exponent, unsigned long long* bad) {
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    const float b = __uint_as_float(((unsigned)(exponent + 127) << 23) | m);
    if (differ(rcp_core(b), __frcp_rn(b))) atomicAdd(bad + 0, 1ull);
    if (differ(rcp_core(-b), __frcp_rn(-b))) atomicAdd(bad + 1, 1ull);
    if (differ(sqrt_core(b), __fsqrt_rn(b))) atomicAdd(bad + 2, 1ull);
    unsigned h = m * 2654435761u + 12345u;
    for (int i = 0; i < 8; ++i) {
        h = h * 1664525u + 1013904223u;
        const float a = __uint_as_float((h & 0x807fffffu) | ((unsigned)(127 - 8 + (h >> 24) % 16) << 23));
        if (differ(div_core(a, b), __fdiv_rn(a, b))) atomicAdd(bad + 3, 1ull);
    }
    if (exponent <= 0 && exponent >= -30) {  // densities in (0, 1], light densities
        const float y = 0.5f + 1.5f * (float)(h >> 8) * (1.0f / 16777216.0f);
        if (differ(pow_ftz(b, y), __powf(b, y))) atomicAdd(bad + 4, 1ull);
    }
    if (exponent <= 6 && b < 80.0f && differ(exp_ftz(-b), __expf(-b))) atomicAdd(bad + 5, 1ull);
}
extern "C" __attribute__((visibility("default"))) int run(int exponent, unsigned long long* host) {
    unsigned long long* d = nullptr;
    if (cudaMalloc((void**)&d, 64) != cudaSuccess) return 1;
    cudaMemset(d, 0, 64);
    check<<<(1 << 23) / 256, 256>>>(exponent, d);
    const cudaError_t e = cudaMemcpy(host, d, 48, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    folder = tmp_path_factory.mktemp("exact_ops")
    (folder / "check.cu").write_text(SOURCE)
    lib = folder / "check.so"
    subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, *build.EXACT, f"-I{build.CSRC}", "-shared", "-o", str(lib),
                    str(folder / "check.cu")], check=True, capture_output=True)
    return C.CDLL(str(lib))


@pytest.mark.parametrize("exponent", [-60, -31, -24, -10, -2, -1, 0, 1, 2, 7, 22, 23, 44, 45, 60])
def test_core_operations_equal_cudas(harness, exponent):
    bad = (C.c_ulonglong * 6)()
    assert harness.run(exponent, bad) == 0
    assert list(bad) == [0] * 6, f"mismatches of rcp, rcp(-), sqrt, quotient, pow, exp at 2^{exponent}: {list(bad)}"
