"""The roots and reciprocals that the pair loops form from approximate instructions
(csrc/sph_device.cuh), on every float of the stated ranges, against sqrtf and the
division: the reciprocal may differ (by an ulp) where the mantissa is all ones and
nowhere else, the root nowhere from 2^-100 to 2^100 and by an ulp below."""
import ctypes as C
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "sph_device.cuh"
using namespace sph;

// out: floats from first to last (bit patterns) that differ, those of them whose
// mantissa is all ones, the largest difference in ulp
__global__ void k_compare(int what, uint32_t first, uint32_t last, unsigned long long* out) {
    unsigned long long n = 0, ones = 0, most = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t b = first + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b <= last; b += stride) {
        const float x = __uint_as_float((uint32_t)b);
        const float got = what ? rcp_exact(x) : sqrt_exact(x, rsqrt_approx(x));
        const float want = what ? 1.0f / x : sqrtf(x);
        const int d = abs((int)(__float_as_uint(got) - __float_as_uint(want)));
        if (d) {
            ++n;
            if (((uint32_t)b & 0x7fffffu) == 0x7fffffu) ++ones;
            if ((unsigned long long)d > most) most = d;
        }
    }
    if (n) {
        atomicAdd(out, n);
        atomicAdd(out + 1, ones);
        atomicMax(out + 2, most);
    }
}
extern "C" int compare(int what, uint32_t first, uint32_t last, unsigned long long* host) {
    unsigned long long* d = nullptr;
    if (cudaMalloc(&d, 24) != cudaSuccess) return 1;
    cudaMemset(d, 0, 24);
    k_compare<<<1216, 256>>>(what, first, last, d);
    const cudaError_t e = cudaMemcpy(host, d, 24, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e != cudaSuccess;
}
"""


def _bits(e):
    """Bit pattern of 2^e."""
    return (e + 127) << 23


@pytest.fixture(scope="module")
def compare(tmp_path_factory):
    from libfluid_gb300 import build as B
    d = tmp_path_factory.mktemp("exact_math")
    (d / "compare.cu").write_text(SOURCE)
    so = os.path.join(d, "compare.so")
    subprocess.run([B.NVCC, *B.NVCC_FLAGS, "-shared", "-o", so, str(d / "compare.cu")], check=True)
    fn = C.CDLL(so).compare
    fn.argtypes = [C.c_int, C.c_uint32, C.c_uint32, C.POINTER(C.c_uint64)]

    def run(what, first, last):
        out = (C.c_uint64 * 3)()
        assert fn(what, first, last, out) == 0
        return tuple(out)
    return run


def test_reciprocal(compare):
    differ, ones, ulps = compare(1, _bits(-126), _bits(126))
    print(differ, ones, ulps)
    assert differ == ones and ulps <= 1


def test_root(compare):
    assert compare(0, _bits(-100), _bits(100)) == (0, 0, 0)
    differ, _, ulps = compare(0, _bits(-126) + 1, _bits(-100))
    print(differ, ulps)
    assert ulps <= 1
