"""Divisions written out in the kernels (csrc/mlp_math.cuh, csrc/fd1d_onchip.cuh) against CUDA's `/`: every float operand
of SiLU and its derivative, and reciprocals of doubles from 2^-1000 to 2^1000."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "fd1d_onchip.cuh"
#include "mlp_math.cuh"
using namespace kwg;
using ull = unsigned long long;
__device__ ull steps(float a, float b)
{
    const long long x = __float_as_int(a) < 0 ? -(long long)(__float_as_int(a) & 0x7fffffff) : __float_as_int(a);
    const long long y = __float_as_int(b) < 0 ? -(long long)(__float_as_int(b) & 0x7fffffff) : __float_as_int(b);
    return (ull)(x > y ? x - y : y - x);
}
__device__ ull steps(double a, double b)
{
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    return (ull)(x > y ? x - y : y - x);
}
// out: [0] operands in range, [1] largest distance in floats of SiLU, [2] operands with one, [3] largest of |SiLU| below -87 (bits),
// [4] SiLU above 87 that is not z, [5] derivative beyond its bound, [6] operands, [7] distance of rcp, [8] rcp of 0, inf, nan finite
__global__ void floats(ull* out)
{
    ull n = 0, far = 0, off = 0, big = 0, low = 0, dbad = 0;
    const ull step = (ull)gridDim.x * blockDim.x;
    for (ull b = blockIdx.x * (ull)blockDim.x + threadIdx.x; b < (1ull << 32); b += step) {
        const float z = __uint_as_float((unsigned)b);
        if (!isfinite(z)) continue;
        const float d = 1.f + __expf(-z), v = silu_f(z);
        if (fabsf(z) <= 87.f) {
            ++n;
            const ull k = steps(v, z / d);
            far = k > far ? k : far;
            off += k > 0;
        } else if (z > 0.f) {
            big += v != z;
        } else {
            const ull m = __float_as_uint(fabsf(v - z / d));
            low = m > low ? m : low;
        }
        if (fabsf(z) <= 1e4f) {
            const float s = z < -87.f ? 0.f : 1.f / d;
            dbad += !(fabsf(dsilu_f(z) - s * (1.f + z * (1.f - s))) <= 0x1p-22f * s * (1.f + fabsf(z)));
        }
    }
    atomicAdd(&out[0], n);
    atomicMax(&out[1], far);
    atomicAdd(&out[2], off);
    atomicMax(&out[3], low);
    atomicAdd(&out[4], big);
    atomicAdd(&out[5], dbad);
}
__global__ void doubles(ull* out)
{
    ull n = 0, far = 0;
    const ull step = (ull)gridDim.x * blockDim.x;
    for (ull i = blockIdx.x * (ull)blockDim.x + threadIdx.x; i < (1ull << 26); i += step) {
        ull h = (i + 1) * 0x9E3779B97F4A7C15ull;
        h = (h ^ (h >> 30)) * 0xBF58476D1CE4E5B9ull;
        h = (h ^ (h >> 27)) * 0x94D049BB133111EBull;
        h ^= h >> 31;
        const int e = i % 2 ? (int)(h >> 52) % 2001 - 1000 : (int)(h >> 52) % 101;  // half of them pivots: 1 to 2^100
        double d = __longlong_as_double((long long)((ull)(1023 + e) << 52 | (h & 0xfffffffffffffull)));
        if (i % 3 == 0) d = -d;
        ++n;
        const ull k = steps(rcp(d), 1. / d);
        far = k > far ? k : far;
    }
    atomicAdd(&out[6], n);
    atomicMax(&out[7], far);
    if (blockIdx.x == 0 && threadIdx.x == 0)
        for (double d : {0., -0., INFINITY * 1., -INFINITY * 1., NAN * 1.}) out[8] += isfinite(rcp(d)) ? 1 : 0;
}
extern "C" int run(ull* host)
{
    ull* out = nullptr;
    if (cudaMalloc(&out, 16 * sizeof(ull)) != cudaSuccess) return 1;
    cudaMemset(out, 0, 16 * sizeof(ull));
    floats<<<4096, 256>>>(out);
    doubles<<<4096, 256>>>(out);
    const cudaError_t e = cudaMemcpy(host, out, 16 * sizeof(ull), cudaMemcpyDeviceToHost);
    cudaFree(out);
    return e == cudaSuccess ? 0 : 2;
}
"""


@pytest.fixture(scope="module")
def counts(built, tmp_path_factory):
    import build_lib

    tmp = tmp_path_factory.mktemp("device_math")
    src, so = str(tmp / "device_math.cu"), str(tmp / "device_math.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build_lib._nvcc(), *build_lib.ARCH, *build_lib.NVFLAGS, "-shared", src, "-o", so, "-lcudart"], check=True)
    out = (ctypes.c_ulonglong * 16)()
    assert ctypes.CDLL(so).run(out) == 0
    os.remove(so)
    return list(out)


def test_silu_is_the_division(counts):
    """The quotient before its rounding is off by 2^-45, half an ulp being 2^-24: the neighbour of `/`'s result for
    about one operand in 2^20 (a factor of 4 beside it), never another."""
    assert counts[0] > 2.0**31
    assert counts[1] <= 1 and counts[2] <= counts[0] * 2.0**-18
    assert np.array([counts[3]], np.uint32).view(np.float32)[0] <= 1.5e-36 and counts[4] == 0


def test_silu_derivative(counts):
    """s within an ulp of 1 / d, which moves the derivative by 2^-23 s (1 + |z|) at most, and as much for its own roundings."""
    assert counts[5] == 0


def test_double_reciprocal(counts):
    """Within an ulp of `/`; nothing finite from zero, infinity or NaN."""
    assert counts[6] == 2**26 and counts[7] <= 1 and counts[8] == 0
