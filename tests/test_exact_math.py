"""The reference form's own reciprocal, square root and quotients (Markstein's corrected
approximations, batched_kernel.cuh) against the compiler's correctly rounded operators:
all significands of the reciprocal, the root (both parities of the exponent) and the sixth,
and 2^32 seeded pairs of the quotient.  They scale with the exponents, so two binades stand
for all within the range they are used for; the ends of that range, and what lies beyond
it (zeros, infinities, NaN), are compared too."""

import ctypes
import subprocess

import pytest

from ffsrl import _build

pytestmark = pytest.mark.gpu

SRC = r"""
#include "batched_kernel.cuh"
using namespace ffsrl::bk;
__device__ unsigned mix(unsigned long long z) {  // splitmix64's finaliser
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull; z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return (unsigned)((z ^ (z >> 31)) >> 16);
}
__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }
__global__ void check(int what, unsigned long long n, unsigned long long* bad) {
    unsigned long long wrong = 0;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const float x = __uint_as_float(0x3f800000u + (unsigned)i);
        if (what == 0) wrong += !same(exact_rcp(x), 1.0f / x);
        if (what == 1) wrong += !same(exact_root(x), sqrtf(x));
        if (what == 2) wrong += !same(sixth(x), x / 6.0f);
        if (what == 3) {
            const unsigned u = mix(2 * i), v = mix(2 * i + 1);
            const float a = __uint_as_float((u & 0x807fffffu) | ((107u + (u >> 23) % 41u) << 23));
            const float b = __uint_as_float((v & 0x807fffffu) | ((107u + (v >> 23) % 41u) << 23));
            wrong += !same(quot(a, b), a / b);
        }
        if (what == 4) {  // values at and beyond the range's ends: the operators decide
            const float e[12] = {0.0f, 1e-45f, 1e-38f, kExactMin, 2.0f * kExactMin, 1.0f, 0.5f * kExactMax, kExactMax,
                                 3.0e38f, __uint_as_float(0x7f800000u), __uint_as_float(0x7fc00000u), -3.0f};
            const float a = e[5 + i % 2], b = e[(i / 2) % 12], c = e[(i / 24) % 11];
            wrong += !same(quot(a, b), a / b);
            const t3<float> q = quot(T3<float>(a, -a, a), b);
            wrong += !same(q.x, a / b) + !same(q.y, -a / b);
            float r[2] = {c, a};
            roots(r);
            wrong += !same(r[0], sqrtf(c)) + !same(r[1], sqrtf(a));
        }
    }
    if (wrong) atomicAdd(bad, wrong);
}
extern "C" long long run(int what, unsigned long long n) {
    unsigned long long *d, h = 0;
    if (cudaMalloc((void**)&d, 8) || cudaMemset(d, 0, 8)) return -1;
    check<<<1216, 256>>>(what, n, d);
    if (cudaMemcpy(&h, d, 8, cudaMemcpyDeviceToHost)) return -1;
    cudaFree(d);
    return (long long)h;
}
"""


@pytest.fixture(scope="module")
def run(gpu, tmp_path_factory):
    d = tmp_path_factory.mktemp("exact")
    (d / "exact.cu").write_text(SRC)
    so = d / "exact.so"
    # the flags of the reference-arithmetic units
    subprocess.run([_build._nvcc(), *_build.ARCH, *_build.COMMON, "-fmad=false", "-shared", str(d / "exact.cu"), "-o",
                    str(so)], check=True)
    f = ctypes.CDLL(str(so)).run
    f.restype, f.argtypes = ctypes.c_longlong, [ctypes.c_int, ctypes.c_ulonglong]
    return f


@pytest.mark.parametrize("what,n", [("reciprocal", 1 << 24), ("root", 1 << 24), ("sixth", 1 << 24), ("quotient", 1 << 32),
                                    ("range", 2 * 12 * 11)])
def test_correctly_rounded(run, what, n):
    assert run(["reciprocal", "root", "sixth", "quotient", "range"].index(what), n) == 0
