"""The reference form's written-out quotients (batched_kernel.cuh) against the compiler's
correctly rounded division for operands of every magnitude: dividends and divisors from the
smallest subnormal to infinity, zeros and NaN, as scalars, vectors and sixths; and a tet's
two edges side by side, with components, stretches and activities down to the subnormals:
the same bits, and in the form for fixed-point sums the same integers."""

import ctypes
import subprocess

import pytest

from ffsrl import _build

pytestmark = pytest.mark.gpu

SRC = r"""
#include "batched_kernel.cuh"
using namespace ffsrl;
using namespace ffsrl::bk;
typedef t3<float> V;
__device__ unsigned mix(unsigned long long z) {  // splitmix64's finaliser
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull; z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return (unsigned)((z ^ (z >> 31)) >> 16);
}
__device__ bool same(float a, float b) { return a == b || (a != a && b != b); }  // (a zero's sign adds nothing)
struct Rng {
    unsigned long long c;
    __device__ unsigned bits() { return mix(++c * 0x9E3779B97F4A7C15ull); }
    __device__ float unit() { return (float)(bits() >> 8) / 16777216.0f; }
    // any sign and significand; an exponent field from lo to hi; now and then a zero
    __device__ float any(int lo, int hi) {
        const unsigned u = bits(), e = (unsigned)(lo + (int)(bits() % (unsigned)(hi - lo + 1)));
        return bits() % 32u == 0u ? 0.0f : __uint_as_float((u & 0x807fffffu) | (e << 23));
    }
};
__device__ void edge(V pu, V pv, float mu, float mv, float L0, float active, V& du, V& dv, int& cu, int& cv, float ks, float sc, int& k) {
    const float w = mu + mv;
    if (w < float(BEPS)) return;
    const V dir = pv - pu;
    const float len = sqrtf(dot(dir, dir));
    if (len < float(BEPS)) { --cu; --cv; return; }
    const float C = len - L0;
    const V d = -C * (dir / len) * ks * active / w;
    du = du - (d * mu) * sc; dv = dv + (d * mv) * sc;
    ++k;
}
__global__ void check(int what, unsigned long long n, int* cnts, int* dyn, unsigned long long* bad, unsigned long long nzero) {
    unsigned long long wrong = 0;
    const unsigned long long i0 = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    for (unsigned long long i = i0; i < n; i += (unsigned long long)gridDim.x * blockDim.x) {
        Rng r{i * 256};
        if (what == 0) {
            const float a = r.any(0, 255), b = r.any(0, 255);
            wrong += !same(quot(a, b), a / b);
        }
        if (what == 1) {
            const V a = T3<float>(r.any(0, 255), r.any(60, 190), r.any(0, 130));
            const float b = r.any(60, 190);
            const V q = quot(a, b);
            wrong += !same(q.x, a.x / b) || !same(q.y, a.y / b) || !same(q.z, a.z / b);
        }
        if (what == 2) {
            const float a = r.any(0, 255);
            wrong += !same(sixth(a), a / 6.0f);
        }
        if (what == 3 || what == 4) {
            // each vector has a component of ordinary size and others of any below it
            V p[4];
            float m[4];
            for (int v = 0; v < 4; ++v) {
                const float c[3] = {r.any(0, 128), r.any(0, 128), r.any(0, 128)};
                p[v] = T3<float>(c[0], c[1], c[2]);
                if (v != 2) (&p[v].x)[r.bits() % 3u] = r.any(110, 130);
                m[v] = r.bits() % 8u == 0u ? 0.0f : 0.5f + r.unit();
            }
            auto rest = [&](V a, V b) {  // unstretched, nearly so, or not
                const V d = b - a;
                const float len = sqrtf(dot(d, d));
                const unsigned u = r.bits() % 3u;
                return u == 0u ? len : u == 1u ? len * (1.0f + 1.2e-7f * (float)(r.bits() % 5u)) : len * r.unit();
            };
            auto active = [&]() { return r.bits() % 2u ? 1.0f : fabsf(r.any(0, 127)); };
            const bool cd = r.bits() % 2u;
            const float l1 = cd ? rest(p[2], p[3]) : rest(p[0], p[2]);
            const float4 ed = make_float4(rest(p[0], p[1]), active(), cd ? l1 : -l1, active());
            const float sc = 1048576.0f, ks = 0.7f;
            V want[4] = {}, got[4] = {};
            int wc[4] = {}, k = 0;
            if (ed.y != 0.0f) edge(p[0], p[1], m[0], m[1], ed.x, ed.y, want[0], want[1], wc[0], wc[1], ks, sc, k);
            if (ed.w != 0.0f) {
                if (ed.z > 0.0f) edge(p[2], p[3], m[2], m[3], ed.z, ed.w, want[2], want[3], wc[2], wc[3], ks, sc, k);
                else edge(p[0], p[2], m[0], m[2], -ed.z, ed.w, want[0], want[2], wc[0], wc[2], ks, sc, k);
            }
            int* cnt = cnts + 4 * i0;
            for (int v = 0; v < 4; ++v) cnt[v] = 0;
            const f2 z{nzero};
            const int g = what == 3 ? fold_edges<false, false>(ed, p[0], p[1], p[2], p[3], m[0], m[1], m[2], m[3], got[0], got[1], got[2],
                                                               got[3], 0, 1, 2, 3, cnt, 1, ks, dyn + i0, sc, z)
                                    : fold_edges<false, true>(ed, p[0], p[1], p[2], p[3], m[0], m[1], m[2], m[3], got[0], got[1], got[2],
                                                              got[3], 0, 1, 2, 3, cnt, 1, ks, dyn + i0, sc, z);
            bool ok = g == k;
            for (int v = 0; v < 4; ++v) {
                ok = ok && cnt[v] == wc[v];
                for (int c = 0; c < 3; ++c) {
                    const float a = (&got[v].x)[c], b = (&want[v].x)[c];
                    ok = ok && (what == 3 ? same(a, b) : __float2ll_rn(a) == __float2ll_rn(b));
                }
            }
            wrong += !ok;
        }
    }
    if (wrong) atomicAdd(bad, wrong);
}
extern "C" long long run(int what, unsigned long long n) {
    const int blocks = 1216, threads = 128;
    unsigned long long *d, h = 0;
    int* c;
    if (cudaMalloc((void**)&d, 8) || cudaMemset(d, 0, 8) || cudaMalloc((void**)&c, blocks * threads * 5 * sizeof(int))) return -1;
    check<<<blocks, threads>>>(what, n, c, c + 4 * blocks * threads, d, 0x8000000080000000ull);  // (known at run time only)
    if (cudaMemcpy(&h, d, 8, cudaMemcpyDeviceToHost)) return -1;
    cudaFree(d);
    cudaFree(c);
    return (long long)h;
}
"""


@pytest.fixture(scope="module")
def run(gpu, tmp_path_factory):
    d = tmp_path_factory.mktemp("quotients")
    (d / "quotients.cu").write_text(SRC)
    so = d / "quotients.so"
    # the flags of the reference-arithmetic units
    subprocess.run([_build._nvcc(), *_build.ARCH, *_build.COMMON, "-fmad=false", "-shared", str(d / "quotients.cu"), "-o",
                    str(so)], check=True)
    f = ctypes.CDLL(str(so)).run
    f.restype, f.argtypes = ctypes.c_longlong, [ctypes.c_int, ctypes.c_ulonglong]
    return f


@pytest.mark.parametrize("what,n", [("scalar", 1 << 28), ("vector", 1 << 26), ("sixth", 1 << 26), ("edges", 1 << 24),
                                    ("fixed-point edges", 1 << 24)])
def test_correctly_rounded_at_every_magnitude(run, what, n):
    assert run(["scalar", "vector", "sixth", "edges", "fixed-point edges"].index(what), n) == 0
