"""One tet's constraints by register pairs (solve_tet_pairs, batched_kernel.cuh) against the
same expressions written value by value with the compiler's operators: every correction has
the same bits and every count is the same, for tets of all sizes from far below to far above
the range of the written-out quotients and roots, flat and collapsed tets, fixed vertices,
constraints that are off, and each kind of folded edge."""

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
__host__ __device__ unsigned mix(unsigned long long z) {  // splitmix64's finaliser
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull; z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return (unsigned)((z ^ (z >> 31)) >> 16);
}
struct Out { float d[12]; int cnt[4]; int bad, dyn; };
__device__ void edge(V pu, V pv, float mu, float mv, float L0, float active, V& du, V& dv, int& cu, int& cv, int& dyn,
                     float ks, float sc, int& k) {
    const float w = mu + mv;
    if (w < float(BEPS)) return;
    const V dir = pv - pu;
    const float len = sqrtf(dot(dir, dir));
    if (len < float(BEPS)) { --cu; --cv; dyn = 1; return; }
    const float C = len - L0;
    const V d = -C * (dir / len) * ks * active / w;
    du = du - (d * mu) * sc; dv = dv + (d * mv) * sc;
    ++k;
}
__device__ Out plain(unsigned fl, const TetRec& rc, const float4* x, bool fold, float ksv, float ksd, float sc, float off) {
    Out o = {};
    V p[4]; float m[4];
    for (int i = 0; i < 4; ++i) { p[i] = T3<float>(x[i].x, x[i].y, x[i].z); m[i] = x[i].w; }
    const V p1 = p[1] - p[0], p2 = p[2] - p[0], p3 = p[3] - p[0];
    const bool anym = m[0] != 0 || m[1] != 0 || m[2] != 0 || m[3] != 0;
    V d[4] = {};
    int k = 0, skip = 0;
    if ((fl & FFSRL_VOLUME) && rc.va.y == 1.0f) {
        V q[4];
        q[1] = cross(p2, p3); q[2] = cross(p3, p1); q[3] = cross(p1, p2); q[0] = -q[1] - q[2] - q[3];
        const float w = m[0] * dot(q[0], q[0]) + m[1] * dot(q[1], q[1]) + m[2] * dot(q[2], q[2]) + m[3] * dot(q[3], q[3]);
        if (fabsf(w) < float(BEPS)) { if (anym) ++skip; }
        else {
            const float dl = -ksv * rc.va.y * (rc.va.x - fabsf(dot(q[3], p3)) / 6.0f) / w;
            for (int i = 0; i < 4; ++i) d[i] = q[i] * dl * (m[i] * sc);
            ++k;
        }
    }
    if (fl & FFSRL_NEOHOOKEAN) {
        const float D[3][3] = {{rc.n0.x, rc.n0.y, rc.n1.z}, {rc.n0.z, rc.n0.w, rc.n1.w}, {rc.n1.x, rc.n1.y, rc.n2.x}};
        V f[3], c[3], g[4], n[4];
        for (int j = 0; j < 3; ++j) f[j] = p1 * D[0][j] + p2 * D[1][j] + p3 * D[2][j];
        c[0] = cross(f[1], f[2]); c[1] = cross(f[2], f[0]); c[2] = cross(f[0], f[1]);
        for (int i = 0; i < 3; ++i) g[i + 1] = c[0] * D[i][0] + c[1] * D[i][1] + c[2] * D[i][2];
        g[0] = -g[1] - g[2] - g[3];
        const float C = dot(f[0], c[0]) - 1.0f - off;
        float w = 0.0f;
        for (int i = 0; i < 4; ++i) { const float l = sqrtf(dot(g[i], g[i])); w = i ? w + l * l * m[i] : l * l * m[i]; }
        if (w < float(BEPS)) { if (anym) ++skip; }
        else {
            float dl = -C / (w + rc.n2.y);
            for (int i = 0; i < 4; ++i) n[i] = g[i] * dl * (m[i] * sc);
            float r = 0.0f;
            for (int j = 0; j < 3; ++j) { const float l = sqrtf(dot(f[j], f[j])); r = j ? r + l * l : l * l; }
            const float rs = sqrtf(r), rsi = 1.0f / rs;
            for (int i = 0; i < 3; ++i) g[i + 1] = (f[0] * D[i][0] + f[1] * D[i][1] + f[2] * D[i][2]) * rsi;
            g[0] = -g[1] - g[2] - g[3];
            for (int i = 0; i < 4; ++i) { const float l = sqrtf(dot(g[i], g[i])); w = i ? w + l * l * m[i] : l * l * m[i]; }
            if (w < float(BEPS)) { if (anym) ++skip; }
            else {
                dl = -rs / (w + rc.n2.z);
                for (int i = 0; i < 4; ++i) d[i] = d[i] + (n[i] + g[i] * dl * (m[i] * sc));
                ++k;
            }
        }
    }
    int cnt[4] = {-skip, -skip, -skip, -skip}, dyn = skip != 0;
    if (fold) {
        if (rc.ed.y != 0.0f) edge(p[0], p[1], m[0], m[1], rc.ed.x, rc.ed.y, d[0], d[1], cnt[0], cnt[1], dyn, ksd, sc, k);
        if (rc.ed.w != 0.0f) {
            if (rc.ed.z > 0.0f) edge(p[2], p[3], m[2], m[3], rc.ed.z, rc.ed.w, d[2], d[3], cnt[2], cnt[3], dyn, ksd, sc, k);
            else edge(p[0], p[2], m[0], m[2], -rc.ed.z, rc.ed.w, d[0], d[2], cnt[0], cnt[2], dyn, ksd, sc, k);
        }
    }
    for (int i = 0; i < 4; ++i) {
        o.cnt[i] = cnt[i];
        if (!isfinite(abs_sum(d[i])) && k) o.bad = 1;
        if (k) { o.d[3 * i] = d[i].x; o.d[3 * i + 1] = d[i].y; o.d[3 * i + 2] = d[i].z; }
    }
    o.dyn = dyn;
    return o;
}
__device__ bool same(float a, float b) { return a == b || (a != a && b != b); }  // (a zero's sign adds nothing)
__global__ void check(Dev<float> D, unsigned fl, int size, int odd, int n, Out* out, unsigned long long* wrong) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    unsigned long long c = (unsigned long long)i << 8;
    auto u = [&]() { return (float)(mix(++c + 977 * size) >> 8) / 16777216.0f; };  // [0, 1)
    const float h = exp2f((float)size);
    float4 x[4];
    for (int v = 0; v < 4; ++v) {
        x[v] = make_float4(h * u(), h * u(), h * u(), u() < 0.2f ? 0.0f : 0.5f + u());
        if (odd == 1 && v == 3) { x[3].x = x[2].x; x[3].y = x[2].y; x[3].z = x[2].z; }       // collapsed
        if (odd == 2) x[v].z = 0.0f;                                                         // flat
        if (odd == 3) x[v].w = 0.0f;                                                         // fixed
        if (odd == 4 && v == 1) x[v].y = u() < 0.5f ? INFINITY : NAN;
    }
    TetRec rc;
    rc.ix = make_uint2(0u | 1u << 16, 2u | 3u << 16);
    float* q = &rc.n0.x;
    for (int e = 0; e < 4; ++e) { q[e] = (u() - 0.5f) * 4.0f / h; (&rc.n1.x)[e] = (u() - 0.5f) * 4.0f / h; }
    rc.n2 = make_float4((u() - 0.5f) * 4.0f / h, 1e-3f * u(), 1e-3f * u(), 0.0f);
    rc.va = make_float2(h * h * h * u() * 0.2f, u() < 0.8f ? 1.0f : 0.0f);
    rc.ed = make_float4(h * u(), u() < 0.8f ? 1.0f : 0.0f, (u() < 0.5f ? -h : h) * (u() + 0.1f), u() < 0.7f ? 1.0f : 0.0f);
    const bool fold = u() < 0.8f;
    const float sc = 1048576.0f;
    const Out want = plain(fl, rc, x, fold, D.ks_volume, D.ks_distance, sc, 0.01f);
    Out& got = out[i];  // zeros (the sums are atomic: global memory)
    bool bad = false;
    const Wide<false> wd{nullptr, 0, nullptr, 0.0f, nullptr};
    solve_tet_pairs<AccAtomic, false>(D, fl, rc, 0, 0, fold, x, got.d, got.cnt, 1, sc, 0.01f, &got.dyn, bad, wd);
    bool ok = bad == (want.bad != 0) && got.dyn == want.dyn;
    for (int v = 0; v < 12; ++v) ok = ok && same(got.d[v], want.d[v]);
    for (int v = 0; v < 4; ++v) ok = ok && got.cnt[v] == want.cnt[v];
    if (!ok) atomicAdd(wrong, 1ull);
}
extern "C" long long run(unsigned fl, int size, int odd, int n) {
    Dev<float> D = {};
    D.nzero = 0x8000000080000000ull;
    D.ks_volume = 0.9f; D.ks_distance = 0.7f;
    unsigned long long *d, h = 0;
    if (cudaMalloc((void**)&d, 8) || cudaMemset(d, 0, 8)) return -1;
    Out* o;
    if (cudaMalloc((void**)&o, n * sizeof(Out)) || cudaMemset(o, 0, n * sizeof(Out))) return -1;
    check<<<(n + 127) / 128, 128>>>(D, fl, size, odd, n, o, d);
    if (cudaMemcpy(&h, d, 8, cudaMemcpyDeviceToHost)) return -1;
    cudaFree(d);
    cudaFree(o);
    return (long long)h;
}
"""


@pytest.fixture(scope="module")
def run(gpu, tmp_path_factory):
    d = tmp_path_factory.mktemp("pairs")
    (d / "pairs.cu").write_text(SRC)
    so = d / "pairs.so"
    # the flags of the reference-arithmetic units
    subprocess.run([_build._nvcc(), *_build.ARCH, *_build.COMMON, "-fmad=false", "-shared", str(d / "pairs.cu"), "-o",
                    str(so)], check=True)
    f = ctypes.CDLL(str(so)).run
    f.restype, f.argtypes = ctypes.c_longlong, [ctypes.c_uint, ctypes.c_int, ctypes.c_int, ctypes.c_int]
    return f


@pytest.mark.parametrize("flags", [1, 4, 5])  # volume, Neo-Hookean, both
@pytest.mark.parametrize("odd", range(5))
def test_pairs_give_the_plain_expressions_bits(run, flags, odd):
    assert [run(flags, size, odd, 20000) for size in (-14, -9, -3, 0, 5, 13, 22, 31)] == [0] * 8
