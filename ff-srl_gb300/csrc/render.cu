// render.cu -- BVH refit and ray-cast renderer (reference: FF_SRL/FF_SRL/bvh.py:30-104,
// 419-454 and render.py:81-121, 276-498, 588-724, 975-1022).
//
// This unit is compiled with -fmad=false: every product and sum rounds as written, so
// with IEEE division and square root the images and boxes equal the CPU restatement's
// bit for bit whenever the summation order is the same (the fused paths).
#include <cuda_runtime.h>
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include "ffsrl_internal.h"
#include "vecmath.cuh"

namespace ffsrl {
namespace {

constexpr int kStackCap = 64;  // traversal stack entries per ray (the reference uses 32)

__device__ __forceinline__ int find_env(const int* __restrict__ node_offset, int n_env, int total, int tid) {
    // env whose AABB range [node_offset[e], next) holds tid; node_offset ascending
    int lo = 0, hi = n_env - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (node_offset[mid] <= tid) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// A leaf's box from its triangles' vertices, and the packed copies of both
__device__ __forceinline__ void refit_leaf(const ffsrl_bvh& b, const float* __restrict__ pts,
                                           const int* __restrict__ faces, int e, int n0, int t0, int base, int node) {
    v3 lo = mk(1e6f, 1e6f, 1e6f), hi = mk(-1e6f, -1e6f, -1e6f);
    int first = b.first_tri_id[n0 + node];
    int cnt = b.tri_count[n0 + node];
    long long fofs = b.env_face_offset[e];
    for (int k = 0; k < cnt; ++k) {
        long long f = fofs + b.tri_id[t0 + first + k];
        // the reference's refit may box another face than the one it traverses
        // (bvh.py:66-74 against render.py:462-470); refit_source holds that face
        const long long fb = b.refit_source ? (long long)b.refit_source[f] : f;
        v3 pA = ld3(pts, faces[3 * fb]), pB = ld3(pts, faces[3 * fb + 1]), pC = ld3(pts, faces[3 * fb + 2]);
        lo = vmin(pA, vmin(pB, vmin(pC, lo)));
        hi = vmax(pA, vmax(pB, vmax(pC, hi)));
        if (fb != f) pA = ld3(pts, faces[3 * f]), pB = ld3(pts, faces[3 * f + 1]), pC = ld3(pts, faces[3 * f + 2]);
        if (b.tri_pos) {
            float4* q = reinterpret_cast<float4*>(b.tri_pos) + 3 * (fofs + first + k);
            q[0] = make_float4(pA.x, pA.y, pA.z, pB.x);
            q[1] = make_float4(pB.y, pB.z, pC.x, pC.y);
            q[2] = make_float4(pC.z, 0.0f, 0.0f, 0.0f);
        }
    }
    if (b.node_box) {
        float4* nb = reinterpret_cast<float4*>(b.node_box) + 2ll * (base + node);
        nb[0] = make_float4(lo.x, lo.y, lo.z, __int_as_float(-1));
        nb[1] = make_float4(hi.x, hi.y, hi.z, __int_as_float(first * 256 + (cnt < 255 ? cnt : 255)));
    }
    st3(b.aabb_min, base + node, lo);
    st3(b.aabb_max, base + node, hi);
}

// An inner node's box from its children's (l0, h0 the left one's), and the packed copy
__device__ __forceinline__ void refit_inner(const ffsrl_bvh& b, int base, int node, int left, v3 l0, v3 h0, v3 l1,
                                            v3 h1, v3& lo, v3& hi) {
    lo = vmin(l0, l1);
    hi = vmax(h0, h1);
    if (b.node_box) {
        // the traversal's child order: the axis along which the children's centres lie
        // farthest apart (bits 0-1) and whether the right child's centre is the higher
        // one (bit 2)
        const v3 d = (l1 + h1) - (l0 + h0);
        const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
        const int axis = (ax >= ay && ax >= az) ? 0 : (ay >= az ? 1 : 2);
        const float da = axis == 0 ? d.x : (axis == 1 ? d.y : d.z);
        float4* nb = reinterpret_cast<float4*>(b.node_box) + 2ll * (base + node);
        nb[0] = make_float4(lo.x, lo.y, lo.z, __int_as_float(left));
        nb[1] = make_float4(hi.x, hi.y, hi.z, __int_as_float(axis | (da > 0.0f ? 4 : 0)));
    }
    st3(b.aabb_min, base + node, lo);
    st3(b.aabb_max, base + node, hi);
}
__device__ __forceinline__ void refit_inner_global(const ffsrl_bvh& b, int base, int node, int left) {
    v3 lo, hi;
    refit_inner(b, base, node, left, ld3(b.aabb_min, base + left), ld3(b.aabb_max, base + left),
                ld3(b.aabb_min, base + left + 1), ld3(b.aabb_max, base + left + 1), lo, hi);
}

// refitBVHLevel (bvh.py:30-104): every env node at `level`
__global__ void k_refit_level(ffsrl_bvh b, const float* __restrict__ pts, const int* __restrict__ faces, int level) {
    int tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= b.total_env_nodes) return;
    int e = find_env(b.env_node_offset, b.num_envs, b.total_env_nodes, tid);
    int topo = b.env_topology[e];
    int n0 = b.topo_node_offset[topo];
    int node = tid - b.env_node_offset[e];
    if (node >= b.topo_node_offset[topo + 1] - n0) return;
    if (b.level[n0 + node] != level) return;
    const int left = b.left_node[n0 + node];
    if (left < 0) refit_leaf(b, pts, faces, e, n0, b.topo_tri_offset[topo], b.env_node_offset[e], node);
    else refit_inner_global(b, b.env_node_offset[e], node, left);
}

// The fused refit of up to two envs an SM runs in two launches (see refit_fused for the others):
// every leaf of every env (or listed env) at once, one thread a node, then the inner nodes of an
// env by one block.  (One block that did an env's leaves and levels in turn waited for global
// memory some five times a level: 1 and 64 envs of 1,791 nodes 27 and 31 us, of 8,919 81 and 94;
// the two launches take 19 and 21, 50 and 61.)
__global__ void __launch_bounds__(256) k_refit_leaves(ffsrl_bvh b, const float* __restrict__ pts,
                                                      const int* __restrict__ faces, const int* __restrict__ ids,
                                                      int chunks) {
    const int k = blockIdx.x / chunks, e = ids ? ids[k] : k;
    if (e < 0 || e >= b.num_envs) return;
    const int topo = b.env_topology[e], n0 = b.topo_node_offset[topo];
    const int nn = b.topo_node_offset[topo + 1] - n0, t0 = b.topo_tri_offset[topo], base = b.env_node_offset[e];
    for (int node = (blockIdx.x % chunks) * blockDim.x + threadIdx.x; node < nn; node += chunks * blockDim.x)
        if (b.left_node[n0 + node] < 0) refit_leaf(b, pts, faces, e, n0, t0, base, node);
}

// Shared memory of the climb: per node its left child and its parent (2 bytes each), per inner
// node its box (24 bytes) and a bit for the first child to arrive
__host__ __device__ inline size_t climb_bytes(int nn) {
    return 24 * (size_t)(nn / 2 + 1) + 4 * (size_t)(nn / 64 + 1) + 4 * (size_t)nn;
}

// Inner nodes of one env per block.  The build numbers the two children of a node 2s + 1 and
// 2s + 2, so pair s stands for an inner node.  A thread takes a pair: two leaves make their
// parent's box at once, a leaf beside an inner node hands its box over, two inner nodes are
// left to others; a thread with a box climbs on for as long as it is the second of a node's
// two children to arrive.  The climb stays in shared memory (a level costs an atomic there
// instead of a barrier and trips to L2), reads the leaves' boxes coalesced and one pair
// ahead, and leaves what goes to global memory to a last pass over all pairs.  The same box
// whichever child comes second: the left child's box is always the first operand.  An env
// whose tree is numbered in another way or does not fit the block's shared memory is refitted
// level by level from global memory.  LEAVES: the block does its env's leaves first.
template <bool LEAVES>
__global__ void __launch_bounds__(LEAVES ? 256 : 1024) k_refit_climb(ffsrl_bvh b, const float* __restrict__ pts,
                                                                     const int* __restrict__ faces, const int* __restrict__ ids,
                                                                     int smem_bytes) {
    extern __shared__ float climb_smem[];
    __shared__ int s_bad;
    const int e = ids ? ids[blockIdx.x] : blockIdx.x;
    if (e < 0 || e >= b.num_envs) return;
    const int topo = b.env_topology[e], n0 = b.topo_node_offset[topo];
    const int nn = b.topo_node_offset[topo + 1] - n0, base = b.env_node_offset[e], step = blockDim.x;
    constexpr unsigned short kNone = 0xffffu;
    float* box = climb_smem;                                              // box[6 s]: the node whose children are pair s
    unsigned* arrived = reinterpret_cast<unsigned*>(box + 6 * (nn / 2 + 1));  // bit s
    unsigned short* left = reinterpret_cast<unsigned short*>(arrived + nn / 64 + 1);  // kNone: a leaf
    unsigned short* parent = left + nn;
    const bool fits = nn < 65535 && (nn & 1) && climb_bytes(nn) <= (size_t)smem_bytes;
    if (LEAVES) {
        for (int node = threadIdx.x; node < nn; node += step)
            if (b.left_node[n0 + node] < 0) refit_leaf(b, pts, faces, e, n0, b.topo_tri_offset[topo], base, node);
        __syncthreads();
    }
    if (fits) {
        if (threadIdx.x == 0) s_bad = 0;
        for (int i = threadIdx.x; i < nn; i += step) parent[i] = kNone;
        for (int i = threadIdx.x; i < nn / 64 + 1; i += step) arrived[i] = 0u;
        __syncthreads();
        for (int i0 = threadIdx.x; i0 < nn; i0 += 4 * step) {
            int l[4];  // four loads in flight
            for (int k = 0; k < 4; ++k) l[k] = i0 + k * step < nn ? b.left_node[n0 + i0 + k * step] : -1;
            for (int k = 0; k < 4; ++k) {
                const int i = i0 + k * step;
                if (i >= nn) break;
                left[i] = l[k] < 0 ? kNone : (unsigned short)l[k];
                if (l[k] < 0) continue;
                if (!(l[k] & 1) || l[k] + 1 >= nn || i >= l[k]) s_bad = 1;
                else parent[l[k]] = parent[l[k] + 1] = (unsigned short)i;
            }
        }
        __syncthreads();
        // a tree: every pair has a parent, and the one that names it
        for (int s = threadIdx.x; s < nn / 2; s += step) {
            const unsigned short p = parent[2 * s + 1];
            if (p == kNone || left[p] != 2 * s + 1) s_bad = 1;
        }
        for (int i = threadIdx.x; i < nn; i += step)  // no two nodes with the same children
            if (left[i] != kNone && !s_bad && parent[left[i]] != i) s_bad = 1;
        __syncthreads();
    }
    if (fits && !s_bad) {
        struct Pair { v3 l0, h0, l1, h1; };
        auto load_pair = [&](int s) {  // (of an inner child nothing is used)
            Pair q;
            const long long g = base + 2ll * s + 1;
            q.l0 = ld3(b.aabb_min, g); q.l1 = ld3(b.aabb_min, g + 1);
            q.h0 = ld3(b.aabb_max, g); q.h1 = ld3(b.aabb_max, g + 1);
            return q;
        };
        auto get = [&](int s, v3& lo, v3& hi) {
            const volatile float* q = box + 6 * s;
            lo = mk(q[0], q[1], q[2]);
            hi = mk(q[3], q[4], q[5]);
        };
        auto put = [&](int s, v3 lo, v3 hi) {
            volatile float* q = box + 6 * s;
            q[0] = lo.x; q[1] = lo.y; q[2] = lo.z; q[3] = hi.x; q[4] = hi.y; q[5] = hi.z;
        };
        const int pairs = nn / 2;
        Pair nx;
        if ((int)threadIdx.x < pairs) nx = load_pair(threadIdx.x);
        for (int s0 = threadIdx.x; s0 < pairs; s0 += step) {
            const Pair q = nx;
            if (s0 + step < pairs) nx = load_pair(s0 + step);
            const bool leaf0 = left[2 * s0 + 1] == kNone, leaf1 = left[2 * s0 + 2] == kNone;
            if (!leaf0 && !leaf1) continue;
            int s = s0;         // the pair this thread's box belongs to
            bool right = !leaf0;  // ... and which of the two it is
            v3 lo = leaf0 ? q.l0 : q.l1, hi = leaf0 ? q.h0 : q.h1;
            bool done = leaf0 && leaf1;  // the pair's node has both its boxes
            if (done) {
                lo = vmin(q.l0, q.l1);
                hi = vmax(q.h0, q.h1);
            } else {
                put(s, lo, hi);  // a leaf's box waits in its parent's place
            }
            for (;;) {
                if (!done) {
                    const unsigned bit = 1u << (s & 31);
                    __threadfence_block();
                    if (!(atomicOr(arrived + (s >> 5), bit) & bit)) break;
                    __threadfence_block();
                    const int sib = 2 * s + (right ? 1 : 2);
                    v3 sl, sh;
                    get(left[sib] == kNone ? s : left[sib] >> 1, sl, sh);
                    lo = right ? vmin(sl, lo) : vmin(lo, sl);
                    hi = right ? vmax(sh, hi) : vmax(hi, sh);
                }
                put(s, lo, hi);
                const int p = parent[2 * s + 1];  // the node this box is of
                if (p == 0) break;
                s = (p - 1) >> 1;
                right = !(p & 1);
                done = false;
            }
        }
        __syncthreads();
        if (threadIdx.x < pairs) nx = load_pair(threadIdx.x);
        for (int s = threadIdx.x; s < pairs; s += step) {
            Pair q = nx;
            if (s + step < pairs) nx = load_pair(s + step);
            if (left[2 * s + 1] != kNone) get(left[2 * s + 1] >> 1, q.l0, q.h0);
            if (left[2 * s + 2] != kNone) get(left[2 * s + 2] >> 1, q.l1, q.h1);
            v3 lo, hi;
            refit_inner(b, base, parent[2 * s + 1], 2 * s + 1, q.l0, q.h0, q.l1, q.h1, lo, hi);
        }
        return;
    }
    const int first = b.topo_level_offset[topo], groups = b.topo_max_level[topo] + 1;
    for (int g = 0; g < groups; ++g) {
        const int s0 = b.level_start[first + g], s1 = b.level_start[first + g + 1];
        for (int k = s0 + threadIdx.x; k < s1; k += blockDim.x) {
            const int node = b.level_node[k], left = b.left_node[n0 + node];
            if (left >= 0) refit_inner_global(b, base, node, left);
        }
        __syncthreads();
    }
}

// n envs (ids null: all).  What is fastest depends on their number and size (us; the climb after
// a launch of its own for the leaves, the climb with its leaves, the levels with their leaves):
//     nodes  envs: 1               64             216            512            1,024          2,048
//     383    14.0 11.1 12.7   15.0 12.5 12.8   16.8 14.3 14.9   23.0 17.2 18.7   33.4 29.2 32.7   51.8 46.9 48.7
//     1,791  18.9 27.6 23.6   21.0 30.9 27.1   31.6 35.5 32.7   57.9 52.4 45.6   112  105  105    211  177  167
//     4,325  30.0 60.9 47.7   35.5 66.1 51.2   62.5 81.1 65.5   134  186  114    244  299  241
//     8,919  50.3 116  84.6   60.5 123  92.8   154  181  149    320  374  248
// With few envs a small tree is a matter of one launch or two, a larger one of the trips to global
// memory; from two envs an SM on (at 300 of 2,557 nodes 45.7, 51.8 and 41.4, at 300 of 4,325 75, 95
// and 80) blocks hide one another's trips, and the levels' do the least work.
int32_t refit_fused(const ffsrl_bvh& b, const float* pts, const int32_t* faces, const int32_t* ids, int n, cudaStream_t s) {
    int dev = 0, sms = 0, most = 0;
    FFSRL_CUDA_TRY(cudaGetDevice(&dev));
    FFSRL_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    FFSRL_CUDA_TRY(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const int mean = b.total_env_nodes / b.num_envs;
    // up to an env per SM a block of the climb may have the SM's shared memory (trees to 14,300
    // nodes) and 1,024 threads; with more, two blocks share it (7,100 nodes)
    const bool few = n <= sms;
    const int limit = most - 1024 - 256, share = few ? limit : most / 2 - 1024 - 256;
    if (n > 2 * sms || (!few && climb_bytes(mean) > (size_t)share)) {
        k_refit_climb<true><<<n, 256, 0, s>>>(b, pts, faces, ids, 0);
        return FFSRL_OK;
    }
    // no tree has more nodes than all topologies together, but one of each other
    const int others = std::max(b.num_topologies, 1) - 1;
    const int largest = b.total_topology_nodes > others ? b.total_topology_nodes - others : INT_MAX;
    if (largest <= 512) {
        const int smem = (int)climb_bytes(largest);  // (8 KB: no limit to raise)
        k_refit_climb<true><<<n, 256, smem, s>>>(b, pts, faces, ids, smem);
        return FFSRL_OK;
    }
    const int chunks = std::max(1, std::min(mean / 256 + 1, 64));
    k_refit_leaves<<<(unsigned)((long long)chunks * n), 256, 0, s>>>(b, pts, faces, ids, chunks);
    const int smem = (int)std::min((size_t)share, climb_bytes(largest));
    // (always the largest: the attribute is the function's, whichever thread set it last)
    FFSRL_CUDA_TRY(cudaFuncSetAttribute(k_refit_climb<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit));
    const int threads = std::min(few ? 1024 : 512, std::max(128, (largest / 2 + 31) / 32 * 32));  // a pair each
    k_refit_climb<false><<<n, threads, smem, s>>>(b, pts, faces, ids, smem);
    return FFSRL_OK;
}

__global__ void k_zero3(float* p, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) st3(p, i, mk(0.0f, 0.0f, 0.0f));
}

// vertex_normal_sum_kernel (render.py:81-105)
__global__ void k_normal_sum(const float* __restrict__ pts, const int* __restrict__ faces, float* nsum, int nf) {
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nf) return;
    int i = faces[3 * f], j = faces[3 * f + 1], k = faces[3 * f + 2];
    v3 a = ld3(pts, i), b = ld3(pts, j), c = ld3(pts, k);
    v3 an = cross(b - a, c - a);
    atomic_add3(nsum, i, an); atomic_add3(nsum, j, an); atomic_add3(nsum, k, an);
}

// normalize_kernel (render.py:113-121)
__global__ void k_normalize(const float* __restrict__ nsum, float* __restrict__ nrm, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) st3(nrm, i, normalize(ld3(nsum, i)));
}

// Area-weighted normals gathered per point in ascending face order (deterministic; the
// same order as a serial run of vertex_normal_sum_kernel), then normalised.
__global__ void k_normal_gather(const float* __restrict__ pts, const int* __restrict__ faces,
                                const int* __restrict__ start, const int* __restrict__ pf, float* __restrict__ nrm,
                                int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    v3 s = mk(0.0f, 0.0f, 0.0f);
    for (int k = start[i]; k < start[i + 1]; ++k) {
        long long f = pf[k];
        v3 a = ld3(pts, faces[3 * f]), b = ld3(pts, faces[3 * f + 1]), c = ld3(pts, faces[3 * f + 2]);
        s = s + cross(b - a, c - a);
    }
    st3(nrm, i, normalize(s));
}

// the same gather for the points of one listed env per block
__global__ void k_normal_gather_envs(const float* __restrict__ pts, const int* __restrict__ faces,
                                     const int* __restrict__ start, const int* __restrict__ pf, float* __restrict__ nrm,
                                     const int* __restrict__ pstart, const int* __restrict__ ids, int num_envs) {
    int e = ids[blockIdx.x];
    if (e < 0 || e >= num_envs) return;
    for (int i = pstart[e] + threadIdx.x; i < pstart[e + 1]; i += blockDim.x) {
        v3 s = mk(0.0f, 0.0f, 0.0f);
        for (int k = start[i]; k < start[i + 1]; ++k) {
            long long f = pf[k];
            v3 a = ld3(pts, faces[3 * f]), b = ld3(pts, faces[3 * f + 1]), c = ld3(pts, faces[3 * f + 2]);
            s = s + cross(b - a, c - a);
        }
        st3(nrm, i, normalize(s));
    }
}

__device__ __forceinline__ v3 quat_rotate(float4 q, v3 x) {
    v3 u = mk(q.x, q.y, q.z);
    float c = 2.0f * q.w * q.w - 1.0f;
    float d = 2.0f * (u.x * x.x + u.y * x.y + u.z * x.z);
    return x * c + u * d + cross(u, x) * (q.w * 2.0f);
}

// intersectAABB (render.py:588-609)
__device__ __forceinline__ bool slab(v3 ro, v3 rd, v3 lo, v3 hi, float& tnear) {
    float t1 = (lo.x - ro.x) / rd.x, t2 = (hi.x - ro.x) / rd.x;
    float t3 = (lo.y - ro.y) / rd.y, t4 = (hi.y - ro.y) / rd.y;
    float t5 = (lo.z - ro.z) / rd.z, t6 = (hi.z - ro.z) / rd.z;
    float tmin = fmax_ref(fmax_ref(fmin_ref(t1, t2), fmin_ref(t3, t4)), fmin_ref(t5, t6));
    float tmax = fmin_ref(fmin_ref(fmax_ref(t1, t2), fmax_ref(t3, t4)), fmax_ref(t5, t6));
    tnear = tmin;
    return (tmax >= 0.0f) && (tmax >= tmin);
}

// Node test of the traversal: intersectAABB's hit && tmin < tMin (render.py:452-454).
// The slab distances are first formed as fma(lo, inv, -ro inv) with the ray's reciprocal
// direction inv and the per-ray products ro inv.  Against the reference's
// (lo - ro) / rd each differs by at most 4.01 u |t| + 1.02 u |ro inv| (u = 2^-24: the
// reciprocal, the product ro inv and the fma each round once; the reference rounds the
// difference and the quotient).  When every part of the decision is farther from its
// threshold than that -- g = 8 u m + 4 u R below, m the sum of the six |t|, R the sum
// of the three |ro inv| -- the decision equals the reference's.  Otherwise, and for
// non-finite distances, the reference's divisions decide.
struct RaySlab {
    v3 inv;    // 1 / rd per axis
    v3 roinv;  // ro * inv per axis
    float g0;  // 4 u (|ro inv|.x + .y + .z)
};

__device__ __forceinline__ RaySlab ray_slab(v3 ro, v3 rd) {
    RaySlab r;
    r.inv = mk(1.0f / rd.x, 1.0f / rd.y, 1.0f / rd.z);
    r.roinv = mk(ro.x * r.inv.x, ro.y * r.inv.y, ro.z * r.inv.z);
    r.g0 = 2.38418579e-7f * ((fabsf(r.roinv.x) + fabsf(r.roinv.y)) + fabsf(r.roinv.z));  // 4 * 2^-24
    return r;
}

__device__ __forceinline__ bool node_hit(v3 ro, v3 rd, const RaySlab& rs, v3 lo, v3 hi, float tMin) {
    float t1 = fmaf(lo.x, rs.inv.x, -rs.roinv.x), t2 = fmaf(hi.x, rs.inv.x, -rs.roinv.x);
    float t3 = fmaf(lo.y, rs.inv.y, -rs.roinv.y), t4 = fmaf(hi.y, rs.inv.y, -rs.roinv.y);
    float t5 = fmaf(lo.z, rs.inv.z, -rs.roinv.z), t6 = fmaf(hi.z, rs.inv.z, -rs.roinv.z);
    // the sum of magnitudes bounds every distance and is infinite or NaN when any of them
    // is (or when the per-ray products are), so the fast path only sees finite values,
    // where fminf/fmaxf pick what the reference's comparisons pick (up to the sign of a
    // zero, which no test below sees)
    float m = ((fabsf(t1) + fabsf(t2)) + (fabsf(t3) + fabsf(t4))) + (fabsf(t5) + fabsf(t6));
    if (m < 3.0e37f && rs.g0 < 3.0e37f) {
        float tmin = fmaxf(fmaxf(fminf(t1, t2), fminf(t3, t4)), fminf(t5, t6));
        float tmax = fminf(fminf(fmaxf(t1, t2), fmaxf(t3, t4)), fmaxf(t5, t6));
        float g = fmaf(m, 4.76837158e-7f, rs.g0);  // 8 u m + 4 u R
        // a certainly-false part decides a miss; all parts certainly true decide a hit
        if (tmax < -g || tmax - tmin < -2.0f * g || tmin > tMin + g) return false;
        if (tmax > g && tmax - tmin > 2.0f * g && tmin < tMin - g) return true;
    }
    float tn;
    bool h = slab(ro, rd, lo, hi, tn);
    return h && tn < tMin;
}

// MTTriRayIntersection (render.py:661-697)
__device__ __forceinline__ float moller_trumbore(v3 a, v3 b, v3 c, v3 ro, v3 rd, v3& p) {
    v3 ab = b - a, ac = c - a;
    v3 pvec = cross(rd, ac);
    float det = dot(ab, pvec);
    if (fabsf(det) < 0.0001f) return -1.0f;
    float invDet = 1.0f / det;
    v3 tvec = ro - a;
    float u = dot(tvec, pvec) * invDet;
    if (u < 0.0f || u > 1.0f) return -1.0f;
    v3 qvec = cross(tvec, ab);
    float v = dot(rd, qvec) * invDet;
    if (v < 0.0f || u + v > 1.0f) return -1.0f;
    float t = dot(ac, qvec) * invDet;
    p = ro + t * rd;
    return t;
}

struct EnvView {
    const int* left; const int* first; const int* count; const int* tri;
    const float* amin; const float* amax;
    const float4* box;   // packed node boxes of the env (or null)
    const float4* tpos;  // leaf triangles of the env in tri-map order, 3 float4 each (or null)
    long long fofs;
    int nn;  // nodes in the topology
};

__device__ __forceinline__ EnvView env_view(const ffsrl_bvh& b, int e) {
    int topo = b.env_topology[e];
    EnvView v;
    int n0 = b.topo_node_offset[topo];
    v.left = b.left_node + n0; v.first = b.first_tri_id + n0; v.count = b.tri_count + n0;
    v.tri = b.tri_id + b.topo_tri_offset[topo];
    long long base = b.env_node_offset[e];
    v.amin = b.aabb_min + 3 * base; v.amax = b.aabb_max + 3 * base;
    v.fofs = b.env_face_offset[e];
    v.nn = b.topo_node_offset[topo + 1] - n0;
    v.box = b.node_box ? reinterpret_cast<const float4*>(b.node_box) + 2 * base : nullptr;
    v.tpos = b.tri_pos ? reinterpret_cast<const float4*>(b.tri_pos) + 3 * v.fofs : nullptr;
    return v;
}

// meshQueryRayManyEnvs (render.py:411-498) over the packed copies written by the refit
// (two 16-byte loads per node, contiguous leaf triangles), visiting the nearer child
// first: the refit stores per inner node the axis along which its children's centres lie
// farthest apart, and the ray's sign along it picks the order.  The result is the
// reference's hit.  The reference visits nodes in a fixed pre-order (right child first),
// prunes a node whose box entry is not nearer than the best hit so far, and keeps the
// first of equally near hits.  Its pre-order visits leaves in descending tri-map position
// (the build puts a node's left child's triangles first) and a leaf's triangles in
// ascending order.  So here a hit is kept when it is nearer, or equally near and earlier
// in that order.  With the same strict pruning, the triangle the reference keeps is never
// pruned, whatever the visiting order: its boxes are entered before it is reached.
// Returns the global face id or -1.
__device__ int query_packed(const EnvView& ev, v3 ro, v3 rd, float& t_hit, v3& p_hit, int* err) {
    int stack[kStackCap];
    int count = 1;
    stack[0] = 0;
    float tMin = 1e6f;
    int hit_tri = -1;
    int best_first = -1, best_k = 0;  // the kept hit's leaf and place in it
    int visits = 0;
    const RaySlab rs = ray_slab(ro, rd);
    while (count) {
        int node = stack[--count];
        if (++visits > ev.nn) {
            atomicExch(err, FFSRL_ERR_STACK_OVERFLOW);
            return -1;
        }
        const float4 a = __ldg(ev.box + 2 * node), c = __ldg(ev.box + 2 * node + 1);
        if (node_hit(ro, rd, rs, mk(a.x, a.y, a.z), mk(c.x, c.y, c.z), tMin)) {
            int left = __float_as_int(a.w);
            if (left == -1) {
                int fc = __float_as_int(c.w);
                int first = fc >> 8, cnt = fc & 255;
                if (cnt == 255) cnt = ev.count[node];
                for (int k = 0; k < cnt; ++k) {
                    const float4* q = ev.tpos + 3ll * (first + k);
                    const float4 q0 = __ldg(q), q1 = __ldg(q + 1), q2 = __ldg(q + 2);
                    v3 A = mk(q0.x, q0.y, q0.z);
                    v3 B = mk(q0.w, q1.x, q1.y);
                    v3 C = mk(q1.z, q1.w, q2.x);
                    v3 p;
                    float t = moller_trumbore(A, B, C, ro, rd, p);
                    if (t > 0.0f && (t < tMin || (t == tMin && hit_tri >= 0 &&
                                                  (first > best_first || (first == best_first && k < best_k))))) {
                        tMin = t;
                        hit_tri = (int)(ev.fofs + ev.tri[first + k]);
                        best_first = first;
                        best_k = k;
                        t_hit = t;
                        p_hit = p;
                    }
                }
            } else {
                if (left < 0 || left + 1 >= ev.nn) {
                    atomicExch(err, FFSRL_ERR_INVALID_ARGUMENT);
                    return -1;
                }
                if (count + 2 > kStackCap) {
                    atomicExch(err, FFSRL_ERR_STACK_OVERFLOW);
                    return -1;
                }
                const int code = __float_as_int(c.w);
                const int axis = code & 3;
                const float da = axis == 0 ? rd.x : (axis == 1 ? rd.y : rd.z);
                // nearer child: the left one when the ray runs towards the right child's side
                const bool left_near = (da > 0.0f) == ((code & 4) != 0);
                stack[count] = left_near ? left + 1 : left;
                stack[count + 1] = left_near ? left : left + 1;
                count += 2;
            }
        }
    }
    if (tMin >= 1e6f) hit_tri = -1;
    return hit_tri;
}

__device__ int query(const EnvView& ev, const float* __restrict__ pts, const int* __restrict__ faces, v3 ro, v3 rd,
                     float& t_hit, v3& p_hit, int* err) {
    if (ev.box && ev.tpos) return query_packed(ev, ro, rd, t_hit, p_hit, err);
    int stack[kStackCap];
    int count = 1;
    stack[0] = 0;
    float tMin = 1e6f;
    int hit_tri = -1;
    int visits = 0;
    const RaySlab rs = ray_slab(ro, rd);
    while (count) {
        int node = stack[--count];
        if (++visits > ev.nn) {  // a valid tree visits each node at most once
            atomicExch(err, FFSRL_ERR_STACK_OVERFLOW);
            return -1;
        }
        if (node_hit(ro, rd, rs, ld3(ev.amin, node), ld3(ev.amax, node), tMin)) {
            int left = ev.left[node];
            if (left == -1) {
                int first = ev.first[node];
                int cnt = ev.count[node];
                for (int k = 0; k < cnt; ++k) {
                    long long f = ev.fofs + ev.tri[first + k];
                    v3 A = ld3(pts, faces[3 * f]), B = ld3(pts, faces[3 * f + 1]), C = ld3(pts, faces[3 * f + 2]);
                    v3 p;
                    float t = moller_trumbore(A, B, C, ro, rd, p);
                    if (t < tMin && t > 0.0f) {
                        tMin = t;
                        hit_tri = (int)f; t_hit = t; p_hit = p;
                    }
                }
            } else {
                if (left < 0 || left + 1 >= ev.nn) {
                    atomicExch(err, FFSRL_ERR_INVALID_ARGUMENT);
                    return -1;
                }
                if (count + 2 > kStackCap) {
                    atomicExch(err, FFSRL_ERR_STACK_OVERFLOW);
                    return -1;
                }
                stack[count] = left;
                stack[count + 1] = left + 1;
                count += 2;
            }
        }
    }
    if (tMin >= 1e6f) hit_tri = -1;
    return hit_tri;
}

struct Shade { v3 color; float depth; };

// shading of drawSimBVHKernelManyEnvs (render.py:334-409): modes 0 grayscale, 1 texture,
// 2 normal map, 3 vertex colour, 4 depth map into `color`; `depth` gets t/50 in every mode
// The object of env e that holds env-local face lf (render.py:360-366: visFaceToObjectId,
// objectUsesTexture, objectNumVisFaceCummulative): its 5-int entry in object_texture.
__device__ __forceinline__ const int* face_object(const ffsrl_render& r, int e, int lf) {
    const int o0 = r.env_objects[2ll * e], no = r.env_objects[2ll * e + 1];
    const int* ob = r.object_texture + 5ll * o0;
    for (int k = 1; k < no; ++k) {
        if (r.object_texture[5ll * (o0 + k)] > lf) break;
        ob = r.object_texture + 5ll * (o0 + k);
    }
    return ob;
}

// texture_interpolation (render.py:123-148): bilinear texel of the interpolated tex
// coordinate; texel (x, y) of a texture at first + y + x*S.  Indices are clamped into the
// texture (the reference reads one texel past the edge at coordinate 1, weighted 0).
__device__ __forceinline__ v3 texel(const ffsrl_render& r, const int* ob, int lf, float u, float v, float w) {
    const int first = ob[1], S = ob[2], c0 = ob[3];
    const int* ti = r.tex_indices + ob[4] + 3ll * (lf - ob[0]);
    const float* ta = r.tex_coords + 2ll * (c0 + ti[0]);
    const float* tb = r.tex_coords + 2ll * (c0 + ti[1]);
    const float* tc = r.tex_coords + 2ll * (c0 + ti[2]);
    float tx = (u * ta[0] + v * tb[0]) + w * tc[0];
    float ty = (u * ta[1] + v * tb[1]) + w * tc[1];
    float fx = tx * float(S - 1), fy = (1.0f - ty) * float(S - 1);
    int x0 = (int)fx, y0 = (int)fy;
    float ax = fx - float(x0), ay = fy - float(y0);
    int x1 = x0 + 1, y1 = y0 + 1;
    x0 = min(max(x0, 0), S - 1); x1 = min(max(x1, 0), S - 1);
    y0 = min(max(y0, 0), S - 1); y1 = min(max(y1, 0), S - 1);
    v3 c00 = ld3(r.texture, (long long)first + y0 + x0 * S), c10 = ld3(r.texture, (long long)first + y0 + x1 * S);
    v3 c01 = ld3(r.texture, (long long)first + y1 + x0 * S), c11 = ld3(r.texture, (long long)first + y1 + x1 * S);
    v3 lower = (1.0f - ax) * c00 + ax * c10;
    v3 upper = (1.0f - ax) * c01 + ax * c11;
    return (1.0f - ay) * lower + ay * upper;
}

__device__ __forceinline__ v3 ray_dir(const ffsrl_render& r, float4 q, int x, int y, int W, int H) {
    float sx = 2.0f * float(x) / float(W) - 1.0f;
    float sy = 2.0f * float(y) / float(H) - 1.0f;
    return normalize(quat_rotate(q, mk(sx * r.camera_tan * r.camera_aspect, sy * r.camera_tan, -1.0f)));
}

// colour and depth of a ray's hit: global face `tri` (-1: none) at distance t, point p
__device__ __forceinline__ Shade shade(const ffsrl_render& r, const EnvView& ev, int e, int tri, float t, v3 p) {
    Shade s;
    s.color = mk(0.0f, 0.0f, 0.0f);
    s.depth = 0.0f;
    if (tri > -1) {
        int i = r.vis_face[3ll * tri], j = r.vis_face[3ll * tri + 1], k = r.vis_face[3ll * tri + 2];
        v3 a = ld3(r.vis_point, i), b = ld3(r.vis_point, j), c = ld3(r.vis_point, k);
        float area = length(cross(b - a, c - a));
        float w = length(cross(b - a, p - a)) / area;
        float v = length(cross(p - a, c - a)) / area;
        float u = 1.0f - w - v;
        v3 n = u * ld3(r.vertex_normal, i) + v * ld3(r.vertex_normal, j) + w * ld3(r.vertex_normal, k);
        v3 col;
        if (r.render_mode == 2) {  // normal map
            col = n * 0.5f + mk(0.5f, 0.5f, 0.5f);
        } else if (r.render_mode == 4) {  // depth map
            float g = t / 50.0f;
            col = mk(g, g, g);
        } else {
            v3 base;
            if (r.render_mode == 0)
                base = mk(1.0f, 1.0f, 1.0f);
            else {
                const int lf = (int)(tri - ev.fofs);
                const int* ob = (r.render_mode == 1 && r.env_objects) ? face_object(r, e, lf) : nullptr;
                if (ob && ob[2] > 0)
                    base = texel(r, ob, lf, u, v, w);
                else
                    base = (ld3(r.vis_point_color, i) + ld3(r.vis_point_color, j) + ld3(r.vis_point_color, k)) / 3.0f;
            }
            float lam = 0.0f;
            for (int l = 0; l < r.num_lights; ++l) {
                float val = r.light_intensity[l] * dot(n, ld3(r.light_dir, l));
                if (val < 0.0f) val = 0.0f;
                lam = lam + val;
            }
            col = lam * base;
        }
        if (col.x > 1.0f) col.x = 1.0f;
        if (col.y > 1.0f) col.y = 1.0f;
        if (col.z > 1.0f) col.z = 1.0f;
        s.color = col;
        float d = t / 50.0f;
        if (d > 1.0f) d = 1.0f;
        s.depth = d;
    }
    return s;
}

__device__ __forceinline__ Shade trace(const ffsrl_render& r, const EnvView& ev, int e, v3 ro, float4 q, int x, int y,
                                       int W, int H) {
    const v3 rd = ray_dir(r, q, x, y, W, H);
    float t = 0.0f;
    v3 p = mk(0.0f, 0.0f, 0.0f);
    const int tri = query(ev, r.vis_point, r.vis_face, ro, rd, t, p, r.error_flag);
    return shade(r, ev, e, tri, t, p);
}

// drawSimBVHKernelManyEnvs (render.py:276-409): one thread per ray, into scratch
__global__ void k_draw(ffsrl_render r, ffsrl_bvh b) {
    const int W = 2 * r.resolution, H = 2 * r.resolution;
    long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (tid >= (long long)W * H * r.num_envs) return;
    int e = (int)(tid / (W * H));
    int et = (int)(tid % (W * H));
    int x = et % W;
    int y = H - et / W;
    int cam = r.num_cameras > 1 ? e : 0;
    v3 ro = ld3(r.camera_pos, cam);
    float4 q = reinterpret_cast<const float4*>(r.camera_rot)[cam];
    EnvView ev = env_view(b, e);
    Shade s = trace(r, ev, e, ro, q, x, y, W, H);
    st3(r.rays, tid, s.color);
    r.ray_depth[tid] = s.depth;
}

// downsample_kernel (render.py:699-724), 2x2 rays per pixel
__global__ void k_downsample(ffsrl_render r) {
    const int R = r.resolution, W = 2 * R;
    long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (tid >= (long long)R * R * r.num_envs) return;
    long long px = tid % R, py = tid / R;
    long long start = py * 2 * W + px * 2;
    v3 c = mk(0.0f, 0.0f, 0.0f);
    float d = 0.0f;
    for (int i = 0; i < 2; ++i)
        for (int j = 0; j < 2; ++j) {
            v3 s = ld3(r.rays, start + i * W + j);
            c = mk(c.x + s.x, c.y + s.y, c.z + s.z);
            d = d + r.ray_depth[start + i * W + j];
        }
    float nsq = float(2 * 2);
    if (r.color) st3(r.color, tid, mk(c.x / nsq, c.y / nsq, c.z / nsq));
    if (r.depth) r.depth[tid] = d / nsq;
}

// The four rays of a pixel sit in consecutive lanes: summed by shuffles in
// downsample_kernel's order ((r00 + r01) + r10) + r11, then divided by 4.
__device__ __forceinline__ void store_pixel(const ffsrl_render& r, const Shade& s, bool valid, int e, int px, int py) {
    const int R = r.resolution, q = threadIdx.x & 3;
    float cx = s.color.x, cy = s.color.y, cz = s.color.z, d = s.depth;
    float ax[3], ay[3], az[3], ad[3];
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
        ax[k - 1] = __shfl_down_sync(0xffffffffu, cx, k);
        ay[k - 1] = __shfl_down_sync(0xffffffffu, cy, k);
        az[k - 1] = __shfl_down_sync(0xffffffffu, cz, k);
        ad[k - 1] = __shfl_down_sync(0xffffffffu, d, k);
    }
    if (valid && q == 0) {
        v3 c = mk(cx, cy, cz);
        for (int k = 0; k < 3; ++k) c = mk(c.x + ax[k], c.y + ay[k], c.z + az[k]);
        float dd = ((d + ad[0]) + ad[1]) + ad[2];
        float nsq = float(2 * 2);
        long long o = (long long)e * R * R + (long long)py * R + px;
        if (r.color) st3(r.color, o, mk(c.x / nsq, c.y / nsq, c.z / nsq));
        if (r.depth) r.depth[o] = dd / nsq;
    }
}

// ---- bundles of rays -----------------------------------------------------------------
// Ray directions (not normalised) as d0 + x dx + y dy over the ray indices
struct Camera { v3 d0, dx, dy; };
__device__ __forceinline__ Camera make_camera(const ffsrl_render& r, float4 q, int W, int H) {
    const float tx = r.camera_tan * r.camera_aspect, ty = r.camera_tan;
    Camera c;
    c.d0 = quat_rotate(q, mk(-tx, -ty, -1.0f));
    c.dx = quat_rotate(q, mk(2.0f * tx / float(W), 0.0f, 0.0f));
    c.dy = quat_rotate(q, mk(0.0f, 2.0f * ty / float(H), 0.0f));
    return c;
}
// The rays of a rectangle of w x h pixels from pixel (px, py), as ranges of the ray indices
// widened by a quarter of the ray spacing on each side
struct Range { float x0, x1, y0, y1; };
__device__ __forceinline__ Range ray_range(int px, int py, int w, int h, int H) {
    return {2.0f * px - 0.25f, 2.0f * (px + w) - 0.75f, H - (2.0f * (py + h) - 0.75f), H - (2.0f * py - 0.25f)};
}
// The four corners of the rectangle: every ray of it lies between them, to within the rounding
// of a direction (some 1e-6 of it; of the outermost corner through very wide lenses)
struct Corners { v3 d[4]; };
__device__ __forceinline__ Corners make_corners(const Camera& c, int px, int py, int w, int h, int H) {
    const Range g = ray_range(px, py, w, h, H);
    const v3 a = c.d0 + g.x0 * c.dx, b = c.d0 + g.x1 * c.dx;
    Corners k;
    k.d[0] = a + g.y0 * c.dy; k.d[1] = b + g.y0 * c.dy; k.d[2] = b + g.y1 * c.dy; k.d[3] = a + g.y1 * c.dy;
    return k;
}
// The camera's axes, z into the picture: what quat_rotate makes of (1, 0, 0), (0, 1, 0) and
// (0, 0, -1)
struct Axes { v3 x, y, z; };
__device__ __forceinline__ Axes make_axes(float4 q) {
    const float c = 2.0f * q.w * q.w - 1.0f;
    Axes a;
    a.x = mk(c + 2.0f * q.x * q.x, 2.0f * (q.x * q.y + q.w * q.z), 2.0f * (q.x * q.z - q.w * q.y));
    a.y = mk(2.0f * (q.x * q.y - q.w * q.z), c + 2.0f * q.y * q.y, 2.0f * (q.y * q.z + q.w * q.x));
    a.z = mk(-2.0f * (q.x * q.z + q.w * q.y), -2.0f * (q.y * q.z - q.w * q.x), -(c + 2.0f * q.z * q.z));
    return a;
}
__device__ __forceinline__ float sum1(v3 a) { return fabsf(a.x) + fabsf(a.y) + fabsf(a.z); }
// A quaternion far from a unit one can make the axes shrink to rounding errors, or nearly
// parallel.  The margins here hold while their volume is not far below that of a rotation's.
__device__ __forceinline__ bool sound(const Axes& a, float4 q) {
    const float n = 1.0f + 2.0f * (q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w);
    return fabsf(dot(cross(a.x, a.y), a.z)) > 0.02f * n * n * n;
}
// The planes through the camera along a rectangle's sides, normals inward.  A side's normal is
// the product of a direction on it and the camera's axis along it, z + e x and y, or z + e y and
// x: perpendicular vectors, whereas two corners of a tile are nearly parallel behind a narrow
// lens, and the rounding of their product then moves the plane by more than any margin (tiles of
// 8 at 1,024 pixels: through a 5 degree lens 6% of the points on their outermost rays lay outside
// their planes).  Rounding moves a normal by some 1e-6 of it, a ray's direction and the edges of a
// box that the slab test sees by less; outside() leaves a relative 4e-6.  (A normal that is not
// finite excludes nothing.)
struct Bundle { v3 n[4]; };
// side i: left, right, lower, upper
__device__ __forceinline__ v3 make_plane(const Axes& c, const Range& g, float tx, float ty, int W, int H, int i) {
    const bool across = i < 2;
    const float t = across ? tx : ty, per = __fdividef(2.0f * t, float(across ? W : H));
    const float e0 = per * (across ? g.x0 : g.y0) - t, e1 = per * (across ? g.x1 : g.y1) - t;
    const v3 xy = cross(c.x, c.y), u = cross(across ? c.z : c.x, across ? c.y : c.z);
    const v3 n = u + (i & 1 ? fmaxf(e0, e1) : fminf(e0, e1)) * xy;
    const float s = (dot(xy, c.z) < 0.0f) == !(i & 1) ? 1.0f : -1.0f;  // (a quaternion may make a mirror image)
    return n * __fdividef(s, sum1(n));
}

__device__ __forceinline__ float fdot(v3 a, v3 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, a.z * b.z)); }
__device__ __forceinline__ v3 fcross(v3 a, v3 b) {
    return mk(fmaf(a.y, b.z, -(a.z * b.y)), fmaf(a.z, b.x, -(a.x * b.z)), fmaf(a.x, b.y, -(a.y * b.x)));
}
// Whether a ray between the corners can pass the triangle test: its determinant and the
// numerators of u and v are linear in the direction, so where the determinant has one sign
// at all corners, and u, v or 1 - u - v the wrong one, by more than the test's own rounding
// (some 1e-6 of the vectors' lengths; 1e-5 here), no ray does.
__device__ __forceinline__ bool may_hit(const Corners& k, v3 ab, v3 ac, v3 tv, v3 qv) {
    const v3 N = fcross(ac, ab), U = fcross(ac, tv);
    float dlo = 3.4e38f, dhi = -3.4e38f, ulo = dlo, uhi = dhi, vlo = dlo, vhi = dhi, wlo = dlo, whi = dhi, len = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float d = fdot(k.d[i], N), u = fdot(k.d[i], U), v = fdot(k.d[i], qv), w = (d - u) - v;
        dlo = fminf(dlo, d); dhi = fmaxf(dhi, d);
        ulo = fminf(ulo, u); uhi = fmaxf(uhi, u);
        vlo = fminf(vlo, v); vhi = fmaxf(vhi, v);
        wlo = fminf(wlo, w); whi = fmaxf(whi, w);
        len = fmaxf(len, sum1(k.d[i]));
    }
    const float a = sum1(ab), c = sum1(ac), t = sum1(tv);
    const float gu = 1e-5f * len * t * c, gv = 1e-5f * len * t * a, gd = 1e-5f * len * a * c, gw = gu + gv + gd;
    if (dlo > gd) return !(uhi < -gu || vhi < -gv || whi < -gw);
    if (dhi < -gd) return !(ulo > gu || vlo > gv || wlo > gw);
    return true;
}

// whether the box [lo, hi], relative to the camera, lies outside one of the planes
__device__ __forceinline__ bool outside(const Bundle& b, v3 lo, v3 hi) {
    const v3 c = mk(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z));
    const v3 h = mk(0.5f * (hi.x - lo.x), 0.5f * (hi.y - lo.y), 0.5f * (hi.z - lo.z));
    const float g = 4e-6f * ((fabsf(c.x) + fabsf(c.y)) + (fabsf(c.z) + h.x) + (h.y + h.z));
    bool out = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const v3 n = b.n[k];
        float s = fmaf(fabsf(n.x), h.x, fmaf(fabsf(n.y), h.y, fmaf(fabsf(n.z), h.z, g)));
        s = fmaf(n.x, c.x, fmaf(n.y, c.y, fmaf(n.z, c.z, s)));
        out |= s < 0.0f;
    }
    return out;
}

// Ray-cast by tiles of T x T pixels, 256 threads each.  What a thread per ray spends its time
// on is the walk down the tree, which neighbouring rays share.  Here a block finds the leaves
// that its tile's rays can reach, all its threads testing a level of the tree at a time
// against the tile's bundle; it prepares their triangles in shared memory (what the triangle
// test computes from the camera and the triangle alone, the faces towards the camera first);
// then each warp takes patches of 4 x 2 pixels (32 rays), keeps the listed triangles its
// patch's rays can reach, a triangle a lane, and tests them one after another, all lanes the
// same triangle.  A tile of 16 with more triangles than the list holds is done in quarters.
// 256 envs of 500-20,000 tets at 128 x 128: a thread per ray takes 1,186 us and 1,900
// instructions a warp of 32 rays with two thirds of its lanes busy, the tiles 747; 8 textured
// envs at 512 x 512: 526 and 290 us.  What bounds it now is issue, 65% of it, and on one env
// the chain of loads, tests and shading of the patch with the most triangles (45 us with one
// warp a patch, 35 with two: launch_rays).
//
// The hit is the traversal's: of the triangles whose test succeeds, the nearest, the first
// in the reference's order among equals.  The traversal reaches a triangle if the ray's slab
// test enters its leaf's box (it then enters the boxes above, as rounding is monotone) and
// every hit before it is farther than that entry, so the nearest one's leaf is put to the slab
// test at the end.  In the rare case that the test fails, or puts the entry no nearer than another
// hit (two triangles hit in a box's corner, or at the same distance in a plane that bounds their
// boxes, where the one that is kept hangs on the order of the traversal), the ray is traversed.
// So is a ray along a coordinate plane, and every ray of an 8 x 8 tile that has too many triangles
// (quarters of those took up to 1.7 times as long) or one of extreme size, or of a tree deeper than
// kSteps levels below the ones tested first.
constexpr int kCand = 448;      // triangles of a tile, 64 bytes of shared memory each
constexpr int kFront = 768;     // nodes of a level
constexpr int kSteps = 40;
constexpr int kList = 160;      // triangles a warp keeps for its four patches
// Levels tested at once at the start.  Tiles of 16, which fill the GPU: at most 255 nodes, one a
// thread.  Tiles of 8, taken for less work, wait for each step more than for what it does: at most
// 2,047 nodes, eight a thread.
template <int T> struct FirstLevel { static constexpr int value = T == 16 ? 7 : 10; };

// The traversal of one ray, kept out of line: few rays take it
struct Hit { int tri; float t; v3 p; };
__device__ __noinline__ Hit traverse(const ffsrl_render* r, const ffsrl_bvh* b, int e, v3 ro, v3 rd) {
    Hit h;
    h.t = 0.0f;
    h.p = mk(0.0f, 0.0f, 0.0f);
    h.tri = query(env_view(*b, e), r->vis_point, r->vis_face, ro, rd, h.t, h.p, r->error_flag);
    return h;
}

template <int T, int HALVES>
__global__ void __launch_bounds__(256 * HALVES, 4 / HALVES) k_rays(const __grid_constant__ ffsrl_render r, const __grid_constant__ ffsrl_bvh b,
                                                 const int* __restrict__ ids, int n_ids) {
    __shared__ float4 s_tri[4 * kCand];  // (ab, ac, tvec, qvec, ac.qvec, leaf, place in the leaf, distance)
    __shared__ unsigned short s_list[T == 16 ? 8 : 1][kList];
    __shared__ int s_front[2][kFront];
    __shared__ int s_leaf[kCand];
    // the tile's planes; its middle ray and the longest ray's length, half its width and height
    __shared__ float4 s_plane[7];
    __shared__ int s_n[3], s_leaves, s_over, s_nf, s_nb;
    __shared__ int s_todo[4][2];  // quarters still to do: x, y
    __shared__ float s_hit[HALVES == 2 ? 8 : 1][3][HALVES == 2 ? 32 : 1];  // the second warp's rays: distance, second, triangle
    constexpr int kThreads = 256 * HALVES;
    const int R = r.resolution, W = 2 * R, H = 2 * R;
    const int tiles_x = (R + T - 1) / T, tiles = tiles_x * tiles_x;
    const int k = blockIdx.x / tiles;
    const int e = ids ? (k < n_ids ? ids[k] : r.num_envs) : k;
    if (e < 0 || e >= r.num_envs) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = HALVES == 2 ? (tid >> 5) & 7 : tid >> 5;
    const int part = HALVES == 2 ? tid >> 8 : 0;  // which of the patch's warps
    const int cam = r.num_cameras > 1 ? e : 0;
    const v3 ro = ld3(r.camera_pos, cam);
    const float4 qr = reinterpret_cast<const float4*>(r.camera_rot)[cam];
    const EnvView ev = env_view(b, e);
    const Camera cm = make_camera(r, qr, W, H);
    const bool packed = ev.box && ev.tpos;
    int todo = 0;  // tiles in s_todo, the same for every thread
    int tx = ((blockIdx.x % tiles) % tiles_x) * T, ty = ((blockIdx.x % tiles) / tiles_x) * T, size = T;
    for (;;) {
        if (tid < 3) s_n[tid] = 0;
        if (tid == 0) { s_leaves = 0; s_nf = 0; s_nb = 0; }
        if (tid < 4) {
            const Axes axes = make_axes(qr);
            const v3 n = make_plane(axes, ray_range(tx, ty, size, size, H), r.camera_tan * r.camera_aspect, r.camera_tan, W, H, tid);
            s_plane[tid] = make_float4(n.x, n.y, n.z, 0.0f);
            if (tid == 0) s_over = !sound(axes, qr);  // (then every ray is traversed)
        }
        if (tid == 32) {
            const Range g = ray_range(tx, ty, size, size, H);
            const v3 mid = cm.d0 + 0.5f * (g.x0 + g.x1) * cm.dx + 0.5f * (g.y0 + g.y1) * cm.dy;
            const v3 across = 0.5f * (g.x1 - g.x0) * cm.dx, up = 0.5f * (g.y1 - g.y0) * cm.dy;
            s_plane[4] = make_float4(mid.x, mid.y, mid.z, sum1(mid) + sum1(across) + sum1(up));
            s_plane[5] = make_float4(across.x, across.y, across.z, 0.0f);
            s_plane[6] = make_float4(up.x, up.y, up.z, 0.0f);
        }
        __syncthreads();
        if (packed) {
            auto plane = [&](int i) { return mk(s_plane[i].x, s_plane[i].y, s_plane[i].z); };
            Bundle F;
#pragma unroll
            for (int i = 0; i < 4; ++i) F.n[i] = plane(i);
            auto visit = [&](int node, int* count, int* front, bool expand) {
                if ((unsigned)node >= (unsigned)ev.nn) { s_over = 1; return; }
                if (*(volatile int*)&s_over) return;  // (the lists are given up: nothing more to find)
                const float4 a = __ldg(ev.box + 2 * node), c = __ldg(ev.box + 2 * node + 1);
                const int left = __float_as_int(a.w);
                if (left != -1 && !expand) return;
                if (outside(F, mk(a.x, a.y, a.z) - ro, mk(c.x, c.y, c.z) - ro)) return;
                if (left == -1) {
                    const int q = atomicAdd(&s_leaves, 1);
                    if (q < kCand) s_leaf[q] = node;
                    else s_over = 1;
                } else {
                    const int q = atomicAdd(count, 2);
                    if (left >= 0 && left + 1 < ev.nn && q + 1 < kFront) {
                        front[q] = left;
                        front[q + 1] = left + 1;
                    } else {
                        s_over = 1;
                    }
                }
            };
            // the nodes of the first level and the leaves above them, from the level lists (deepest
            // level first), or the root
            if (b.level_node && b.level_start && b.topo_level_offset) {
                const int topo = b.env_topology[e], lo = b.topo_level_offset[topo], deepest = b.topo_max_level[topo];
                const int g = max(0, deepest - FirstLevel<T>::value);
                const int s0 = b.level_start[lo + g], s1 = b.level_start[lo + g + 1], s2 = b.level_start[lo + deepest + 1];
                for (int i0 = s0 + tid; i0 < s2; i0 += 4 * kThreads) {
                    int node[4];  // four loads in flight
                    for (int m = 0; m < 4; ++m) node[m] = i0 + kThreads * m < s2 ? b.level_node[i0 + kThreads * m] : -1;
                    for (int m = 0; m < 4; ++m)
                        if (i0 + kThreads * m < s2) visit(node[m], &s_n[0], s_front[0], i0 + kThreads * m < s1);
                }
            } else if (tid == 0) {
                visit(0, &s_n[0], s_front[0], true);
            }
            __syncthreads();
            // step j takes the s_n[j % 3] nodes of s_front[j & 1]; every thread sees the same
            // count, as step j + 1 is the next to change it
            int step = 0;
            for (;; ++step) {
                const int n = min(s_n[step % 3], kFront);
                if (n == 0 || step == kSteps) break;
                if (tid == 0) s_n[(step + 2) % 3] = 0;
                for (int i = tid; i < n; i += kThreads)
                    visit(s_front[step & 1][i], &s_n[(step + 1) % 3], s_front[(step + 1) & 1], true);
                __syncthreads();
            }
            if (step == kSteps && tid == 0) s_over = 1;
            const int leaves = s_over ? 0 : s_leaves;
            for (int i = tid; i < leaves; i += kThreads) {
                const int node = s_leaf[i];
                const int fc = __float_as_int(__ldg(ev.box + 2 * node + 1).w), first = fc >> 8;
                int cnt = fc & 255;
                if (cnt == 255) cnt = ev.count[node];
                for (int m = 0; m < cnt; ++m) {
                    const float4* q = ev.tpos + 3ll * (first + m);
                    const float4 q0 = __ldg(q), q1 = __ldg(q + 1), q2 = __ldg(q + 2);
                    const v3 A = mk(q0.x, q0.y, q0.z);
                    const v3 ab = mk(q0.w, q1.x, q1.y) - A, ac = mk(q1.z, q1.w, q2.x) - A, tv = ro - A, qv = cross(tv, ab);
                    const float tn = dot(ac, qv);
                    const int at = tn > 0.0f ? atomicAdd(&s_nf, 1) : kCand - 1 - atomicAdd(&s_nb, 1);
                    if ((unsigned)at >= (unsigned)kCand) continue;  // too many: counted below
                    // No ray finds a hit of it nearer than its own box lies (its leaf's box may be
                    // another face's), less what rounding can do to a distance: some 32 units in
                    // the last place of |ab| |ac| (|tv| + |ab| + |ac|) over the determinant, which
                    // is 1e-4 at least, and much more where no ray of the tile grazes the triangle
                    const v3 lo = vmin(vmin(ab, ac), mk(0.0f, 0.0f, 0.0f)) - tv, hi = vmax(vmax(ab, ac), mk(0.0f, 0.0f, 0.0f)) - tv;
                    const v3 gap = mk(fmaxf(fmaxf(lo.x, -hi.x), 0.0f), fmaxf(fmaxf(lo.y, -hi.y), 0.0f), fmaxf(fmaxf(lo.z, -hi.z), 0.0f));
                    const v3 N = fcross(ac, ab), mid = plane(4), across = plane(5), up = plane(6);
                    const float len = s_plane[4].w, sab = sum1(ab), sac = sum1(ac), stv = sum1(tv);
                    // Beyond these sizes the tests below could overflow, or take for below zero what
                    // the triangle test rounds to -0 (and NaN is left to it)
                    if (!(sab * sac < 1e14f && stv * (sab + sac) < 1e30f)) s_over = 1;
                    const float det = fabsf(fdot(mid, N)) - fabsf(fdot(across, N)) - fabsf(fdot(up, N)) - 1e-5f * len * sab * sac;
                    const float off = __fdividef(2e-6f * sab * sac * (stv + sab + sac) * len, fmaxf(det, 1e-4f * len));
                    const float near = 0.9999f * length(gap) - off;
                    s_tri[4 * at] = make_float4(ab.x, ab.y, ab.z, ac.x);
                    s_tri[4 * at + 1] = make_float4(ac.y, ac.z, tv.x, tv.y);
                    s_tri[4 * at + 2] = make_float4(tv.z, qv.x, qv.y, qv.z);
                    s_tri[4 * at + 3] = make_float4(tn, __int_as_float(node), __int_as_float(m), near);
                }
            }
        }
        __syncthreads();
        int nf = s_nf, nb = s_nb;  // triangles facing the camera, and others
        const bool listed = packed && !s_over && nf + nb <= kCand;
        if (packed && !listed && size > 8) {
            // the quarters instead
            size = 8;
            if (tid < 4) {
                s_todo[tid][0] = tx + (tid & 1) * 8;
                s_todo[tid][1] = ty + (tid >> 1) * 8;
            }
            todo = 4;
        } else {
            // the triangles of the list from which a warp's rays can hit, by lane: whether triangle
            // c is one of them for the rays between corners k
            auto reach = [&](const Corners& k, int c) {
                const float4 A = s_tri[4 * c], B = s_tri[4 * c + 1], C = s_tri[4 * c + 2];
                return may_hit(k, mk(A.x, A.y, A.z), mk(A.w, B.x, B.y), mk(B.z, B.w, C.x), mk(C.y, C.z, C.w));
            };
            // a warp's patches: four of 4 x 2 pixels in a region of 8 x 4 (tiles of 16), or one.
            // The region's triangles are picked from the tile's first, a patch's from those.
            const bool four = T == 16 && size == 16;
            const int rx = tx + (warp & 1) * (four ? 8 : 4), ry = ty + (warp >> 1) * (four ? 4 : 2);
            bool own = false;  // the warp's list is s_list, or the tile's
            if (four && listed && nf + nb > 32) {
                const Corners K = make_corners(cm, rx, ry, 8, 4, H);
                int n = 0, f = 0;
                for (int side = 0; side < 2; ++side) {
                    const int c0 = side ? kCand - nb : 0, c1 = side ? kCand : nf;
                    for (int cb = c0; cb < c1; cb += 32) {
                        const bool in = cb + lane < c1 && reach(K, cb + lane);
                        const unsigned mask = __ballot_sync(0xffffffffu, in);
                        const int at = n + __popc(mask & ((1u << lane) - 1u));
                        if (in && at < kList) s_list[T == 16 ? warp : 0][at] = (unsigned short)(cb + lane);
                        n += __popc(mask);
                    }
                    if (!side) f = n;
                }
                if (n <= kList) { own = true; nf = f; nb = n - f; }
                __syncwarp();
            }
            for (int patch = 0; patch < (four ? 4 : 1); ++patch) {
                const int pw = rx + (patch & 1) * 4, ph = ry + (patch >> 1) * 2;
                const int j = lane >> 2, q = lane & 3;
                const int px = pw + (j & 3), py = ph + (j >> 2);
                const bool valid = px < R && py < R;
                Shade s;
                s.color = mk(0.0f, 0.0f, 0.0f);
                s.depth = 0.0f;
                if (!listed || nf + nb > 0) {
                    const v3 rd = ray_dir(r, qr, 2 * px + (q & 1), H - (2 * py + (q >> 1)), W, H);  // ray as in downsample_kernel
                    // a ray along a coordinate plane: its slab test has no finite distances, so a
                    // leaf may be entered and a box above it not
                    bool walk = valid && (!listed || rd.x == 0.0f || rd.y == 0.0f || rd.z == 0.0f);
                    Hit hit;
                    hit.tri = -1; hit.t = 0.0f; hit.p = mk(0.0f, 0.0f, 0.0f);
                    if (listed) {
                        const Corners K = make_corners(cm, pw, ph, 4, 2, H);
                        float tMin = valid && !walk ? 1e6f : 0.0f;  // (a lane at 0 hits nothing)
                        float second = 1e6f;  // no hit but the best one is nearer
                        int best = -1;
                        // moller_trumbore on a prepared triangle, in two parts.  First the numerators
                        // against the determinant, by more than rounding: a division only for
                        // the triangles a ray is in, or nearly
                        auto near_in = [&](int c, float& det, float& nu, float& nv) {
                            const float4 A = s_tri[4 * c], B = s_tri[4 * c + 1], C = s_tri[4 * c + 2];
                            const v3 pvec = cross(rd, mk(A.w, B.x, B.y));
                            det = dot(mk(A.x, A.y, A.z), pvec);
                            nu = dot(mk(B.z, B.w, C.x), pvec);
                            nv = dot(rd, mk(C.y, C.z, C.w));
                            const float ad = fabsf(det), su = det < 0.0f ? -nu : nu, sv = det < 0.0f ? -nv : nv;
                            return !(ad < 0.0001f || su < -1e-30f || sv < -1e-30f || su > 1.00001f * ad || su + sv > 1.00002f * ad);
                        };
                        // a hit of triangle c at distance t
                        auto take = [&](int c, float t, const float4& D) {
                            if (t > tMin) { second = fminf(second, t); return; }
                            second = tMin;
                            if (t == tMin) {  // the traversal keeps the first of equals in the reference's order
                                if (best < 0) return;
                                const float4 E = s_tri[4 * best + 3];
                                const int f0 = ev.first[__float_as_int(D.y)], f1 = ev.first[__float_as_int(E.y)];
                                if (!(f0 > f1 || (f0 == f1 && __float_as_int(D.z) < __float_as_int(E.z)))) return;
                            }
                            tMin = t;
                            best = c;
                        };
                        auto test = [&](int c, float det, float nu, float nv) {
                            const float4 D = s_tri[4 * c + 3];
                            const float invDet = 1.0f / det;
                            const float u = nu * invDet;
                            if (u < 0.0f || u > 1.0f) return;
                            const float v = nv * invDet;
                            if (v < 0.0f || u + v > 1.0f) return;
                            const float t = D.x * invDet;
                            if (!(t > 0.0f)) return;
                            take(c, t, D);
                        };
                        float far = 1e6f;
                        for (int side = 0; side < 2; ++side) {
                            const int c0 = !side ? 0 : own ? nf : kCand - nb, c1 = c0 + (side ? nb : nf);
                            for (int cb = c0 + 32 * part; cb < c1; cb += 32 * HALVES) {
                                // what lies behind every ray's hit so far, and a little more, is left out
                                far = 1.00001f * __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(tMin)));
                                int c = cb + lane;
                                bool in = c < c1;
                                if (in) {
                                    if (own) c = s_list[T == 16 ? warp : 0][c];
                                    in = s_tri[4 * c + 3].w <= far && reach(K, c);
                                }
                                unsigned mask = __ballot_sync(0xffffffffu, in);
                                while (mask) {  // two at a time: a patch full of triangles waits for each in turn
                                    const int l0 = __ffs(mask) - 1;
                                    mask &= mask - 1;
                                    const int l1 = mask ? __ffs(mask) - 1 : l0;
                                    const int ca = __shfl_sync(0xffffffffu, c, l0), cb2 = __shfl_sync(0xffffffffu, c, l1);
                                    float da, ua, va, db, ub, vb;
                                    const bool ia = near_in(ca, da, ua, va), ib = near_in(cb2, db, ub, vb) && mask;
                                    mask &= mask - 1;
                                    if (ia) test(ca, da, ua, va);
                                    if (ib) test(cb2, db, ub, vb);
                                }
                            }
                        }
                        second = fminf(second, far);  // (the hits left out are behind this)
                        if constexpr (HALVES == 2) {
                            // the first warp takes the second's hits as it would one triangle's
                            if (part == 1) {
                                s_hit[warp][0][lane] = tMin;
                                s_hit[warp][1][lane] = second;
                                s_hit[warp][2][lane] = __int_as_float(best);
                            }
                            asm volatile("bar.sync %0, 64;" ::"r"(1 + warp) : "memory");
                            const float t = s_hit[warp][0][lane];
                            const int other = __float_as_int(s_hit[warp][2][lane]);
                            if (part == 0) {
                                if (other >= 0) take(other, t, s_tri[4 * other + 3]);
                                second = fminf(second, s_hit[warp][1][lane]);
                            }
                            asm volatile("bar.sync %0, 64;" ::"r"(1 + warp) : "memory");  // (read before the next tile's)
                        }
                        if (best >= 0) {
                            const float4 D = s_tri[4 * best + 3];
                            const int leaf = __float_as_int(D.y);
                            const float4 a = __ldg(ev.box + 2 * leaf), c = __ldg(ev.box + 2 * leaf + 1);
                            float tn;
                            if (slab(ro, rd, mk(a.x, a.y, a.z), mk(c.x, c.y, c.z), tn) && tn < second) {
                                hit.t = tMin;
                                hit.p = ro + tMin * rd;
                                hit.tri = (int)(ev.fofs + ev.tri[ev.first[leaf] + __float_as_int(D.z)]);
                            } else {
                                walk = true;
                            }
                        }
                    }
                    if (HALVES == 2 && part == 1) continue;
                    if (walk) hit = traverse(&r, &b, e, ro, rd);
                    if (valid) s = shade(r, ev, e, hit.tri, hit.t, hit.p);
                }
                if (part == 0) store_pixel(r, s, valid, e, px, py);
            }
        }
        if (todo == 0) return;
        __syncthreads();
        --todo;
        tx = s_todo[todo][0]; ty = s_todo[todo][1];
    }
}

// A thread per ray: a block traverses the rays of 8 x 8 pixels, a warp those of 4 x 2
__global__ void __launch_bounds__(256) k_rays_alone(const __grid_constant__ ffsrl_render r, const __grid_constant__ ffsrl_bvh b,
                                                    const int* __restrict__ ids, int n_ids) {
    const int R = r.resolution, W = 2 * R, H = 2 * R;
    const int tiles_x = (R + 7) / 8, tiles = tiles_x * tiles_x;
    const int k = blockIdx.x / tiles, tile = blockIdx.x % tiles;
    const int e = ids ? (k < n_ids ? ids[k] : r.num_envs) : k;
    const int warp = threadIdx.x >> 5, j = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
    const int px = (tile % tiles_x) * 8 + (warp & 1) * 4 + (j & 3), py = (tile / tiles_x) * 8 + (warp >> 1) * 2 + (j >> 2);
    const bool valid = e >= 0 && e < r.num_envs && px < R && py < R;
    Shade s;
    s.color = mk(0.0f, 0.0f, 0.0f);
    s.depth = 0.0f;
    if (valid) {
        const int cam = r.num_cameras > 1 ? e : 0;
        const v3 ro = ld3(r.camera_pos, cam);
        const float4 qr = reinterpret_cast<const float4*>(r.camera_rot)[cam];
        const EnvView ev = env_view(b, e);
        s = trace(r, ev, e, ro, qr, 2 * px + (q & 1), H - (2 * py + (q >> 1)), W, H);  // ray as in downsample_kernel
    }
    store_pixel(r, s, valid, e, px, py);
}

// Which kernel is fastest hangs on how densely a tile's pixels are covered with triangles and on
// how much there is to do.  What the sizes tell of both: `dense`, an env's nodes (about its
// triangles) over the pixels of a unit angle's square, and `work`, those pixels over all envs.
// Time over that of a thread per ray, mean and worst, of 8 x 8 tiles with two warps a patch, of
// 8 x 8 and of 16 x 16 tiles (1,116 images of ellipsoids of 500-46,640 tets with their instrument,
// alone and mixed, 1 to 216 envs, 72 to 700 pixels, lenses of 22, 40 and 60 degrees):
//     dense  work < 100,000              to 200,000                  to 800,000                  to 2.4 million              above
//     < .02                              0.56 0.6  0.57 0.6  1.1 1.3 0.68 1.2  0.60 0.8  1.0 1.4 0.84 1.5  0.64 1.0  0.7 1.1 1.1 1.6  0.68 1.1  0.47 0.9
//     < .08  0.66 0.8  0.76 1.0  1.5 1.8 0.67 1.1  0.75 1.2  1.4 2.6 0.70 1.1  0.68 1.1  1.2 1.7 0.87 1.4  0.70 1.2  0.9 1.5 1.0 1.5  0.67 1.0  0.56 1.1
//     < .16  0.73 1.1  0.86 1.2  1.7 2.3 0.79 1.2  0.87 1.2  1.5 1.9 0.92 1.2  0.86 1.2  1.3 2.0 1.10 1.4  0.85 1.1  1.0 1.4 1.2 1.6  0.79 1.1  0.67 1.0
//     < .32  0.83 1.1  0.93 1.2  1.9 2.5 1.03 1.2  1.04 1.2  1.6 1.9 1.20 1.4  1.06 1.2  1.5 1.9 1.32 1.5  0.98 1.1  1.1 1.2 1.3 1.6  0.87 1.1  0.77 1.1
//     more   1.03 1.2  1.09 1.2  2.1 2.4 1.18 1.3  1.18 1.2  2.0 2.5 1.34 1.5  1.14 1.2  1.7 2.4 1.48 1.7  1.09 1.2  1.3 1.6 1.5 1.7  1.00 1.2  0.99 1.3
// Tiles of 16 want some 600 blocks, too.  Through wider lenses (100 degrees, 372 images) most
// tiles are empty, which costs a thread per ray next to nothing: two warps a patch gain below a work
// of 100,000 and a density of .08 (0.70, worst 0.7), tiles of 16 above 800,000 and below .16 (0.79,
// 1.0), tiles of 8 nowhere to speak of.  In images of up to 64 pixels a tile holds much of the mesh.
// By this rule the images of the three lenses take 0.62 of a thread per ray's time (the best kernel
// for each 0.61), those of 100 degrees 0.97; the worst image 1.23.
void launch_rays(const ffsrl_render& r, const ffsrl_bvh& b, const int32_t* ids, int n, cudaStream_t s) {
    auto tiles = [&](int t) { return ((long long)(r.resolution + t - 1) / t) * ((r.resolution + t - 1) / t) * n; };
    const float lens = std::max(std::fabs(r.camera_tan), std::fabs(r.camera_tan * r.camera_aspect));
    const float per_angle = (float)r.resolution / lens, work = (float)n * per_angle * per_angle;
    const float dense = (float)b.total_env_nodes / (float)b.num_envs / (per_angle * per_angle);
    const bool wide = lens > 0.75f;
    bool t16, t8x2, t8;
    if (work >= 2.4e6f) t16 = dense < 0.64f && tiles(16) >= 600;
    else if (work >= 1.2e6f) t16 = dense < 0.32f && tiles(16) >= 1024;
    else t16 = wide && (work >= 8e5f ? dense < 0.16f : work >= 4e5f && dense < 0.02f);
    if (wide) {
        t8x2 = work < 1e5f && dense < 0.08f;
        t8 = false;
    } else {
        t8x2 = (work < 2e5f && dense < 0.16f) || (work < 1e5f && dense < 0.32f);
        t8 = dense < 0.16f;
    }
    if (r.resolution > 64 && t16) k_rays<16, 1><<<(unsigned)tiles(16), 256, 0, s>>>(r, b, ids, n);
    else if (r.resolution > 64 && t8x2) k_rays<8, 2><<<(unsigned)tiles(8), 512, 0, s>>>(r, b, ids, n);
    else if (r.resolution > 64 && t8) k_rays<8, 1><<<(unsigned)tiles(8), 256, 0, s>>>(r, b, ids, n);
    else k_rays_alone<<<(unsigned)tiles(8), 256, 0, s>>>(r, b, ids, n);
}

int32_t check_bvh(const ffsrl_bvh* b) {
    if (!b || b->num_envs <= 0 || !b->env_topology || !b->env_node_offset || !b->env_face_offset ||
        !b->topo_node_offset || !b->topo_tri_offset || !b->topo_max_level || !b->left_node || !b->first_tri_id ||
        !b->tri_count || !b->level || !b->tri_id || !b->aabb_min || !b->aabb_max || b->total_env_nodes <= 0)
        return fail(FFSRL_ERR_INVALID_ARGUMENT, "ffsrl_bvh: missing arrays or empty");
    if (!b->node_box != !b->tri_pos)
        return fail(FFSRL_ERR_INVALID_ARGUMENT, "ffsrl_bvh: node_box and tri_pos go together");
    if ((((uintptr_t)b->node_box) & 15) || (((uintptr_t)b->tri_pos) & 15))
        return fail(FFSRL_ERR_INVALID_ARGUMENT, "ffsrl_bvh: node_box and tri_pos must be 16-byte aligned");
    return FFSRL_OK;
}

int32_t check_render(const ffsrl_render* r) {
    if (!r || r->num_envs <= 0 || r->resolution <= 0 || !r->vis_point || !r->vis_face || !r->vis_point_color ||
        !r->vertex_normal || !r->camera_pos || !r->camera_rot || r->num_cameras <= 0 ||
        (r->num_lights > 0 && (!r->light_dir || !r->light_intensity)) || !r->error_flag)
        return fail(FFSRL_ERR_INVALID_ARGUMENT, "ffsrl_render: missing arrays");
    if (r->render_mode < 0 || r->render_mode > 4)
        return fail(FFSRL_ERR_INVALID_ARGUMENT, "ffsrl_render: render_mode must be 0..4");
    if (r->env_objects && (!r->object_texture || !r->texture || !r->tex_coords || !r->tex_indices))
        return fail(FFSRL_ERR_INVALID_ARGUMENT,
                    "ffsrl_render: env_objects needs object_texture, texture, tex_coords and tex_indices");
    if (r->num_cameras != 1 && r->num_cameras != r->num_envs)
        return fail(FFSRL_ERR_INVALID_ARGUMENT, "ffsrl_render: num_cameras must be 1 or num_envs");
    if (((uintptr_t)r->camera_rot) & 15)
        return fail(FFSRL_ERR_INVALID_ARGUMENT, "ffsrl_render: camera_rot must be 16-byte aligned");
    return FFSRL_OK;
}

}  // namespace
}  // namespace ffsrl

using namespace ffsrl;

extern "C" int32_t ffsrl_bvh_refit_levels(const ffsrl_bvh* b, const float* pts, const int32_t* faces, void* stream) {
    if (int32_t st = check_bvh(b)) return st;
    if (!pts || !faces) return fail(FFSRL_ERR_INVALID_ARGUMENT, "ffsrl_bvh_refit_levels: null points/faces");
    for (int L = b->max_level; L >= 0; --L)
        k_refit_level<<<grid_for(b->total_env_nodes, 256), 256, 0, (cudaStream_t)stream>>>(*b, pts, faces, L);
    FFSRL_LAUNCH_CHECK("ffsrl_bvh_refit_levels");
    return FFSRL_OK;
}

extern "C" int32_t ffsrl_bvh_refit_fused(const ffsrl_bvh* b, const float* pts, const int32_t* faces, void* stream) {
    if (int32_t st = check_bvh(b)) return st;
    if (!pts || !faces || !b->level_node || !b->level_start || !b->topo_level_offset)
        return fail(FFSRL_ERR_INVALID_ARGUMENT, "ffsrl_bvh_refit_fused: needs level grouping arrays");
    if (int32_t st = refit_fused(*b, pts, faces, nullptr, b->num_envs, (cudaStream_t)stream)) return st;
    FFSRL_LAUNCH_CHECK("ffsrl_bvh_refit_fused");
    return FFSRL_OK;
}

extern "C" int32_t ffsrl_render_reference(const ffsrl_render* r, const ffsrl_bvh* b, void* stream) {
    if (int32_t st = check_render(r)) return st;
    if (int32_t st = check_bvh(b)) return st;
    if (!r->normal_sum || !r->rays || !r->ray_depth)
        return fail(FFSRL_ERR_INVALID_ARGUMENT, "ffsrl_render_reference: needs normal_sum, rays, ray_depth scratch");
    cudaStream_t s = (cudaStream_t)stream;
    const int P = r->num_vis_points, Fv = r->num_vis_faces;
    k_zero3<<<grid_for(P, 256), 256, 0, s>>>(r->normal_sum, P);
    if (Fv > 0) k_normal_sum<<<grid_for(Fv, 256), 256, 0, s>>>(r->vis_point, r->vis_face, r->normal_sum, Fv);
    k_normalize<<<grid_for(P, 256), 256, 0, s>>>(r->normal_sum, r->vertex_normal, P);
    long long rays = 4ll * r->resolution * r->resolution * r->num_envs;
    k_draw<<<grid_for(rays, 128), 128, 0, s>>>(*r, *b);
    long long pix = (long long)r->resolution * r->resolution * r->num_envs;
    k_downsample<<<grid_for(pix, 256), 256, 0, s>>>(*r);
    FFSRL_LAUNCH_CHECK("ffsrl_render_reference");
    return FFSRL_OK;
}

extern "C" int32_t ffsrl_render_fused(const ffsrl_render* r, const ffsrl_bvh* b, void* stream) {
    if (int32_t st = check_render(r)) return st;
    if (int32_t st = check_bvh(b)) return st;
    if (!r->point_face_start || !r->point_face)
        return fail(FFSRL_ERR_INVALID_ARGUMENT, "ffsrl_render_fused: needs the point->face CSR");
    cudaStream_t s = (cudaStream_t)stream;
    const int P = r->num_vis_points;
    k_normal_gather<<<grid_for(P, 256), 256, 0, s>>>(r->vis_point, r->vis_face, r->point_face_start, r->point_face,
                                                     r->vertex_normal, P);
    launch_rays(*r, *b, nullptr, r->num_envs, s);
    FFSRL_LAUNCH_CHECK("ffsrl_render_fused");
    return FFSRL_OK;
}

extern "C" int32_t ffsrl_bvh_refit_fused_envs(const ffsrl_bvh* b, const float* pts, const int32_t* faces,
                                              const int32_t* env_ids, int32_t n, void* stream) {
    if (int32_t st = check_bvh(b)) return st;
    if (n < 0 || (n > 0 && (!pts || !faces || !env_ids || !b->level_node || !b->level_start || !b->topo_level_offset)))
        return fail(FFSRL_ERR_INVALID_ARGUMENT, "ffsrl_bvh_refit_fused_envs");
    if (n == 0) return FFSRL_OK;
    if (int32_t st = refit_fused(*b, pts, faces, env_ids, n, (cudaStream_t)stream)) return st;
    FFSRL_LAUNCH_CHECK("ffsrl_bvh_refit_fused_envs");
    return FFSRL_OK;
}

extern "C" int32_t ffsrl_render_fused_envs(const ffsrl_render* r, const ffsrl_bvh* b, const int32_t* env_ids,
                                           int32_t n, void* stream) {
    if (int32_t st = check_render(r)) return st;
    if (int32_t st = check_bvh(b)) return st;
    if (n < 0 || (n > 0 && (!env_ids || !r->point_face_start || !r->point_face || !r->env_point_start)))
        return fail(FFSRL_ERR_INVALID_ARGUMENT, "ffsrl_render_fused_envs: needs env ids, point->face CSR, env point ranges");
    if (n == 0) return FFSRL_OK;
    cudaStream_t s = (cudaStream_t)stream;
    k_normal_gather_envs<<<n, 256, 0, s>>>(r->vis_point, r->vis_face, r->point_face_start, r->point_face,
                                           r->vertex_normal, r->env_point_start, env_ids, r->num_envs);
    launch_rays(*r, *b, env_ids, n, s);
    FFSRL_LAUNCH_CHECK("ffsrl_render_fused_envs");
    return FFSRL_OK;
}
