// gi_kernels.cu -- sm_100a kernels of the mesh-mesh intersector.
//
// Build (once per mesh, replaces the reference's level-cut / forest builders,
// include/third-party/cubql/level_cut_builder.h:278-364 and forest_builder.h:405-517,
// which loop on the host with a device sync per tree level):
//   k_tri_boxes (and validation) -> k_morton_hist -> radix sort -> k_karras_leaves (leaves + binary tree)
//   -> k_state_tables -> k_wide_flags -> k_collapse (size-greedy 4-wide nodes,
//   their boxes from a pyramid of the sorted leaves' boxes) -> k_cut
// Large meshes: one host round trip, for the wide-node count (the node array's size).
//
// Intersect (replaces crossCheck.cu, DualTreeStep.cu, rapidDescendKernel.cu and the
// chunk loop of SingleTreeBatchIntersector.cu:170-455 in the reference):
//   k_traverse_blocks  one persistent launch: seeding from the cut pairs, BVH4 x
//               BVH4 traversal in the blocks' shared memory (16 child pairs per
//               node pair), a pool through which loaded blocks hand node pairs to
//               idle ones, and the first filter stage on the leaf pairs.
//   k_finish    sorted output of up to kFinMax results: the exact stage for the
//               escalated pairs, ordering, correctly rounded endpoints, and the
//               write to the host, in one launch.
//   k_exact, k_segments, ordering kernels  the same in separate launches, for
//               larger or unsorted results.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <type_traits>

#include "gi_classify.cuh"
#include "gi_launch.h"
#include "gi_sort.cuh"

namespace gi {

static std::atomic<unsigned long long> g_launches{0};
void note_launches(unsigned n)
{
    g_launches.fetch_add(n, std::memory_order_relaxed);
}
unsigned long long launch_count()
{
    return g_launches.load(std::memory_order_relaxed);
}

// ===========================================================================
// Build
// ===========================================================================
__device__ __forceinline__ unsigned f2ord(float f)
{
    unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned u)
{
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// Boxes are 6 consecutive values (lo xyz, hi xyz): 24 B for float (8-byte
// aligned), 48 B for double (16-byte aligned), moved as three 2-vectors.
template <class S>
struct Vec2Of;
template <>
struct Vec2Of<float> {
    using T = float2;
};
template <>
struct Vec2Of<double> {
    using T = double2;
};
template <class S>
__device__ __forceinline__ void load_box_cg(const S* p, S b[6])
{
    using V = typename Vec2Of<S>::T;
    const V* q = reinterpret_cast<const V*>(p);
    const V a = __ldcg(q), c = __ldcg(q + 1), d = __ldcg(q + 2);
    b[0] = a.x, b[1] = a.y, b[2] = c.x, b[3] = c.y, b[4] = d.x, b[5] = d.y;
}
template <class S>
__device__ __forceinline__ void store_box(S* p, const S b[6])
{
    using V = typename Vec2Of<S>::T;
    V* q = reinterpret_cast<V*>(p);
    q[0] = V{b[0], b[1]};
    q[1] = V{b[2], b[3]};
    q[2] = V{b[4], b[5]};
}

// One child slot of a wide node, as whole 16-byte vectors.
__device__ __forceinline__ void store_kid(WKid* kd, const float b[6], uint32_t ref)
{
    float4* q = reinterpret_cast<float4*>(kd);
    q[0] = make_float4(b[0], b[1], b[2], __uint_as_float(ref));
    q[1] = make_float4(b[3], b[4], b[5], 0.0f);
}
__device__ __forceinline__ void store_kid(WKid64* kd, const double b[6], uint32_t ref)
{
    double2* q = reinterpret_cast<double2*>(kd);
    q[0] = make_double2(b[0], b[1]);
    q[1] = make_double2(b[2], b[3]);
    q[2] = make_double2(b[4], b[5]);
    *reinterpret_cast<uint4*>(q + 3) = make_uint4(ref, 0u, 0u, 0u);
}

// FP32 boxes rounded outward (so every exact triangle lies inside its box) and
// centroid bounds.  The reference rounds to nearest (src/common/utils.cu:639),
// which can drop true pairs; outward rounding keeps the candidate set a superset.
// The same launch checks every vertex coordinate against the supported domain
// and every index against the vertex array (the boxes clamp it meanwhile), in
// the loads it needs anyway; a launch of its own took 4 to 11 us.
//
// Words of a build's header on the device, zero before the build.
enum { kHdrErr = 0, kHdrMin = 1, kHdrMax = 4, kHdrWide = 7, kHdrWords = 8 };
constexpr int kTriBoxThreads = 256;
__global__ void __launch_bounds__(kTriBoxThreads, 4) k_tri_boxes(const double* __restrict__ V, uint32_t nv,
                                                              const uint32_t* __restrict__ T, uint32_t nt,
                                                              float* __restrict__ box, double* __restrict__ box64,
                                                              unsigned* __restrict__ hdr)
{
    pdl_enter();
    float cmin[3] = {INFINITY, INFINITY, INFINITY}, cmax[3] = {-INFINITY, -INFINITY, -INFINITY};
    unsigned bad = 0;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < 3ull * nv; c += (size_t)gridDim.x * blockDim.x) {
        const double x = V[c], ax = fabs(x);
        if (!(ax <= 0x1p100) || (x != 0.0 && ax < 0x1p-100)) bad |= 2u;
    }
    // two triangles per iteration, all their loads issued before any use
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += 2 * stride) {
        const uint32_t tt[2] = {t, t + stride < nt ? t + stride : t};
        uint32_t ix[2][3];
        double v[2][9];
#pragma unroll
        for (int q = 0; q < 2; q++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const uint32_t x = T[3 * (size_t)tt[q] + j];
                if (x >= nv) bad |= 1u;
                ix[q][j] = min(x, nv - 1u);
            }
#pragma unroll
        for (int q = 0; q < 2; q++)
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const double3 p = load_vertex(V, ix[q][j]);
                v[q][3 * j] = p.x;
                v[q][3 * j + 1] = p.y;
                v[q][3 * j + 2] = p.z;
            }
#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (q == 1 && tt[1] == t) break;
            const size_t o = 6 * (size_t)tt[q];
            float fb[6];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const double a = v[q][k], b = v[q][3 + k], c = v[q][6 + k];
                const double lo = fmin(a, fmin(b, c)), hi = fmax(a, fmax(b, c));
                fb[k] = __double2float_rd(lo);
                fb[3 + k] = __double2float_ru(hi);
                if (box64) {
                    box64[o + k] = lo;
                    box64[o + 3 + k] = hi;
                }
                const float cc = 0.5f * fb[k] + 0.5f * fb[3 + k];
                cmin[k] = fminf(cmin[k], cc);
                cmax[k] = fmaxf(cmax[k], cc);
            }
            store_box(box + o, fb);
        }
    }
    // block reduction, then one set of atomics per block: per-warp atomics on
    // the same six words serialised in L2 and dominated the kernel
    __shared__ float red[kTriBoxThreads / 32][6];
    for (int k = 0; k < 3; k++) {
        for (int o = 16; o > 0; o >>= 1) {
            cmin[k] = fminf(cmin[k], __shfl_xor_sync(0xffffffffu, cmin[k], o));
            cmax[k] = fmaxf(cmax[k], __shfl_xor_sync(0xffffffffu, cmax[k], o));
        }
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0)
        for (int k = 0; k < 3; k++) {
            red[w][k] = cmin[k];
            red[w][3 + k] = cmax[k];
        }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int k = threadIdx.x;
        float v = red[0][k];
        for (int q = 1; q < kTriBoxThreads / 32; q++) v = k < 3 ? fminf(v, red[q][k]) : fmaxf(v, red[q][k]);
        // the minima as maxima of the complement: a header of zeros is neutral
        atomicMax(&hdr[kHdrMin + k], k < 3 ? ~f2ord(v) : f2ord(v));
    }
    if (bad) atomicOr(&hdr[kHdrErr], bad);
}

__device__ __forceinline__ uint32_t spread10(uint32_t x)
{
    x &= 0x3ffu;
    x = (x | (x << 16)) & 0x030000FFu;
    x = (x | (x << 8)) & 0x0300F00Fu;
    x = (x | (x << 4)) & 0x030C30C3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

// Box centre coordinate c quantised to 10 bits over [lo, lo + ext].
__device__ __forceinline__ uint32_t morton_axis(float c, float lo, float ext)
{
    float f = ext > 0.0f ? (c - lo) / ext : 0.0f;
    f = fminf(fmaxf(f, 0.0f), 1.0f);
    return (uint32_t)fminf(f * 1024.0f, 1023.0f);
}

// 30-bit Morton keys of the triangles (their box centres quantised to 10 bits
// per axis over the centroid bounds of the header) with identity values, a tile's
// triangles per block, and each block's counts of the first radix digit where
// k_rs_hist would write them, so the sort's first pass needs no histogram launch.
// All of a thread's box loads are issued before its first shared-memory atomic.
template <int BITS, int ITEMS, bool FEW>
__global__ void __launch_bounds__(kRsThreads) k_morton_hist(const float* __restrict__ box, uint32_t nt,
                                                            const unsigned* __restrict__ hdr,
                                                            RsElem* __restrict__ out, uint32_t* __restrict__ counts,
                                                            uint32_t ntiles)
{
    pdl_enter();
    constexpr uint32_t kDig = 1u << BITS;
    __shared__ uint32_t h[kDig];
    for (uint32_t d = threadIdx.x; d < kDig; d += kRsThreads) h[d] = 0;
    float lo[3], ext[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        lo[k] = ord2f(~hdr[kHdrMin + k]);
        ext[k] = ord2f(hdr[kHdrMax + k]) - lo[k];
    }
    const uint32_t base = blockIdx.x * (kRsThreads * ITEMS);
    uint32_t kk[ITEMS];
#pragma unroll
    for (int it = 0; it < ITEMS; it++) {
        const uint32_t t = base + it * kRsThreads + threadIdx.x;
        kk[it] = 0;
        if (t < nt) {
            const float2* b2 = reinterpret_cast<const float2*>(box + 6 * (size_t)t);
            const float2 a = b2[0], b = b2[1], c = b2[2];  // lo x, y | lo z, hi x | hi y, z
            const uint32_t qx = morton_axis(0.5f * a.x + 0.5f * b.y, lo[0], ext[0]);
            const uint32_t qy = morton_axis(0.5f * a.y + 0.5f * c.x, lo[1], ext[1]);
            const uint32_t qz = morton_axis(0.5f * b.x + 0.5f * c.y, lo[2], ext[2]);
            kk[it] = (spread10(qx) << 2) | (spread10(qy) << 1) | spread10(qz);
        }
    }
    __syncthreads();  // the histogram is cleared
#pragma unroll
    for (int it = 0; it < ITEMS; it++) {
        const uint32_t t = base + it * kRsThreads + threadIdx.x;
        if (t < nt) {
            out[t] = (RsElem)kk[it] << 32 | t;
            atomicAdd(&h[kk[it] & (kDig - 1u)], 1u);
        }
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d < kDig; d += kRsThreads) counts[rs_count_at<BITS, FEW>(d, blockIdx.x, ntiles)] = h[d];
}

__device__ __forceinline__ int kdelta(const uint32_t* __restrict__ keys, int n, int i, int j)
{
    if (j < 0 || j >= n) return -1;
    uint32_t a = keys[i], b = keys[j];
    if (a == b) return 32 + __clz((unsigned)(i ^ j));
    return __clz(a ^ b);
}

// Karras 2012 radix-tree construction over sorted Morton keys (ties by index),
// internal node i (i < n - 1).  child[i] = (left ref, right ref, leaves under
// left, leaves under right); parent[] of the internal children (the root's is -1).
__device__ __forceinline__ void karras_node(int i, const uint32_t* __restrict__ keys, int n, uint4* __restrict__ child,
                                            int* __restrict__ parent)
{
    int d = (kdelta(keys, n, i, i + 1) - kdelta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = kdelta(keys, n, i, i - d);
    int lmax = 2;
    while (kdelta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (kdelta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = kdelta(keys, n, i, j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (kdelta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    int gamma = i + s * d + min(d, 0);
    uint32_t left = (min(i, j) == gamma) ? (kLeaf | (uint32_t)gamma) : (uint32_t)gamma;
    uint32_t right = (max(i, j) == gamma + 1) ? (kLeaf | (uint32_t)(gamma + 1)) : (uint32_t)(gamma + 1);
    const int lo = min(i, j), hi = max(i, j);
    child[i] = make_uint4(left, right, (uint32_t)(gamma - lo + 1), (uint32_t)(hi - gamma));
    if (!(left & kLeaf)) parent[left] = i;
    if (!(right & kLeaf)) parent[right] = i;
    if (i == 0) parent[0] = -1;
}

// Unions of the sorted leaves' boxes over aligned runs of 2^L leaves (level L,
// entry e: leaves [e 2^L, (e + 1) 2^L)), L = 1 .. levels.  Every node of the
// radix tree covers consecutive leaves, so its box is the union of a few entries
// (range_box), read by whoever needs it, without a bottom-up pass over the tree.
// k_state_tables writes the levels that a block completes from its own leaves and
// one block of k_wide_flags the rest, beside work of the same latency.  (A
// bottom-up refit, an atomic arrival per node and level, took 61 us of a 1.3M-
// triangle build and 26 of a 300k one; the pyramid adds 14 us to k_state_tables
// and 15 to k_collapse at 1.3M, 2.5 and 0.5 at 300k.)
constexpr int kPyrLevels = 32;
constexpr int kPyrBlock = 8;  // levels that a block completes from its own leaves
constexpr int kPyrThreads = 1 << kPyrBlock;
template <class S>
struct Pyramid {
    S* box;                    // 6 values an entry
    uint32_t off[kPyrLevels];  // first entry of level L (L >= 1)
    int levels;
};

template <class S>
__device__ __forceinline__ void box_union(S (&b)[6], const S (&o)[6])
{
#pragma unroll
    for (int k = 0; k < 3; k++) {
        b[k] = min(b[k], o[k]);
        b[3 + k] = max(b[3 + k], o[3 + k]);
    }
}

// Levels 1 .. kPyrBlock of the pyramid over the block's leaves (thread = leaf):
// shuffles within a warp, shared memory within the block.  Every thread calls.
template <class S>
__device__ __forceinline__ void pyramid_block(const S* __restrict__ leafBox, int n, const Pyramid<S>& pyr)
{
    __shared__ S s_box[kPyrThreads / 32][6];
    const unsigned p = blockIdx.x * (unsigned)kPyrThreads + threadIdx.x;
    S b[6] = {(S)INFINITY, (S)INFINITY, (S)INFINITY, (S)-INFINITY, (S)-INFINITY, (S)-INFINITY};
    if (p < (unsigned)n) load_box_cg(leafBox + 6 * (size_t)p, b);
    const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
#pragma unroll
    for (int L = 1; L <= 5; L++) {
        S o[6];
#pragma unroll
        for (int q = 0; q < 6; q++) o[q] = __shfl_xor_sync(0xffffffffu, b[q], 1 << (L - 1));
        box_union(b, o);
        if (L <= pyr.levels && (lane & ((1u << L) - 1u)) == 0u && p < (unsigned)n)
            store_box(pyr.box + 6 * ((size_t)pyr.off[L] + (p >> L)), b);
    }
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 6; q++) s_box[w][q] = b[q];
    __syncthreads();
    // thread t of each level: its entry's warps t << (L - 5) ...
    for (int L = 6; L <= kPyrBlock && L <= pyr.levels; L++) {
        const unsigned width = 1u << (L - 5), x0 = threadIdx.x * width;
        const size_t first = (size_t)blockIdx.x * kPyrThreads + ((size_t)threadIdx.x << L);
        if (threadIdx.x < (unsigned)(kPyrThreads >> L) && first < (size_t)n) {
            S u[6], v[6];
#pragma unroll
            for (int q = 0; q < 6; q++) u[q] = s_box[x0][q];
            for (unsigned x = 1; x < width; x++) {
#pragma unroll
                for (int q = 0; q < 6; q++) v[q] = s_box[x0 + x][q];
                box_union(u, v);
            }
            store_box(pyr.box + 6 * ((size_t)pyr.off[L] + (first >> L)), u);
        }
    }
}

// The levels above a block's, by one block.
template <class S>
__device__ __forceinline__ void pyramid_top(int n, const Pyramid<S>& pyr)
{
    for (int L = kPyrBlock + 1; L <= pyr.levels; L++) {
        const uint32_t below = (uint32_t)(((unsigned long long)n + (1ull << (L - 1)) - 1u) >> (L - 1));
        const uint32_t here = (below + 1u) / 2u;
#pragma unroll 4
        for (uint32_t e = threadIdx.x; e < here; e += kPyrThreads) {
            S u[6], v[6];
            const S* const src = pyr.box + 6 * ((size_t)pyr.off[L - 1] + 2u * (size_t)e);
            const S* const src2 = 2u * e + 1u < below ? src + 6 : src;
            load_box_cg(src, u);
            load_box_cg(src2, v);
            box_union(u, v);
            store_box(pyr.box + 6 * ((size_t)pyr.off[L] + e), u);
        }
        __syncthreads();
    }
}

// Union of the boxes of the leaves [a, e): at most two entries a level, and the
// loads of two levels in flight at once (their addresses depend on a and e
// alone).  k_collapse at 300k / 1.3M triangles: 18 / 65 us with one level, 13 / 60
// with two, 13 / 63 with three, 15 / 67 with four (registers).
template <class S>
__device__ __forceinline__ void range_box(const S* __restrict__ leafBox, const Pyramid<S>& pyr, uint32_t a, uint32_t e, S (&b)[6])
{
    constexpr int kAhead = 2;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        b[k] = (S)INFINITY;
        b[3 + k] = (S)-INFINITY;
    }
    for (int L = 0; a < e; L += kAhead) {
        S o[2 * kAhead][6];
#pragma unroll
        for (int s = 0; s < kAhead; s++) {
            const S* const level = L + s == 0 || a >= e ? leafBox : pyr.box + 6 * (size_t)pyr.off[L + s];
            const bool ua = a < e && (a & 1u);
            const S* const pa = level + 6 * (size_t)a;
            a += ua ? 1u : 0u;
            const bool ue = a < e && (e & 1u);
            e -= ue ? 1u : 0u;
            const S* const pe = level + 6 * (size_t)e;
#pragma unroll
            for (int k = 0; k < 6; k++) o[2 * s][k] = o[2 * s + 1][k] = k < 3 ? (S)INFINITY : (S)-INFINITY;
            if (ua) load_box_cg(pa, o[2 * s]);
            if (ue) load_box_cg(pe, o[2 * s + 1]);
            if (a < e) {
                a >>= 1;
                e >>= 1;
            }
        }
#pragma unroll
        for (int s = 0; s < 2 * kAhead; s++) box_union(b, o[s]);
    }
}

// Leaves in sorted order (position p < n: the box and the vertex indices of
// triangle vals[p]) and the radix tree's internal node p (p < n - 1), in one
// launch: both are gathers or searches bound by latency, so each thread has
// two independent chains in flight.
template <class S>
__global__ void k_karras_leaves(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals, int n,
                                const uint32_t* __restrict__ T, const S* __restrict__ boxOrig,
                                S* __restrict__ leafBox, uint4* __restrict__ leafTri, uint4* __restrict__ child,
                                int* __restrict__ parent)
{
    pdl_enter();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const uint32_t tri = vals[p];
    S b[6];
    load_box_cg(boxOrig + 6 * (size_t)tri, b);
    uint4 t4 = make_uint4(0u, 0u, 0u, 0u);
    if (leafTri) t4 = make_uint4(T[3 * (size_t)tri], T[3 * (size_t)tri + 1], T[3 * (size_t)tri + 2], tri);
    if (p < n - 1) karras_node(p, keys, n, child, parent);
    store_box(leafBox + 6 * (size_t)p, b);
    if (leafTri) leafTri[p] = t4;
}

__device__ __forceinline__ unsigned arrive_acq_rel(unsigned* f)
{
    unsigned old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(f) : "memory");
    return old;
}

// ---------------------------------------------------------------------------
// Collapse of the binary radix tree into the 4-wide BVH, size-greedy.
//
// A wide node is made from a binary node r by opening r and then, twice, the
// part with the most leaves (ties: the leftmost part), as long as that part is
// an internal node; the parts stay in left-to-right order.  Each binary node is
// thus either a wide node (state W) or opened in the second (O2) or third (O3)
// step of its wide ancestor's expansion.  Opening the largest part shrinks
// the largest subtree of a wide node faster than taking grandchildren by
// depth parity does on the unbalanced trees that Morton splits give on a
// surface: on a 1.3 M-triangle sphere the pair tree of two such meshes has
// one level and a fifth of its node pairs fewer.
//
// A node's state follows from its parent's through a 3-entry table that
// depends only on the leaf counts around it (k_state_tables).  k_wide_flags
// composes the tables up the parent chain until the composition no longer
// depends on the state above (about five steps a node), so no top-down pass
// over the levels is needed.
constexpr unsigned kStW = 0u, kStO2 = 1u, kStO3 = 2u;
constexpr unsigned kErrBuild = 4u;  // error word bit: an inconsistent wide tree (not expected)

// position (0..2) of the first maximum of three counts
__device__ __forceinline__ unsigned first_max3(uint32_t a, uint32_t b, uint32_t c)
{
    unsigned k = 0;
    uint32_t m = a;
    if (b > m) {
        m = b;
        k = 1;
    }
    if (c > m) k = 2;
    return k;
}

// tab[y] bits 2s..2s+1: the state of internal node y (y >= 1) when its parent
// is in state s (s = W, O2; a child of an O3 node is always W).
template <class S>
__global__ void __launch_bounds__(kPyrThreads) k_state_tables(int n, const uint4* __restrict__ child, const int* __restrict__ parent,
                               uint8_t* __restrict__ tab, const S* __restrict__ leafBox,
                               const __grid_constant__ Pyramid<S> pyr)
{
    pdl_enter();
    pyramid_block(leafBox, n, pyr);
    int y = blockIdx.x * blockDim.x + threadIdx.x;
    if (y < 1 || y >= n - 1) return;
    const int p = parent[y];
    const uint4 c = child[p];
    const bool left = c.x == (uint32_t)y;
    const uint32_t z = left ? c.y : c.x;
    const uint32_t ny = left ? c.z : c.w, nz = left ? c.w : c.z;
    // parent in W: step 2 opens the larger child (tie: the left one)
    unsigned sW;
    if (left ? ny >= nz : ny > nz) {
        sW = kStO2;
    } else {  // the sibling z (internal: nz > ny >= 2) was opened; step 3 over the three parts
        const uint4 g = child[z];
        const uint32_t n0 = g.z, n1 = g.w;
        sW = (left ? first_max3(ny, n0, n1) == 0u : first_max3(n0, n1, ny) == 2u) ? kStO3 : kStW;
    }
    // parent in O2 (opened by its own parent r): step 3 over p's children and p's sibling
    unsigned sO2 = kStW;
    const int r = parent[p];
    if (r >= 0) {
        const uint4 cr = child[r];
        const bool pleft = cr.x == (uint32_t)p;
        const uint32_t ns = pleft ? cr.w : cr.z;
        const uint32_t n0 = c.z, n1 = c.w;
        const unsigned mine = pleft ? (left ? 0u : 1u) : (left ? 1u : 2u);
        const unsigned k = pleft ? first_max3(n0, n1, ns) : first_max3(ns, n0, n1);
        sO2 = k == mine ? kStO3 : kStW;
    }
    tab[y] = (uint8_t)(sW | (sO2 << 2) | (kStW << 4));
}

// widx[i]: the wide node that binary node i becomes, or kEmpty.  The root is wide
// node 0; a block's others take consecutive places from one atomic on the
// header's count (the order of the blocks' runs varies from build to build and
// shows in no result; a scan of the flags kept it, for three launches more).
template <class S>
__global__ void __launch_bounds__(kPyrThreads) k_wide_flags(int n, const int* __restrict__ parent, const uint8_t* __restrict__ tab,
                                                    uint32_t* __restrict__ widx, unsigned* __restrict__ hdr,
                                                    const __grid_constant__ Pyramid<S> pyr)
{
    pdl_enter();
    if (blockIdx.x == 0) pyramid_top(n, pyr);
    __shared__ unsigned s_warp[8], s_base;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool wide = false;
    if (i > 0 && i < n - 1) {
        unsigned f = tab[i];  // state of i as a function of the state of the node above the chain
        int x = parent[i];
        for (int guard = 0; x > 0 && guard < n; guard++) {
            const unsigned f0 = f & 3u, f1 = (f >> 2) & 3u, f2 = (f >> 4) & 3u;
            if (f0 == f1 && f1 == f2) break;
            const unsigned t = __ldg(tab + x);
            f = ((f >> (2u * (t & 3u))) & 3u) | (((f >> (2u * ((t >> 2) & 3u))) & 3u) << 2) |
                (((f >> (2u * ((t >> 4) & 3u))) & 3u) << 4);
            x = parent[x];
        }
        wide = (f & 3u) == kStW;  // the root is a wide node
    }
    const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const unsigned m = __ballot_sync(0xffffffffu, wide);
    if (lane == 0) s_warp[w] = __popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned tot = 0;
        for (unsigned q = 0; q < 8u; q++) {
            const unsigned t = s_warp[q];
            s_warp[q] = tot;
            tot += t;
        }
        s_base = tot ? atomicAdd(&hdr[kHdrWide], tot) : 0u;
    }
    __syncthreads();
    if (i < n - 1) widx[i] = i == 0 ? 0u : (wide ? 1u + s_base + s_warp[w] + __popc(m & ((1u << lane) - 1u)) : kEmpty);
}

// Writes wide node widx[i] from binary node i: the size-greedy expansion of i
// (the same choices as k_state_tables), each child with the box of the leaves it
// covers (a left child's leaves end at its own index, a right child's begin
// there).  An internal part that is not a wide node, or whose index is out of
// range, cannot arise; it is written as an empty slot and flagged in *bad rather
// than followed.
//
// A block finds the children of its 256 binary nodes' wide nodes first, one
// thread a node, and then fills the child slots, one thread a slot: one node in
// two is wide, and a child with many leaves costs only its own thread the
// longer union.
constexpr int kColThreads = 256;
template <class S, class NodeT>
__global__ void __launch_bounds__(kColThreads) k_collapse(int n, const uint4* __restrict__ child, const uint32_t* __restrict__ widx,
                           uint32_t nw, const S* __restrict__ leafBox, const __grid_constant__ Pyramid<S> pyr,
                           NodeT* __restrict__ nodes, unsigned* __restrict__ bad)
{
    pdl_enter();
    __shared__ unsigned s_n;
    __shared__ uint32_t s_wi[kColThreads];
    __shared__ uint32_t s_ref[kColThreads * 4], s_lo[kColThreads * 4], s_num[kColThreads * 4];
    if (threadIdx.x == 0) s_n = 0u;
    __syncthreads();
    const int i = blockIdx.x * kColThreads + threadIdx.x;
    uint32_t wi = i < n - 1 ? widx[i] : kEmpty;
    if (wi != kEmpty && wi >= nw) {
        atomicOr(bad, kErrBuild);
        wi = kEmpty;
    }
    if (wi != kEmpty) {
        const uint4 c = child[i];
        uint32_t slot[4] = {c.x, c.y, kEmpty, kEmpty};
        uint32_t num[4] = {c.z, c.w, 0u, 0u};
        uint32_t right = 2u;  // bit k: part k is a right child
        int ns = 2;
#pragma unroll
        for (int step = 0; step < 2; step++) {
            int b = 0;
#pragma unroll
            for (int k = 1; k < 2 + step; k++)
                if (k < ns && num[k] > num[b]) b = k;
            if (num[b] < 2u) break;
            const uint4 g = child[slot[b]];
#pragma unroll
            for (int k = 3; k > 0; k--)
                if (k <= ns && k > b + 1) {
                    slot[k] = slot[k - 1];
                    num[k] = num[k - 1];
                }
            right = (right & ((1u << b) - 1u)) | (2u << b) | ((right >> (b + 1)) << (b + 2));
            slot[b] = g.x;
            slot[b + 1] = g.y;
            num[b] = g.z;
            num[b + 1] = g.w;
            ns++;
        }
        const unsigned at = atomicAdd(&s_n, 1u);
        s_wi[at] = wi;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t r = k < ns ? slot[k] : kEmpty, leaf = r & ~kLeaf;
            s_ref[4 * at + k] = r;
            s_num[4 * at + k] = num[k];
            s_lo[4 * at + k] = ((right >> k) & 1u) ? leaf : leaf - (num[k] - 1u);
        }
    }
    __syncthreads();
    for (unsigned t = threadIdx.x; t < 4u * s_n; t += kColThreads) {
        uint32_t r = s_ref[t], ref = kEmpty;
        if (r != kEmpty && !(r & kLeaf)) {
            ref = widx[r];
            if (ref >= nw) {
                atomicOr(bad, kErrBuild);
                r = ref = kEmpty;
            }
        } else {
            ref = r;
        }
        S bx[6] = {(S)INFINITY, (S)INFINITY, (S)INFINITY, (S)-INFINITY, (S)-INFINITY, (S)-INFINITY};
        if (r != kEmpty) range_box(leafBox, pyr, s_lo[t], s_lo[t] + s_num[t], bx);
        store_kid(&nodes[s_wi[t >> 2]].kid[t & 3u], bx, ref);
    }
}

// Cuts of the wide BVH: the root expanded three and four times (leaves met on
// the way are kept), each entry's box from its parent's child slot.  One block
// expands a level at a time, an entry per thread, the children placed by a
// block scan, so entries keep the order of a sequential expansion.  Output:
// the depth-3 cut (at most 4^3 entries) at [0, kCutMax), the depth-4 cut (at
// most 4^4) at [kCutMax, kCutCap); ncut[0], ncut[1] their sizes.  The
// traversal starts from all pairs of two meshes' cuts.
constexpr int kCutThreads = kCut4Max;
template <class S, class NodeT>
__global__ void __launch_bounds__(kCutThreads) k_cut(const NodeT* __restrict__ nodes, const S* __restrict__ leafBox,
                                                     uint32_t root, uint32_t* __restrict__ cutRef,
                                                     S* __restrict__ cutBox, uint32_t* __restrict__ ncut)
{
    pdl_enter();
    __shared__ uint32_t r[2][kCut4Max];
    __shared__ S b[2][kCut4Max][6];
    __shared__ uint32_t sw[33];
    const unsigned tid = threadIdx.x;
    if (root & kLeaf) {
        if (tid == 0) {
            for (int c = 0; c < 2; c++) {
                const unsigned o = c ? kCutMax : 0u;
                cutRef[o] = root;
                for (int k = 0; k < 6; k++) cutBox[6 * o + k] = leafBox[6 * (size_t)(root & ~kLeaf) + k];
            }
            ncut[0] = ncut[1] = 1u;
        }
        return;
    }
    if (tid == 0) r[0][0] = root;  // the root's own box is never used: it is expanded first
    __syncthreads();
    unsigned n = 1, cur = 0;
    for (int depth = 1; depth <= 4; depth++) {
        // n <= 4^(depth-1) <= kCutThreads: one entry per thread
        const uint32_t ref = tid < n ? r[cur][tid] : kLeaf;
        const bool node = tid < n && !(ref & kLeaf);
        unsigned cnt = 0;
        if (tid < n) {
            if (!node) cnt = 1;
            else
                for (int c = 0; c < 4; c++) cnt += nodes[ref].kid[c].ref != kEmpty;
        }
        unsigned tot;
        const unsigned ex = block_exclusive_scan(cnt, sw, &tot);
        const unsigned nx = cur ^ 1u;
        if (tid < n) {
            if (!node) {
                r[nx][ex] = ref;
                for (int k = 0; k < 6; k++) b[nx][ex][k] = b[cur][tid][k];
            } else {
                const NodeT& nd = nodes[ref];
                unsigned m = ex;
                for (int c = 0; c < 4; c++) {
                    const auto& kid = nd.kid[c];
                    if (kid.ref == kEmpty) continue;
                    r[nx][m] = kid.ref;
                    for (int q = 0; q < 3; q++) {
                        b[nx][m][q] = kid.lo[q];
                        b[nx][m][3 + q] = kid.hi[q];
                    }
                    m++;
                }
            }
        }
        __syncthreads();
        n = tot;
        cur = nx;
        if (depth >= 3) {
            const unsigned o = depth == 3 ? 0u : (unsigned)kCutMax;
            for (unsigned e = tid; e < n; e += kCutThreads) {
                cutRef[o + e] = r[cur][e];
                for (int k = 0; k < 6; k++) cutBox[6 * (o + e) + k] = b[cur][e][k];
            }
            if (tid == 0) ncut[depth - 3] = n;
        }
    }
}

#define GI_TRY(x)                                \
    do {                                         \
        cudaError_t e_ = (x);                    \
        if (e_ != cudaSuccess) return e_;        \
    } while (0)

// One piece of device memory handed out in aligned parts.
struct Carve {
    char* p;
    template <class T>
    T* take(size_t n)
    {
        T* q = (T*)p;
        p += (sizeof(T) * n + 255) & ~(size_t)255;
        return q;
    }
};

// Wide nodes of n triangles at most.  A node has four children unless it holds
// only two or three leaves; with a, b, c nodes of four, three and two children,
// 3a + 2b + c = n - 1 and 3b + 2c <= n, so a + b + c <= 2n / 3.
static uint32_t wide_bound(uint32_t n)
{
    return 2u * (n / 3u) + 2u;
}

// Above this many triangles the node array has its exact size, for a host round
// trip in the middle of the build (15 us of an idle GPU); below, the size of the
// bound, and the build is queued in one go.  (At 2^19 triangles the bound is 45 MB;
// a surface's tree takes about 33 MB of it, any tree 22 at least; twice that in
// FP64.  MeshBuffers::bytes counts the tree, and a budgeted context, which admits
// by it, has exact arrays at every size.)
constexpr uint32_t kExactNodesAbove = 1u << 19;
// Radix tiles of 1,024 keys up to this many triangles, else 3,072: the sort's
// kernels have a block per tile, and 3,072 leave most SMs idle (20 k triangles
// made seven blocks, 11-13 us a kernel; 300 k ninety-nine).
constexpr uint32_t kSmallTilesUpTo = 1u << 19;

bool build_wants_exact(uint32_t nt)
{
    return nt > kExactNodesAbove;
}

cudaError_t build_bvh(MeshBuffers& m, bool fp64, bool exact_nodes, unsigned* h_words, cudaMemPool_t pool, cudaStream_t st)
{
    const uint32_t n = m.nt;
    constexpr int kMortonDigit = 10;  // 30-bit keys: three passes
    constexpr uint32_t kDig = 1u << kMortonDigit;
    const bool small = n <= kSmallTilesUpTo;
    const uint32_t tile = kRsThreads * (small ? kRsItemsSmall : kRsItems), ntiles = (n + tile - 1) / tile;
    const uint32_t bound = n > 1 ? wide_bound(n) : 0u;
    // scratch in one allocation
    char* mem = nullptr;
    unsigned* hdr;
    float* box;
    double* box64;
    RsElem *e0, *e1;
    uint32_t *k0, *v0, *counts, *totals, *widx;
    uint4* child;
    int* parent;
    uint8_t* tab;
    Pyramid<float> py = {};
    Pyramid<double> py64 = {};
    // levels until one entry covers everything
    uint32_t off[kPyrLevels] = {}, entries = 0;
    int levels = 0;
    for (uint32_t m_ = n; m_ > 1;) {
        m_ = (m_ + 1u) / 2u;
        off[++levels] = entries;
        entries += m_;
    }
    for (;;) {
        Carve c{mem};
        hdr = c.take<unsigned>(kHdrWords);
        box = c.take<float>(6 * (size_t)n);
        box64 = fp64 ? c.take<double>(6 * (size_t)n) : nullptr;
        e0 = c.take<RsElem>(n);
        e1 = c.take<RsElem>(n);
        k0 = c.take<uint32_t>(n);
        v0 = c.take<uint32_t>(n);
        counts = c.take<uint32_t>((size_t)kDig * ntiles);
        totals = c.take<uint32_t>(kDig);
        child = c.take<uint4>(n);
        parent = c.take<int>(n);
        tab = c.take<uint8_t>(n);
        widx = c.take<uint32_t>(n);
        if (fp64) py64.box = c.take<double>(6 * (size_t)entries);
        else py.box = c.take<float>(6 * (size_t)entries);
        if (mem) break;
        GI_TRY(pool_alloc(&mem, (size_t)(c.p - mem) + 256, pool, st));
    }
    struct Free {
        void* p;
        cudaStream_t st;
        ~Free() { cudaFreeAsync(p, st); }
    } free_{mem, st};
    py.levels = py64.levels = levels;
    for (int L = 0; L < kPyrLevels; L++) py.off[L] = py64.off[L] = off[L];
    GI_TRY(cudaMemsetAsync(hdr, 0, sizeof(unsigned) * kHdrWords, st));
    constexpr int tb = 256;
    static_assert(kPyrThreads == tb && kColThreads == tb, "one block count serves all");
    const int gb = (int)((n + tb - 1) / tb);
    // Kernels that follow another kernel in the stream are launched as its
    // programmatic dependents (launch_dep): each waits for its predecessor at
    // its first statement, so only the next launch's latency overlaps the tail
    // of the current kernel (0.474 -> 0.446 ms per 1.3M-triangle build on
    // B200).  A kernel that follows a copy or a memset is a plain launch.
    // four resident blocks per SM, each looping: the centroid bounds take one set of atomics per block
    const uint32_t work = std::max(n, m.nv);
    const int gboxes = (int)((work + 2 * kTriBoxThreads - 1) / (2 * kTriBoxThreads));
    k_tri_boxes<<<gboxes < 1 ? 1 : (gboxes < 592 ? gboxes : 592), kTriBoxThreads, 0, st>>>(m.verts, m.nv, m.tris, n, box, box64, hdr);
    note_launches(1);
    if (!fp64) {  // (both trees have the same; a failed FP64 build leaves the FP32 one's)
        m.root = kEmpty;
        m.nnodes = 0;
    }
    if (n == 0) {
        GI_TRY(cudaGetLastError());
        return cudaMemcpyAsync(h_words, hdr, sizeof(unsigned) * kHdrWords, cudaMemcpyDeviceToHost, st);
    }
    auto sort = [&](auto items, auto few) {
        constexpr int kItems = decltype(items)::value;
        constexpr bool kFew = decltype(few)::value;
        launch_dep(k_morton_hist<kMortonDigit, kItems, kFew>, ntiles, kRsThreads, st, (const float*)box, n,
                   (const unsigned*)hdr, e0, counts, ntiles);
        radix_sort<kMortonDigit, kItems, kFew>(e0, e1, k0, v0, n, 30, counts, totals, st);
    };
    if (!small) sort(std::integral_constant<int, kRsItems>(), std::false_type());
    else if (ntiles <= kRsFew) sort(std::integral_constant<int, kRsItemsSmall>(), std::true_type());
    else sort(std::integral_constant<int, kRsItemsSmall>(), std::false_type());
    // leaves in sorted order, and the binary radix tree
    if (!fp64) {
        launch_dep(k_karras_leaves<float>, gb, tb, st, (const uint32_t*)k0, (const uint32_t*)v0, (int)n,
                   (const uint32_t*)m.tris, (const float*)box, m.leafBox, m.leafTri, child, parent);
    } else {
        GI_TRY(pool_alloc(&m.leafBox64, sizeof(double) * 6 * n, pool, st));
        launch_dep(k_karras_leaves<double>, gb, tb, st, (const uint32_t*)k0, (const uint32_t*)v0, (int)n,
                   (const uint32_t*)m.tris, (const double*)box64, m.leafBox64, (uint4*)nullptr, child, parent);
    }
    if (n == 1) {
        m.root = kLeaf | 0u;
    } else {
        const int gi_ = (int)((n - 1 + tb - 1) / tb);
        if (!fp64) {
            launch_dep(k_state_tables<float>, gb, kPyrThreads, st, (int)n, (const uint4*)child, (const int*)parent, tab,
                       (const float*)m.leafBox, py);
            launch_dep(k_wide_flags<float>, gi_, kPyrThreads, st, (int)n, (const int*)parent, (const uint8_t*)tab, widx, hdr, py);
        } else {
            launch_dep(k_state_tables<double>, gb, kPyrThreads, st, (int)n, (const uint4*)child, (const int*)parent, tab,
                       (const double*)m.leafBox64, py64);
            launch_dep(k_wide_flags<double>, gi_, kPyrThreads, st, (int)n, (const int*)parent, (const uint8_t*)tab, widx, hdr, py64);
        }
        uint32_t cap = bound;
        const bool exact = exact_nodes || build_wants_exact(n);
        if (exact) {
            GI_TRY(cudaMemcpyAsync(h_words, hdr, sizeof(unsigned) * kHdrWords, cudaMemcpyDeviceToHost, st));
            GI_TRY(cudaStreamSynchronize(st));
            cap = std::min(bound, 1u + h_words[kHdrWide]);
        }
        // (a plain launch after the host round trip, a dependent one otherwise)
        auto collapse = [&](auto kern, auto... args) {
            if (exact) kern<<<gi_, kColThreads, 0, st>>>(args...);
            else launch_dep(kern, gi_, kColThreads, st, args...);
        };
        if (!fp64) {
            GI_TRY(pool_alloc(&m.nodes, sizeof(WNode) * (size_t)cap, pool, st));
            collapse(k_collapse<float, WNode>, (int)n, (const uint4*)child, (const uint32_t*)widx, cap,
                     (const float*)m.leafBox, py, m.nodes, hdr + kHdrErr);
        } else {
            GI_TRY(pool_alloc(&m.nodes64, sizeof(WNode64) * (size_t)cap, pool, st));
            collapse(k_collapse<double, WNode64>, (int)n, (const uint4*)child, (const uint32_t*)widx, cap,
                     (const double*)m.leafBox64, py64, m.nodes64, hdr + kHdrErr);
        }
        m.root = 0;
        note_launches(3);
    }
    // depth-3 and depth-4 cuts, per precision (their sizes are the same); the sizes
    // stay on the device, where the seeding reads them
    if (!fp64) {
        launch_dep(k_cut<float, WNode>, 1, kCutThreads, st, (const WNode*)m.nodes, (const float*)m.leafBox, m.root,
                   m.cutRef, m.cutBox, m.ncuts);
    } else {
        GI_TRY(pool_alloc(&m.cutBox64, sizeof(double) * 6 * kCutCap, pool, st));
        GI_TRY(pool_alloc(&m.cutRef64, sizeof(uint32_t) * kCutCap, pool, st));
        launch_dep(k_cut<double, WNode64>, 1, kCutThreads, st, (const WNode64*)m.nodes64, (const double*)m.leafBox64,
                   m.root, m.cutRef64, m.cutBox64, m.ncuts);
    }
    note_launches(3);
    GI_TRY(cudaGetLastError());
    return cudaMemcpyAsync(h_words, hdr, sizeof(unsigned) * kHdrWords, cudaMemcpyDeviceToHost, st);
}

unsigned build_result(MeshBuffers& m, bool fp64, const unsigned* h_words)
{
    const uint32_t n = m.nt;
    if (n > 1) m.nnodes = 1u + h_words[kHdrWide];
    if (!fp64)
        m.bytes += sizeof(float) * 6 * (size_t)n + sizeof(uint4) * (size_t)n + sizeof(WNode) * (size_t)m.nnodes;
    else
        m.bytes += sizeof(double) * 6 * (size_t)n + sizeof(WNode64) * (size_t)m.nnodes;
    return h_words[kHdrErr];
}

size_t mesh_arena_bytes(uint32_t nv, uint32_t nt)
{
    MeshBuffers m;
    m.nv = nv;
    m.nt = nt;
    return mesh_arena(m, nullptr);
}
size_t mesh_arena(MeshBuffers& m, void* mem)
{
    Carve c{(char*)mem};
    // 16 bytes past the last vertex: the kernels read a vertex as the two
    // aligned 16-byte vectors that hold it (load_vertex)
    m.verts = c.take<double>(3 * (size_t)(m.nv ? m.nv : 1) + 2);
    m.tris = c.take<uint32_t>(3 * (size_t)(m.nt ? m.nt : 1));
    if (m.nt) {
        m.leafTri = c.take<uint4>(m.nt);
        m.leafBox = c.take<float>(6 * (size_t)m.nt);
        m.cutBox = c.take<float>(6 * kCutCap);
        m.cutRef = c.take<uint32_t>(kCutCap);
        m.ncuts = c.take<uint32_t>(2);
    }
    return (size_t)(c.p - (char*)mem);
}

// ===========================================================================
// Traversal
// ===========================================================================
template <class S>
struct Box {
    S lo[3], hi[3];
};

// Conservative world box of a local box under a pose:
//   centre' = Rf c + bf, half' = |Rf| h, padded by rho (|Rf|(|c| + h) + padm) + tau.
// rho = 2^-19 (FP32) / 2^-48 (FP64) covers, with a margin of >= 3x, the rounding of
// Rf and bf, of the box arithmetic, of c and h, and of the FP64 posed vertices.
// The map's rows are read as 16-byte vectors (from the constant bank for a single
// pair, four loads from a batch's job in memory).
__device__ __forceinline__ void map_box(const BoxMap& P, Box<float>& b)
{
    float c[3], h[3], s[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        c[k] = 0.5f * b.lo[k] + 0.5f * b.hi[k];
        h[k] = 0.5f * b.hi[k] - 0.5f * b.lo[k];
        s[k] = fabsf(c[k]) + h[k];
    }
#pragma unroll
    for (int r = 0; r < 3; r++) {
        const float4 w = P.row[r];
        const float wc = fmaf(w.z, c[2], fmaf(w.y, c[1], fmaf(w.x, c[0], w.w)));
        const float wh = fmaf(fabsf(w.z), h[2], fmaf(fabsf(w.y), h[1], fabsf(w.x) * h[0]));
        const float mag = fmaf(fabsf(w.z), s[2], fmaf(fabsf(w.y), s[1], fmaf(fabsf(w.x), s[0], P.padm[r])));
        const float pad = fmaf(0x1p-19f, mag, 0x1p-120f);
        b.lo[r] = wc - wh - pad;
        b.hi[r] = wc + wh + pad;
    }
}
__device__ __forceinline__ void world_box(const DevPose& P, Box<double>& b)
{
    double c[3], h[3];
    for (int k = 0; k < 3; k++) {
        c[k] = 0.5 * b.lo[k] + 0.5 * b.hi[k];
        h[k] = 0.5 * b.hi[k] - 0.5 * b.lo[k];
    }
    for (int r = 0; r < 3; r++) {
        double wc = P.b64[r], wh = 0.0, mag = P.padm64[r];
        for (int k = 0; k < 3; k++) {
            double a = P.R[3 * r + k];
            wc = fma(a, c[k], wc);
            wh = fma(fabs(a), h[k], wh);
            mag = fma(fabs(a), fabs(c[k]) + h[k], mag);
        }
        double pad = fma(0x1p-48, mag, 0x1p-300);
        b.lo[r] = wc - wh - pad;
        b.hi[r] = wc + wh + pad;
    }
}

// World box -> conservative box in the local frame of pose P (inverse map
// local = Ri*w + bi, Ri = R^T).  Same construction and bound as world_box; the
// pad also covers the error of R^T as the inverse (inv_eta <= 2^-30) and the
// FP64 rounding of the posed vertices.
__device__ __forceinline__ void local_box(const DevPose& P, Box<double>& b)
{
    double c[3], h[3];
    for (int k = 0; k < 3; k++) {
        c[k] = 0.5 * b.lo[k] + 0.5 * b.hi[k];
        h[k] = 0.5 * b.hi[k] - 0.5 * b.lo[k];
    }
    const double rel = 0x1p-48 + P.inv_eta;
    for (int r = 0; r < 3; r++) {
        double wc = P.bi64[r], wh = 0.0, mag = P.padmi64[r];
        for (int k = 0; k < 3; k++) {
            double a = P.Ri64[3 * r + k];
            wc = fma(a, c[k], wc);
            wh = fma(fabs(a), h[k], wh);
            mag = fma(fabs(a), fabs(c[k]) + h[k], mag);
        }
        double pad = fma(rel, mag, 0x1p-300);
        b.lo[r] = wc - wh - pad;
        b.hi[r] = wc + wh + pad;
    }
}
__device__ __forceinline__ void world_box(const DevPose& P, Box<float>& b)
{
    map_box(P.fw, b);
}

template <bool F64>
struct Prec;
template <>
struct Prec<false> {
    using S = float;
    using Node = WNode;
    static __device__ __forceinline__ const Node* nodes(const MeshDev& M) { return M.nodes; }
    static __device__ __forceinline__ const S* leafBox(const MeshDev& M) { return M.leafBox; }
};
template <>
struct Prec<true> {
    using S = double;
    using Node = WNode64;
    static __device__ __forceinline__ const Node* nodes(const MeshDev& M) { return M.nodes64; }
    static __device__ __forceinline__ const S* leafBox(const MeshDev& M) { return M.leafBox64; }
};

template <class S>
__device__ __forceinline__ bool overlap(const Box<S>& a, const Box<S>& b)
{
    return a.lo[0] <= b.hi[0] && b.lo[0] <= a.hi[0] && a.lo[1] <= b.hi[1] && b.lo[1] <= a.hi[1] &&
           a.lo[2] <= b.hi[2] && b.lo[2] <= a.hi[2];
}

__device__ __forceinline__ unsigned warp_append(bool pred, unsigned* counter)
{
    const unsigned lane = threadIdx.x & 31;
    unsigned m = __ballot_sync(0xffffffffu, pred);
    if (m == 0) return 0;
    unsigned leader = __ffs(m) - 1;
    unsigned base = 0;
    if (lane == leader) base = atomicAdd(counter, (unsigned)__popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    return base + __popc(m & ((1u << lane) - 1u));
}

__device__ __forceinline__ unsigned ld_cg_u32(const unsigned* p)
{
    return __ldcg(p);
}

template <bool F64>
__device__ __forceinline__ void load_tri(const MeshDev& M, const DevPose& P, uint32_t pos, double3* out,
                                         uint32_t* tri_id)
{
    uint4 t = __ldg(M.leafTri + pos);
    out[0] = world_vertex(M.verts, t.x, P);
    out[1] = world_vertex(M.verts, t.y, P);
    out[2] = world_vertex(M.verts, t.z, P);
    *tri_id = t.w;
}

// The job of an entry: one job travels in the kernel's parameters (constant
// bank), a batch's in memory.
template <bool MULTI>
__device__ __forceinline__ const JobDev& job_at(const Bufs& B, uint32_t j)
{
    if constexpr (MULTI) return B.jobs[j];
    else return B.job0;
}

// Child k of a node reference: a wide node's slot, or the leaf itself (k = 0; the
// other three are empty).  The four lanes of a quad read one node's line.
__device__ __forceinline__ void load_kid(const MeshDev& M, uint32_t ref, unsigned k, Box<float>& b, uint32_t& c)
{
    if (ref & kLeaf) {
        c = kEmpty;
        if (k == 0u) {
            const float2* lb = reinterpret_cast<const float2*>(M.leafBox + 6 * (size_t)(ref & ~kLeaf));
            const float2 u = __ldg(lb), v = __ldg(lb + 1), w = __ldg(lb + 2);
            b.lo[0] = u.x, b.lo[1] = u.y, b.lo[2] = v.x;
            b.hi[0] = v.y, b.hi[1] = w.x, b.hi[2] = w.y;
            c = ref;
        }
        return;
    }
    const float4* p = reinterpret_cast<const float4*>(&M.nodes[ref].kid[k]);
    const float4 u = __ldg(p), v = __ldg(p + 1);
    b.lo[0] = u.x, b.lo[1] = u.y, b.lo[2] = u.z;
    b.hi[0] = v.x, b.hi[1] = v.y, b.hi[2] = v.z;
    c = __float_as_uint(u.w);
}
__device__ __forceinline__ void load_kid(const MeshDev& M, uint32_t ref, unsigned k, Box<double>& b, uint32_t& c)
{
    const double2* p;
    c = kEmpty;
    if (ref & kLeaf) {
        if (k != 0u) return;
        p = reinterpret_cast<const double2*>(M.leafBox64 + 6 * (size_t)(ref & ~kLeaf));
        c = ref;
    } else {
        p = reinterpret_cast<const double2*>(&M.nodes64[ref].kid[k]);
        c = __ldg(reinterpret_cast<const uint32_t*>(p + 3));
    }
    const double2 u = __ldg(p), v = __ldg(p + 1), w = __ldg(p + 2);
    b.lo[0] = u.x, b.lo[1] = u.y, b.lo[2] = v.x;
    b.hi[0] = v.y, b.hi[1] = w.x, b.hi[2] = w.y;
}

constexpr unsigned kBlkThreads = 256, kBlkWarps = kBlkThreads / 32;
// consecutive idle polls of a block (a second or more), and how often they begin
// again because other blocks, with node pairs that they cannot share out, still work
constexpr unsigned kIdleSpins = 1u << 22, kIdleRounds = 64u;

__device__ __forceinline__ unsigned ld_vol(const unsigned* p)
{
    return *(const volatile unsigned*)p;
}

// Acquire load: the loads after it see what the writer published before its
// release (fence + tag store), without waiting for this thread's own stores
__device__ __forceinline__ unsigned ld_acq(const unsigned* p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Programmatic dependent launch: the launch that follows on the stream (the
// call's finish) may be scheduled now; it waits for this grid's completion and
// memory before it reads anything (wait_prior_grid).  Without such a launch
// both are no-ops.
__device__ __forceinline__ void allow_dependent_launch()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void wait_prior_grid()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A traversal block's counts at its end: summed over its warps in shared
// memory, then one atomic per counter for the block (every warp's own atomics
// on the same three words queued up at the end of the launch).  Every thread
// of the block must call it.
__device__ __forceinline__ void block_stats(Counters* C, unsigned long long visited, unsigned long long decided,
                                            unsigned long long tested, unsigned levels = 0u)
{
    __shared__ unsigned long long s_stats[4][kBlkWarps];
    for (int o = 16; o > 0; o >>= 1) {
        visited += __shfl_xor_sync(0xffffffffu, visited, o);
        decided += __shfl_xor_sync(0xffffffffu, decided, o);
        tested += __shfl_xor_sync(0xffffffffu, tested, o);
        levels = max(levels, __shfl_xor_sync(0xffffffffu, levels, o));
    }
    const unsigned warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31u) == 0u) {
        s_stats[0][warp] = visited;
        s_stats[1][warp] = decided;
        s_stats[2][warp] = tested;
        s_stats[3][warp] = levels;
    }
    __syncthreads();
    if (threadIdx.x < 4u) {
        unsigned long long t = 0;
        for (unsigned w = 0; w < kBlkWarps; w++)
            t = threadIdx.x == 3u ? max(t, s_stats[3][w]) : t + s_stats[threadIdx.x][w];
        if (threadIdx.x == 3u) {
            if (t) atomicMax(&C->levels, (unsigned)t);
        } else if (t) {
            atomicAdd(threadIdx.x == 0u ? &C->node_pairs : (threadIdx.x == 1u ? &C->filter_decided : &C->tested), t);
        }
    }
}

// ---------------------------------------------------------------------------
// Block traversal (BVH4 x BVH4, one cooperative launch): the blocks work alone
// on their own node pairs, in shared memory, and hand over what they cannot
// expand at once to blocks that have run out.
//
// A block holds a ring of node pairs and a list of leaf pairs (candidates) in
// shared memory.  An iteration pops up to 64 of the newest node pairs, one per
// quad of lanes, and pushes the overlapping children; 256 candidates are
// filtered at a time, one per thread, as soon as there are so many; results
// wait in shared memory and are appended to the result list in one piece.  A
// block starts from its share of the seed tests (the pairs of the two meshes'
// cut entries).
//
// Sharing out: a block without node pairs takes a ticket (q_head) and polls
// that slot of the pool.  Every iteration a block looks, with loads that its
// node loads hide, how many tickets are ahead of the slots given out (pool's low half);
// if some are, what it holds beyond one iteration's 64 node pairs goes to them
// from the oldest end (the largest subtrees), up to 64 a slot.  Slots are
// published by the call's tag in their flag word (release; a poll acquires it),
// so nothing is cleared between calls.
//
// A call's slots are given out once.  Near the pool's end blocks keep what they
// have (only one that would exceed its ring still gives, and past the end the call
// reruns with a larger pool); the host is told (`starved`) and takes a larger
// pool for the context's next call.
//
// Termination: the high half of `pool` counts blocks that work plus slots given
// out and not yet taken, less the grid's blocks.  A hand-over raises it in the
// same atomic that reserves its slots, a block lowers it when it runs out, and
// a taken slot's count becomes its taker's; so it reaches -blocks when, and
// only when, no node pair is left.  Every wait is bounded (longer while `starved`
// counts on); a spent wait sets kErrTimeout and the block ends.
//
// What bounds it is latency: an iteration is a chain of a shared-memory pop, a
// node load, a box transform, the tests and two block barriers, 1.2-2 us with
// three blocks per SM.  The forms it replaces handed every generation of node
// pairs to other SMs through L2, level by level with a grid barrier (5 us a
// level, 11 levels for two meshes of 1.3 M triangles) or through a queue of
// tagged slots.  Traversal with the filter, launch included, the better of those
// and this one: two UV spheres of 1,216 triangles 38 -> 21 us, of 20,224 57 -> 31,
// two spheres of 200 k 97 -> 53, of 1.3 M 96 -> 52 (FP64 form 100 -> 56), 48
// pairs of 10 k to 100 k in a batch 156 -> 134, coplanar 512 x 512 grids 216 ->
// 202; 256 pairs of 1 k to 200 k 484 -> 519.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long globaltimer_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void st_release_u32(unsigned* p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// resident blocks per SM that the registers are cut for, [batch].  A single pair
// is bound by latency: a fourth block's tighter registers cost small meshes 1 us;
// a batch is bound by work (256 pairs: 564 us of traversal with three, 519 with
// four, although its 64 registers spill: 220 bytes of stores in the FP32 form, 464
// in FP64; a single pair's 80 do not in FP32, 68 bytes in FP64).
constexpr int kBlkPerSm[2] = {3, 4};
constexpr unsigned kBlkUnits = kBlkThreads / 4;  // node pairs per iteration, and per slot of the pool
constexpr unsigned kBlkRing = 32 * kBlkUnits;               // node pairs a block holds (an iteration pushes at most 16 per unit)
constexpr unsigned kBlkHigh = kBlkRing - 16 * kBlkUnits;      // ... and may hold when an iteration begins
constexpr unsigned kBlkCand = kBlkThreads + 16 * kBlkUnits;  // candidates: less than a filter pass, and an iteration's
constexpr unsigned kBlkRes = 2 * kBlkThreads;    // results a block holds (a filter pass makes at most one per thread)
static_assert((kBlkRing & (kBlkRing - 1u)) == 0u, "ring index by mask");
static_assert(kBlkUnits + kBlkThreads <= kBlkHigh, "seeds are taken below one iteration's node pairs");

// a warp's child boxes of B, field by field, four children of a quad together
template <class S>
struct QuadBoxes {
    S f[6][32];
    uint32_t ref[32];
};
template <bool F64, bool MULTI>
struct BlockShared {
    QuadBoxes<typename Prec<F64>::S> x[kBlkThreads / 32];
    uint2 ring[kBlkRing];
    uint2 cand[kBlkCand];
    uint4 res[kBlkRes];
    uint32_t ring_job[MULTI ? kBlkRing : 1];
    uint32_t cand_job[MULTI ? kBlkCand : 1];
    unsigned push[2];  // pushed by the iteration: node pairs (low half), candidates (high half)
    unsigned nres, base, hungry, room, ticket, state;
};

// Segments that a construction code stands for.
__device__ __forceinline__ uint32_t code_segments(unsigned code)
{
    const unsigned kind = code & 3u;
    return kind == 3u ? 3u : (kind ? 1u : 0u);
}

// A result's key into its partition, for the one-launch finish: into the
// partition's bucket at the slot that one atomic on its count returns, or beyond
// the bucket on one overflow list.  The partitions divide the conceivable pairs
// evenly, in order (by the key's top bits, a job with a small mesh A had all its
// results in one partition).  ns: the result's segments (1 unless the exact
// stage found it).
__device__ __forceinline__ unsigned long long fin_key(const FinBufs& F, uint32_t job, uint32_t a, uint32_t b)
{
    return ((unsigned long long)job << (F.bits_a + F.bits_b)) | ((unsigned long long)a << F.bits_b) | b;
}
template <bool MULTI>
__device__ __forceinline__ void fin_insert(const Bufs& B, const uint4& r, uint32_t idx, unsigned ns)
{
    const FinBufs& F = B.fin;
    const unsigned long long key = fin_key(F, r.x, r.y, r.z);
    const unsigned long long rank = (job_at<MULTI>(B, r.x).a0 + r.y) * F.stride + r.z;
    const unsigned part = min((unsigned)__umul64hi(rank, F.scale), (unsigned)kFinParts - 1u);
    const unsigned slot = atomicAdd(F.count + part, 1u);
    const uint32_t v = idx | (ns << 30);
    if (slot < (unsigned)F.bucket) {
        F.bkey[(size_t)part * F.bucket + slot] = key;
        F.bval[(size_t)part * F.bucket + slot] = v;
    } else {
        const unsigned o = atomicAdd(&B.cnt->fin_over, 1u);
        if (o < (unsigned)kFinOverflow) {
            F.okey[o] = key;
            F.oval[o] = make_uint2(v, slot | (part << 20));
        }
    }
    if (ns != 1u) {
        atomicAdd(F.extra + part, ns - 1u);
        B.cnt->odd = 1u;
    }
}

// Results held by the block to the global list (all threads; nres is uniform).
template <bool F64, bool MULTI>
__device__ __forceinline__ void block_flush(const Bufs& B, BlockShared<F64, MULTI>& s, unsigned nres)
{
    __syncthreads();
    if (nres == 0u) return;
    if (threadIdx.x == 0) s.base = atomicAdd(&B.cnt->res, nres);
    __syncthreads();
    const unsigned base = s.base;
    for (unsigned k = threadIdx.x; k < nres; k += kBlkThreads) {
        if (base + k < B.cap_res) {
            B.res[base + k] = s.res[k];
            if (B.fin.on) fin_insert<MULTI>(B, s.res[k], base + k, 1u);
        } else {
            atomicOr(&B.cnt->overflow, kOvfRes);
        }
    }
    if (threadIdx.x == 0) s.nres = 0u;
    __syncthreads();
}

// First filter stage on the block's last `m` candidates (m <= 256), one per
// thread; every thread of the block calls it.
template <bool F64, bool MULTI>
__device__ __forceinline__ void block_filter(const Bufs& B, BlockShared<F64, MULTI>& s, unsigned cn, unsigned m,
                                             unsigned long long& decided, unsigned long long& tested)
{
    Counters* C = B.cnt;
    const unsigned tid = threadIdx.x;
    const bool have = tid < m;
    int dec = DEC_NO;
    uint4 r = make_uint4(0u, 0u, 0u, 0u);
    uint2 c = make_uint2(0u, 0u);
    if (have) {
        c = s.cand[cn - 1u - tid];
        if constexpr (MULTI) r.x = s.cand_job[cn - 1u - tid];
        tested++;
        const JobDev& J = job_at<MULTI>(B, r.x);
        const uint4 ta = __ldg(J.A.leafTri + c.x), tb = __ldg(J.B.leafTri + c.y);
        double3 P[3], Q[3];
        P[0] = world_vertex(J.A.verts, ta.x, J.pa);
        P[1] = world_vertex(J.A.verts, ta.y, J.pa);
        P[2] = world_vertex(J.A.verts, ta.z, J.pa);
        Q[0] = world_vertex(J.B.verts, tb.x, J.pb);
        Q[1] = world_vertex(J.B.verts, tb.y, J.pb);
        Q[2] = world_vertex(J.B.verts, tb.z, J.pb);
        if constexpr (F64) dec = classify_fast<double>(P, Q, &r.w);
        else dec = classify_fast<float>(P, Q, &r.w);
        decided += (dec != DEC_ESC);
        r.y = ta.w;
        r.z = tb.w;
    }
    const unsigned at = warp_append(have && dec == DEC_YES, &s.nres);
    if (have && dec == DEC_YES) s.res[at] = r;
    const bool esc = have && dec == DEC_ESC;
    const unsigned pe = warp_append(esc, &C->esc);
    if (esc) {
        if (pe < B.cap_esc) B.esc[pe] = make_uint4(r.x, c.x, c.y, 0u);
        else atomicOr(&C->overflow, kOvfEsc);
    }
    __syncthreads();
    const unsigned nres = s.nres;
    __syncthreads();  // read alike by all before the next pass adds to it
    if (nres > kBlkRes - kBlkThreads) block_flush<F64, MULTI>(B, s, nres);
}

// Seed test t: the pair of cut entries it names, if their world boxes overlap.
// A batch has kCutMax x kCutMax tests per job on the depth-3 cuts, one pair the
// nA x nB tests of its depth-4 cuts.
template <bool F64, bool MULTI>
__device__ __forceinline__ bool seed_test(const Bufs& B, unsigned t, unsigned nA, unsigned nB, uint32_t& job, uint2& ab)
{
    using S = typename Prec<F64>::S;
    unsigned coff = (unsigned)kCutMax;
    job = 0;
    if constexpr (MULTI) {
        coff = 0u;
        job = t / (unsigned)(kCutMax * kCutMax);
        t %= (unsigned)(kCutMax * kCutMax);
    }
    const JobDev& J = job_at<MULTI>(B, job);
    if constexpr (MULTI) {
        if (!J.A.nt || !J.B.nt) return false;  // an empty mesh has no cut (null sizes)
        nA = __ldg(J.A.ncuts);
        nB = __ldg(J.B.ncuts);
    }
    if (t >= nA * nB) return false;
    const unsigned i = coff + t / nB, j = coff + t % nB;
    const S* ba_ = F64 ? (const S*)J.A.cutBox64 : (const S*)J.A.cutBox;
    const S* bb_ = F64 ? (const S*)J.B.cutBox64 : (const S*)J.B.cutBox;
    Box<S> ba, bb;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        ba.lo[k] = __ldg(ba_ + 6 * i + k);
        ba.hi[k] = __ldg(ba_ + 6 * i + 3 + k);
        bb.lo[k] = __ldg(bb_ + 6 * j + k);
        bb.hi[k] = __ldg(bb_ + 6 * j + 3 + k);
    }
    ab = make_uint2(__ldg((F64 ? J.A.cutRef64 : J.A.cutRef) + i), __ldg((F64 ? J.B.cutRef64 : J.B.cutRef) + j));
    if (!J.pa.identity) world_box(J.pa, ba);
    if (!J.pb.identity) world_box(J.pb, bb);
    return overlap(ba, bb);
}

// One node pair per quad of lanes, lane `sub` owning child `sub` of both nodes:
// it maps its own child boxes to the world frame, the quad exchanges B's four
// through shared memory (x holds a warp's 8 quads; a 16-byte read gives one
// field of all four), and the lane tests its A child against them.  Called by
// all 32 lanes; lanes without a node pair (have = false) get no children.
// fm / cm: bit j set when (own A child, B child j) overlap and lead to a node
// pair / a leaf pair; B's child refs stay in x.ref (until the warp's next call).
//
// A batch also tests B's boxes in B's own frame (A's world boxes mapped back
// through B's pose): the world box of a rotated box is wider than the box, and
// each test alone is conservative.  That removes a quarter of its node pairs
// for about a third more work per pair (256 pairs of 1 k to 200 k triangles:
// 649 us of traversal without, 559 with), which pays where the traversal is
// bound by work, not for one pair, which is bound by latency.
template <class S>
struct Vec4 {
    S v[4];
};
__device__ __forceinline__ Vec4<float> lds4(const float* p)
{
    const float4 q = *reinterpret_cast<const float4*>(p);
    return {q.x, q.y, q.z, q.w};
}
__device__ __forceinline__ Vec4<double> lds4(const double* p)
{
    const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
    return {a.x, a.y, b.x, b.y};
}
template <class S>
__device__ __forceinline__ void quad_put(QuadBoxes<S>& x, const Box<S>& b)
{
    const unsigned lane = threadIdx.x & 31u;
#pragma unroll
    for (int q = 0; q < 3; q++) {
        x.f[q][lane] = b.lo[q];
        x.f[3 + q][lane] = b.hi[q];
    }
}
// bit j: box a meets box j of the quad
template <class S>
__device__ __forceinline__ unsigned quad_meets(const QuadBoxes<S>& x, const Box<S>& a)
{
    const unsigned q4 = threadIdx.x & 28u;
    bool ov[4] = {true, true, true, true};
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const Vec4<S> lo = lds4(&x.f[q][q4]), hi = lds4(&x.f[3 + q][q4]);
#pragma unroll
        for (int j = 0; j < 4; j++) ov[j] = ov[j] & (a.lo[q] <= hi.v[j]) & (lo.v[j] <= a.hi[q]);
    }
    return (ov[0] ? 1u : 0u) | (ov[1] ? 2u : 0u) | (ov[2] ? 4u : 0u) | (ov[3] ? 8u : 0u);
}
template <bool F64, bool MULTI>
__device__ __forceinline__ void block_expand(const Bufs& B, QuadBoxes<typename Prec<F64>::S>& x, const uint4& ent,
                                             bool have, unsigned sub, unsigned& fm, unsigned& cm, uint32_t& ca)
{
    using S = typename Prec<F64>::S;
    const JobDev& J = job_at<MULTI>(B, have ? ent.x : 0u);
    const unsigned lane = threadIdx.x & 31u, q4 = lane & 28u;
    Box<S> a, b;
    uint32_t mb = kEmpty;
    ca = kEmpty;
#pragma unroll
    for (int q = 0; q < 3; q++) a.lo[q] = a.hi[q] = b.lo[q] = b.hi[q] = S(0);
    unsigned m = 0xFu;
    if constexpr (MULTI && !F64) {
        if (have) {
            load_kid(J.A, ent.y, sub, a, ca);
            load_kid(J.B, ent.z, sub, b, mb);
            if (J.pa.fw.use) map_box(J.pa.fw, a);
        }
        if (B.two_frame) {  // uniform over the launch
            quad_put(x, b);
            __syncwarp();
            if (have && J.pb.inv.use) {
                Box<S> al = a;
                map_box(J.pb.inv, al);
                m = quad_meets(x, al);
            }
            __syncwarp();
        }
        if (have && J.pb.fw.use) map_box(J.pb.fw, b);
    } else {
        if (have) {
            load_kid(J.A, ent.y, sub, a, ca);
            load_kid(J.B, ent.z, sub, b, mb);
            if (!J.pa.identity) world_box(J.pa, a);
        }
        if (MULTI && B.two_frame) {
            quad_put(x, b);
            __syncwarp();
            if (have && J.pb.inv_ok) {
                Box<S> al = a;
                if constexpr (F64) local_box(J.pb, al);
                m = quad_meets(x, al);
            }
            __syncwarp();
        }
        if (have && !J.pb.identity) world_box(J.pb, b);
    }
    quad_put(x, b);
    x.ref[lane] = mb;
    __syncwarp();
    const uint4 r4 = *reinterpret_cast<const uint4*>(&x.ref[q4]);
    const uint32_t cb[4] = {r4.x, r4.y, r4.z, r4.w};
    m &= quad_meets(x, a);
    unsigned there = 0, leaf = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        there |= (cb[j] != kEmpty ? 1u : 0u) << j;
        leaf |= (cb[j] >> 31) << j;
    }
    m = ca != kEmpty ? m & there : 0u;
    cm = (ca & kLeaf) ? m & leaf : 0u;
    fm = m & ~cm;
}

// Hands the block's `m` oldest node pairs (ring positions rb ..) to `d` slots of
// the pool (m <= 64 d), as evenly as whole entries allow; all threads call it.
// Slots past the pool's end are dropped and flagged (the call reruns with a
// larger pool); they count as taken.
template <bool F64, bool MULTI>
__device__ __forceinline__ void block_give(const Bufs& B, BlockShared<F64, MULTI>& s, unsigned rb, unsigned m, unsigned d)
{
    Counters* C = B.cnt;
    const unsigned nslots = B.cap_queue / kBlkUnits, tid = threadIdx.x;
    if (tid == 0) s.base = (unsigned)atomicAdd(&C->pool, ((unsigned long long)d << 32) + d);
    __syncthreads();
    const unsigned base = s.base, q = (m + d - 1u) / d;
    for (unsigned k = tid; k < m; k += kBlkThreads) {
        const unsigned c = k / q, at = (rb + k) & (kBlkRing - 1u);
        const uint2 ab = s.ring[at];
        uint32_t job = 0;
        if constexpr (MULTI) job = s.ring_job[at];
        if (base + c < nslots) B.queue[(size_t)(base + c) * kBlkUnits + (k - c * q)] = make_uint4(job, ab.x, ab.y, min(q, m - c * q));
    }
    __syncthreads();
    if (tid < d) {
        if (base + tid < nslots) {
            // an empty slot (the entries did not divide) is published with no entries
            if (tid * q >= m) B.queue[(size_t)(base + tid) * kBlkUnits] = make_uint4(0u, kEmpty, kEmpty, 0u);
            st_release_u32(B.qflag + base + tid, B.tag);
        } else {
            atomicOr(&C->overflow, kOvfFrontier);
            atomicAdd(&C->pool, ~0ull << 32);
        }
    }
}

template <bool F64, bool MULTI>
__global__ void __launch_bounds__(kBlkThreads, kBlkPerSm[MULTI ? 1 : 0]) k_traverse_blocks(const __grid_constant__ Bufs B)
{
    extern __shared__ __align__(16) unsigned char blk_dyn[];
    BlockShared<F64, MULTI>& s = *reinterpret_cast<BlockShared<F64, MULTI>*>(blk_dyn);
    Counters* C = B.cnt;
    const unsigned tid = threadIdx.x, lane = tid & 31u, unit = tid >> 2, sub = tid & 3u;
    const unsigned G = gridDim.x, b = blockIdx.x;
    const unsigned nslots = B.cap_queue / kBlkUnits;
    const unsigned lt = (1u << lane) - 1u;
    allow_dependent_launch();
    if (b == 0 && tid == 0) C->t_start = globaltimer_ns();
    if (tid == 0) {
        s.push[0] = s.push[1] = 0u;
        s.nres = 0u;
    }
    // the block's share of the seed tests: one pair's with the grid's stride (its
    // overlapping cut entries cluster), a batch's in runs of one block's threads
    // (lanes then share a job)
    unsigned nA = 0, nB = 0, total;
    if constexpr (MULTI) {
        total = B.njobs * (unsigned)(kCutMax * kCutMax);
    } else {
        if (B.job0.A.nt && B.job0.B.nt) {  // an empty mesh has no cut (null sizes)
            nA = __ldg(B.job0.A.ncuts + 1);
            nB = __ldg(B.job0.B.ncuts + 1);
        }
        total = nA * nB;
    }
    const unsigned deal = MULTI ? (total + kBlkThreads - 1u) / kBlkThreads : total;  // dealt to the blocks in turn
    const unsigned share = deal > b ? (deal - b + G - 1u) / G : 0u;
    const unsigned chunks = MULTI ? share : (share + kBlkThreads - 1u) / kBlkThreads;
    unsigned taken = 0;
    unsigned long long visited = 0, decided = 0, tested = 0;
    // node pairs at ring positions rb .. rb + sn - 1, candidates 0 .. cn - 1 (alike in all threads)
    unsigned rb = 0, sn = 0, cn = 0, it = 0;
    __syncthreads();
    for (;;) {
        if (cn >= kBlkThreads) {
            block_filter<F64, MULTI>(B, s, cn, kBlkThreads, decided, tested);
            cn -= kBlkThreads;
            continue;
        }
        if (sn > kBlkHigh) {  // too many for another iteration
            const unsigned m = kBlkHigh / 2u;
            block_give<F64, MULTI>(B, s, rb, m, m / kBlkUnits);
            rb += m;
            sn -= m;
            continue;
        }
        if (taken < chunks && sn < kBlkUnits) {
            const unsigned c = taken++;
            __syncthreads();
            if (tid == 0) s.push[(it & 1u) ^ 1u] = 0u;  // read by all before this barrier
            const unsigned t = MULTI ? (c * G + b) * kBlkThreads + tid : (c * kBlkThreads + tid) * G + b;
            uint32_t job = 0;
            uint2 ab = make_uint2(kLeaf, kLeaf);
            const bool ov = t < total && seed_test<F64, MULTI>(B, t, nA, nB, job, ab);
            const bool cand = ov && (ab.x & kLeaf) && (ab.y & kLeaf), node = ov && !cand;
            const unsigned bn = __ballot_sync(0xffffffffu, node), bc = __ballot_sync(0xffffffffu, cand);
            unsigned old = 0;
            if (lane == 0 && (bn | bc)) old = atomicAdd(&s.push[it & 1u], __popc(bn) + (__popc(bc) << 16));
            old = __shfl_sync(0xffffffffu, old, 0);
            if (node) {
                const unsigned at = (rb + sn + (old & 0xffffu) + __popc(bn & lt)) & (kBlkRing - 1u);
                s.ring[at] = ab;
                if constexpr (MULTI) s.ring_job[at] = job;
            }
            if (cand) {
                const unsigned at = cn + (old >> 16) + __popc(bc & lt);
                s.cand[at] = make_uint2(ab.x & ~kLeaf, ab.y & ~kLeaf);
                if constexpr (MULTI) s.cand_job[at] = job;
            }
            __syncthreads();
            const unsigned p = s.push[it & 1u];
            sn += p & 0xffffu;
            cn += p >> 16;
            it++;
            continue;
        }
        if (sn == 0u) {
            // out of node pairs: a ticket, and while its slot is not there the candidates left
            if (tid == 0) {
                s.ticket = atomicAdd(&C->q_head, 1u);
                atomicAdd(&C->pool, ~0ull << 32);
            }
            unsigned state = 0;
            for (;;) {
                if (tid == 0) {
                    const unsigned t = s.ticket;
                    unsigned st = 0, seen = 0, rounds = 0;
                    for (unsigned spins = 0;;) {
                        if (t < nslots && ld_acq(B.qflag + t) == B.tag) {
                            st = 1u;
                            break;
                        }
                        if ((unsigned)(*(volatile unsigned long long*)&C->pool >> 32) == 0u - G) {
                            st = 2u;
                            break;
                        }
                        if (cn) break;  // candidates first
                        if (spins) __nanosleep(64);
                        if (++spins < kIdleSpins) continue;
                        const unsigned now = ld_vol(&C->starved);
                        if (now == seen || ++rounds > kIdleRounds) break;
                        seen = now;
                        spins = 0;
                    }
                    if (!st && !cn) {
                        atomicOr(&C->err, kErrTimeout);
                        st = 2u;
                    }
                    s.state = st;
                }
                __syncthreads();
                state = s.state;
                if (state == 1u || !cn) break;
                while (cn) {
                    const unsigned m = min(cn, kBlkThreads);
                    block_filter<F64, MULTI>(B, s, cn, m, decided, tested);
                    cn -= m;
                }
                if (state == 2u) break;
            }
            if (state == 2u) break;
            const uint4* const slot = B.queue + (size_t)s.ticket * kBlkUnits;
            const unsigned m = min(__ldcg(slot).w, kBlkUnits);
            if (tid < m) {
                const uint4 e = __ldcg(slot + tid);
                s.ring[tid] = make_uint2(e.y, e.z);
                if constexpr (MULTI) s.ring_job[tid] = e.x;
            }
            rb = 0;
            sn = m;
            __syncthreads();
            continue;
        }
        const unsigned take = min(sn, kBlkUnits);
        const bool have = unit < take;
        uint4 ent = make_uint4(0u, kEmpty, kEmpty, 0u);
        if (have) {
            const unsigned at = (rb + sn - 1u - unit) & (kBlkRing - 1u);
            const uint2 ab = s.ring[at];
            ent.y = ab.x;
            ent.z = ab.y;
            if constexpr (MULTI) ent.x = s.ring_job[at];
            visited += sub == 0u ? 1u : 0u;
        }
        sn -= take;
        // tickets and slots, looked at while the nodes load
        unsigned head = 0, tail = 0;
        if (tid == 0) {
            head = ld_vol(&C->q_head);
            tail = ld_vol(reinterpret_cast<const unsigned*>(&C->pool));
        }
        __syncthreads();  // the popped entries are read before the pushes reuse their places
        if (tid == 0) s.push[(it & 1u) ^ 1u] = 0u;  // read by all before this barrier
        unsigned fm = 0, cm = 0;
        uint32_t ca = kEmpty;
        if (__any_sync(0xffffffffu, have)) {
            block_expand<F64, MULTI>(B, s.x[tid >> 5], ent, have, sub, fm, cm, ca);
            // places of the lane's children: a warp scan of both counts in one word
            const unsigned mine = __popc(fm) + (__popc(cm) << 16);
            unsigned inc = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= (unsigned)o) inc += y;
            }
            unsigned old = 0;
            if (lane == 31u && inc) old = atomicAdd(&s.push[it & 1u], inc);
            old = __shfl_sync(0xffffffffu, old, 31) + inc - mine;
            unsigned f = rb + sn + (old & 0xffffu), c = cn + (old >> 16);
            for (unsigned left = fm | cm; left; left &= left - 1u) {  // two children at most, mostly
                const unsigned j = __ffs(left) - 1u;
                const uint32_t rB = s.x[tid >> 5].ref[(lane & 28u) + j];
                if ((cm >> j) & 1u) {
                    s.cand[c] = make_uint2(ca & ~kLeaf, rB & ~kLeaf);
                    if constexpr (MULTI) s.cand_job[c] = ent.x;
                    c++;
                } else {
                    s.ring[f & (kBlkRing - 1u)] = make_uint2(ca, rB);
                    if constexpr (MULTI) s.ring_job[f & (kBlkRing - 1u)] = ent.x;
                    f++;
                }
            }
        }
        if (tid == 0) {
            // tickets waiting; none where the pool is nearly full (every block may give 16 slots at once)
            const bool room = tail + 16u * G < nslots;
            s.hungry = room && (int)(head - tail) > 0 ? head - tail : 0u;
            if (!room && (int)(head - tail) > 0) atomicAdd(&C->starved, 1u);
        }
        __syncthreads();
        const unsigned p = s.push[it & 1u], hungry = s.hungry;
        sn += p & 0xffffu;
        cn += p >> 16;
        it++;
        if (hungry && sn > B.keep) {
            const unsigned m0 = sn - B.keep, d = min(min(hungry, 16u), (m0 + kBlkUnits - 1u) / kBlkUnits);
            const unsigned m = min(m0, d * kBlkUnits);
            block_give<F64, MULTI>(B, s, rb, m, d);
            rb += m;
            sn -= m;
        }
    }
    block_flush<F64, MULTI>(B, s, s.nres);
    block_stats(C, visited, decided, tested, it);
}

// ===========================================================================
// Exact stage and segments
// ===========================================================================
// Exact stage over the escalated pairs, grid-stride over the threads of the
// launch (nth a multiple of 32): intersecting pairs are appended to the results.
template <bool MULTI>
__device__ __forceinline__ void exact_stage(const Bufs& B, unsigned gtid, unsigned nth)
{
    Counters* C = B.cnt;
    const unsigned lane = threadIdx.x & 31;
    unsigned ne = ld_cg_u32(&C->esc);
    if (ne > B.cap_esc) ne = B.cap_esc;
    unsigned long long nexact = 0;
    for (unsigned base = gtid - lane; base < ne; base += nth) {
        const unsigned i = base + lane;
        const bool have = i < ne;
        bool yes = false;
        uint32_t ta = 0, tb = 0, job = 0;
        unsigned code = 0;
        if (have) {
            uint4 c = __ldcg(B.esc + i);
            job = c.x;
            const JobDev& J = job_at<MULTI>(B, job);
            double3 pts[6];
            load_tri<false>(J.A, J.pa, c.y, pts, &ta);
            load_tri<false>(J.B, J.pb, c.z, pts + 3, &tb);
            ExactSigns S{&C->err, 0ull};
            yes = decide_escalated(pts, B.precision == 0, &code, S);
            nexact += S.nexact;
        }
        unsigned pr = warp_append(yes, &C->res);
        if (yes) {
            const uint4 r = make_uint4(job, ta, tb, code);
            if (pr < B.cap_res) {
                B.res[pr] = r;
                if (B.fin.on) fin_insert<MULTI>(B, r, pr, B.fin.segments ? code_segments(code) : 1u);
            } else {
                atomicOr(&C->overflow, kOvfResExact);
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) nexact += __shfl_xor_sync(0xffffffffu, nexact, o);
    if (lane == 0 && nexact) atomicAdd(&C->exact_signs, nexact);
}

__global__ void __launch_bounds__(128) k_exact(Bufs B)
{
    exact_stage<true>(B, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

__device__ __forceinline__ void load_tri_orig(const MeshDev& M, const DevPose& P, uint32_t tri, double3* out)
{
    const uint32_t* t = M.tris + 3 * (size_t)tri;
    out[0] = world_vertex(M.verts, __ldg(t), P);
    out[1] = world_vertex(M.verts, __ldg(t + 1), P);
    out[2] = world_vertex(M.verts, __ldg(t + 2), P);
}

// The point of construction code `c` of a result: fast path on values in
// registers (vertices chosen by selects), the exact construction, which reloads
// the triangles, when the rounding test fails.
static __device__ __noinline__ bool result_point_exact(const JobDev& J, uint32_t a, uint32_t b, unsigned c,
                                                       unsigned drop, double3& q, unsigned long long* exact_points)
{
    double3 pts[6];
    load_tri_orig(J.A, J.pa, a, pts);
    load_tri_orig(J.B, J.pb, b, pts + 3);
    return code_point_exact(pts, c, drop, q, exact_points);
}
__device__ __forceinline__ bool result_point(const double3* P, const double3* Q, const JobDev& J, const uint4& rr,
                                             unsigned c, unsigned drop, double3& q, unsigned long long* exact_points)
{
    const double3 P0 = P[0], P1 = P[1], P2 = P[2], Q0 = Q[0], Q1 = Q[1], Q2 = Q[2];
    if (c < kCodePlane) {
        q = c < 3u ? sel3((int)c, P0, P1, P2) : sel3((int)c - 3, Q0, Q1, Q2);
        return true;
    }
    if (c < kCodeLine) {
        const unsigned e = (c - kCodePlane) >> 1;
        const bool onP = e < 3u, rev = (c & 1u) != 0u;
        const int i = (int)(onP ? e : e - 3u), j = i == 2 ? 0 : i + 1;
        const double3 T0 = onP ? P0 : Q0, T1 = onP ? P1 : Q1, T2 = onP ? P2 : Q2;
        const double3 U0 = onP ? Q0 : P0, U1 = onP ? Q1 : P1, U2 = onP ? Q2 : P2;
        if (construct_plane_fast(U0, U1, U2, sel3(rev ? j : i, T0, T1, T2), sel3(rev ? i : j, T0, T1, T2), q)) return true;
    } else {
        const unsigned n = (c - kCodeLine) >> 2;
        const bool onQ = ((c - kCodeLine) & 2u) != 0u, rev = ((c - kCodeLine) & 1u) != 0u;
        const int e1 = (int)(n / 3u), e2 = (int)(n % 3u), f1 = e1 == 2 ? 0 : e1 + 1, f2 = e2 == 2 ? 0 : e2 + 1;
        const double3 a1 = sel3(e1, P0, P1, P2), b1 = sel3(f1, P0, P1, P2);
        const double3 a2 = sel3(e2, Q0, Q1, Q2), b2 = sel3(f2, Q0, Q1, Q2);
        const double3 a = onQ ? a2 : a1, b = onQ ? b2 : b1;
        if (construct_line_fast(onQ ? a1 : a2, onQ ? b1 : b2, rev ? b : a, rev ? a : b, drop, q)) return true;
    }
    return result_point_exact(J, rr.y, rr.z, c, drop, q, exact_points);
}

// Segments of one result (up to 3, 6 doubles each, at o) from its construction
// code.  `per` threads (1 or 2, adjacent lanes) share it, thread `half`
// constructing the points half, half + per, ..
template <bool MULTI>
__device__ __forceinline__ void result_segments(const Bufs& B, const uint4& rr, double* o, unsigned half = 0u,
                                                unsigned per = 1u)
{
    Counters* C = B.cnt;
    const unsigned kind = rr.w & 3u, drop = (rr.w >> 2) & 3u;
    if (!kind) return;
    const JobDev& J = job_at<MULTI>(B, rr.x);
    double3 P[3], Q[3];
    load_tri_orig(J.A, J.pa, rr.y, P);
    load_tri_orig(J.B, J.pb, rr.z, Q);
    for (unsigned k = half; k < kind; k += per) {
        double3 q;
        if (!result_point(P, Q, J, rr, (rr.w >> (4u + 6u * k)) & 63u, drop, q, &C->exact_points))
            atomicOr(&C->err, kErrExactCapacity);
        // point k opens segment k; it ends the other segment it belongs to
        // (a point alone ends its own, of a triangle's three the one before)
        double* const x = o + 6u * (kind == 2u ? 0u : k) + (kind == 2u ? 3u * k : 0u);
        x[0] = q.x;
        x[1] = q.y;
        x[2] = q.z;
        if (kind != 2u) {
            double* const y = o + 6u * (kind == 1u ? 0u : (k + 2u) % 3u) + 3u;
            y[0] = q.x;
            y[1] = q.y;
            y[2] = q.z;
        }
    }
}

// The segments of every result (general path), a result per thread.  Bound by
// the FP64 pipe (double-double) and the gathers.  It classified the results
// without an endpoint pattern again, exactly: on two coplanar 512 x 512 grids
// (1.36 M results) that was 14.0 ms of instruction fetches and local memory;
// building from the construction code takes 0.27 ms.
__global__ void __launch_bounds__(128) k_segments(Bufs B, double* __restrict__ segs, uint32_t* __restrict__ nseg)
{
    Counters* C = B.cnt;
    const unsigned gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned nth = gridDim.x * blockDim.x;
    if (ld_cg_u32(&C->overflow)) return;
    unsigned nres = ld_cg_u32(&C->res);
    if (nres > B.cap_res) nres = B.cap_res;
    for (unsigned i = gtid; i < nres; i += nth) {
        const uint4 rr = __ldcg(B.res + i);
        nseg[i] = code_segments(rr.w);
        result_segments<true>(B, rr, segs + 18 * (size_t)i);
    }
}

// ===========================================================================
// Ordering: results sorted by (job, a, b) with an LSD radix sort whose sizes
// come from the device counters (no host round trip).  One kernel builds the
// keys and the digit histograms of every pass, one scans them, and each pass
// is one scatter kernel: tiles of 4096 items take their global offset per
// digit by decoupled look-back over the preceding tiles (bounded waits).
// The gather kernel applies the permutation and places the segments, finding
// its segment offset by the same look-back.
// ===========================================================================
constexpr int kOsThreads = 256;
constexpr int kOsItems = 16;
constexpr int kOsTile = kOsThreads * kOsItems;
constexpr int kOsWarps = kOsThreads / 32;
constexpr int kOsGatherTile = 1024;

__device__ __forceinline__ unsigned res_count(const Bufs& B)
{
    if (ld_cg_u32(&B.cnt->overflow)) return 0u;
    unsigned n = ld_cg_u32(&B.cnt->res);
    return n > B.cap_res ? B.cap_res : n;
}

__device__ __forceinline__ unsigned long long order_key(const uint4& r, const OrderBufs& O)
{
    return ((unsigned long long)r.x << (O.bits_a + O.bits_b)) | ((unsigned long long)r.y << O.bits_b) | r.z;
}

// Keys, identity values and the histograms of every digit pass; the last
// block to finish scans the histograms into digit bases (and clears them for
// the next call), so no separate scan launch is needed.
__global__ void __launch_bounds__(kOsThreads) k_os_hist(Bufs B, OrderBufs O)
{
    __shared__ unsigned h[kOsMaxPasses][256];
    __shared__ uint32_t sw[33];
    __shared__ unsigned s_last;
    const unsigned n = res_count(B);
    for (int p = 0; p < O.passes; p++) h[p][threadIdx.x] = 0;
    // look-back status of every pass and of the gather starts unset
    const unsigned ntiles = (n + kOsTile - 1) / kOsTile;
    const size_t nstat = (size_t)(O.passes + 1) * O.ntiles_cap * 256;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < nstat; k += (size_t)gridDim.x * blockDim.x) {
        const size_t t = (k / 256) % O.ntiles_cap;
        if (t < ntiles) O.status[k] = 0u;
    }
    const unsigned ngather = (n + kOsGatherTile - 1) / kOsGatherTile;
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k < ngather; k += gridDim.x * blockDim.x)
        O.gstatus[k] = 0u;
    if (blockIdx.x == 0 && threadIdx.x <= (unsigned)O.passes) O.tile_ctr[threadIdx.x] = 0u;
    __syncthreads();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned long long key = order_key(__ldcg(B.res + i), O);
        O.keys[0][i] = key;
        O.vals[0][i] = i;
        for (int p = 0; p < O.passes; p++) atomicAdd(&h[p][(unsigned)(key >> (8 * p)) & 255u], 1u);
    }
    __syncthreads();
    for (int p = 0; p < O.passes; p++)
        if (h[p][threadIdx.x]) atomicAdd(&O.hist[p * 256 + threadIdx.x], h[p][threadIdx.x]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(&O.tile_ctr[kOsMaxPasses + 1], 1u) == gridDim.x - 1) ? 1u : 0u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int p = 0; p < O.passes; p++) {
        const unsigned v = __ldcg(&O.hist[p * 256 + threadIdx.x]);
        unsigned tot;
        const unsigned ex = block_exclusive_scan(v, sw, &tot);
        O.base[p * 256 + threadIdx.x] = ex;
        O.hist[p * 256 + threadIdx.x] = 0u;
    }
    if (threadIdx.x == 0) O.tile_ctr[kOsMaxPasses + 1] = 0u;
}

__global__ void __launch_bounds__(kOsThreads) k_os_scatter(Bufs B, OrderBufs O, int pass)
{
    __shared__ unsigned wc[kOsWarps][256];
    __shared__ unsigned tile_base[256];
    __shared__ unsigned s_tile;
    const unsigned n = res_count(B);
    const unsigned ntiles = (n + kOsTile - 1) / kOsTile;
    if (threadIdx.x == 0) s_tile = atomicAdd(&O.tile_ctr[pass], 1u);
    __syncthreads();
    const unsigned tile = s_tile;
    if (tile >= ntiles) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int shift = 8 * pass;
    const unsigned long long* kin = O.keys[pass & 1];
    const uint32_t* vin = O.vals[pass & 1];
    unsigned long long* kout = O.keys[(pass + 1) & 1];
    uint32_t* vout = O.vals[(pass + 1) & 1];
    for (int d = lane; d < 256; d += 32) wc[w][d] = 0;
    __syncwarp();
    const unsigned seg = tile * kOsTile + w * 32 * kOsItems;
    unsigned long long key[kOsItems];
    uint32_t val[kOsItems], rank[kOsItems], dig[kOsItems];
    const unsigned lt = (1u << lane) - 1u;
    // all loads first (independent, in flight together), then the ranking
#pragma unroll
    for (int c = 0; c < kOsItems; c++) {
        const unsigned i = seg + c * 32 + lane;
        key[c] = i < n ? __ldcg(kin + i) : 0ull;
        val[c] = i < n ? __ldcg(vin + i) : 0u;
    }
#pragma unroll
    for (int c = 0; c < kOsItems; c++) {
        const unsigned i = seg + c * 32 + lane;
        const bool ok = i < n;
        const unsigned d = ok ? ((unsigned)(key[c] >> shift) & 255u) : 256u;
        dig[c] = d;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        rank[c] = ok ? wc[w][d] + __popc(peers & lt) : 0u;
        __syncwarp();
        if (ok && (peers & lt) == 0) wc[w][d] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    {
        const unsigned d = threadIdx.x;
        unsigned run = 0;
        for (int q = 0; q < kOsWarps; q++) {
            const unsigned t = wc[q][d];
            wc[q][d] = run;
            run += t;
        }
        unsigned excl;
        lookback(O.status + (size_t)pass * O.ntiles_cap * 256 + d, tile, 256, run, &excl, &B.cnt->err);
        tile_base[d] = O.base[pass * 256 + d] + excl;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < kOsItems; c++) {
        const unsigned d = dig[c];
        if (d < 256u) {
            const unsigned pos = tile_base[d] + wc[w][d] + rank[c];
            kout[pos] = key[c];
            vout[pos] = val[c];
        }
    }
}

// sorted position k -> pairs_out[k], job_out[k]; the segments of the pair go
// to the prefix sum of the segment counts (tile look-back).  One item per
// thread, so every load of a thread is issued at once.  A tile's segments are
// one run of the output: it is written 16 bytes a lane from a list of their
// sources.  What fits into the host's arrays goes there as well, at the link's
// rate and at the result's own size (the copies that did this afterwards moved
// the size guessed before the call, a quarter more than the last result).
__global__ void __launch_bounds__(kOsGatherTile) k_os_gather(Bufs B, OrderBufs O, const double* __restrict__ segs,
                                                             const uint32_t* __restrict__ nseg, int32_t* pairs_out,
                                                             uint32_t* job_out, double* segs_out,
                                                             int32_t* segpair_out, HostOut H, int want_segments, int sorted)
{
    __shared__ uint32_t sw[33];
    __shared__ unsigned s_tile, s_base;
    __shared__ uint32_t s_src[3 * kOsGatherTile];  // a segment's pair, its place in the results
    __shared__ uint16_t s_at[3 * kOsGatherTile];   // ... and its place in the tile, 4 x that + the segment's number
    const unsigned n = res_count(B);
    const unsigned ntiles = (n + kOsGatherTile - 1) / kOsGatherTile;
    if (threadIdx.x == 0) s_tile = atomicAdd(&O.tile_ctr[O.passes], 1u);
    __syncthreads();
    const unsigned tile = s_tile;
    if (tile >= ntiles) return;
    const unsigned k0 = tile * kOsGatherTile, k = k0 + threadIdx.x;
    const bool ok = k < n;
    const unsigned src = ok ? (sorted ? __ldcg(O.vals[O.passes & 1] + k) : k) : 0u;
    const unsigned c = (ok && want_segments) ? __ldcg(nseg + src) : 0u;
    const uint4 r = ok ? __ldcg(B.res + src) : make_uint4(0u, 0u, 0u, 0u);
    unsigned tot;
    const unsigned ex = block_exclusive_scan(c, sw, &tot);
    if (threadIdx.x == 0) {
        unsigned excl;
        lookback(O.gstatus, tile, 1, tot, &excl, &B.cnt->err);
        s_base = excl;
        if (tile == ntiles - 1) B.cnt->nseg = excl + tot;
    }
    for (unsigned q = 0; q < c; q++) {  // c <= 3
        s_src[ex + q] = src;
        s_at[ex + q] = (uint16_t)(4u * threadIdx.x + q);
    }
    __syncthreads();
    if (ok) {
        const int2 p = make_int2((int32_t)r.y, (int32_t)r.z);
        reinterpret_cast<int2*>(pairs_out)[k] = p;
        job_out[k] = r.x;
        if (k < H.pairs_cap) {
            reinterpret_cast<int2*>(H.pairs)[k] = p;
            if (H.job) H.job[k] = r.x;
        }
    }
    const size_t base = s_base;
#pragma unroll 3
    for (unsigned j = threadIdx.x; j < 3u * tot; j += kOsGatherTile) {
        const unsigned s = j / 3u, part = j - 3u * s;
        const double2 v = __ldcg(reinterpret_cast<const double2*>(segs + 18 * (size_t)s_src[s] + 6 * (s_at[s] & 3u)) + part);
        reinterpret_cast<double2*>(segs_out)[3 * base + j] = v;
        if (base + s < H.segs_cap) reinterpret_cast<double2*>(H.segs)[3 * base + j] = v;
    }
    for (unsigned s = threadIdx.x; s < tot; s += kOsGatherTile) {
        const int32_t at = (int32_t)(k0 + (s_at[s] >> 2));
        segpair_out[base + s] = at;
        if (base + s < H.segs_cap) H.segpair[base + s] = at;
    }
}

size_t order_scratch_bytes(uint32_t cap, int passes)
{
    size_t ntiles = (cap + kOsTile - 1) / kOsTile;
    return 2 * sizeof(unsigned long long) * (size_t)cap + 2 * sizeof(uint32_t) * (size_t)cap +
           sizeof(uint32_t) * ((size_t)(passes + 1) * ntiles * 256 + 2 * kOsMaxPasses * 256 + kOsMaxPasses + 2 +
                               (size_t)cap / kOsGatherTile + 1 + kOrderSmallBlocks) +
           8192;
}

OrderBufs make_order_bufs(void* scratch, uint32_t cap, int bits_a, int bits_b, int bits_job)
{
    OrderBufs O;
    O.bits_a = bits_a;
    O.bits_b = bits_b;
    O.passes = (bits_a + bits_b + bits_job + 7) / 8;
    O.ntiles_cap = (cap + kOsTile - 1) / kOsTile;
    char* p = (char*)scratch;
    auto take = [&](size_t bytes) {
        char* q = p;
        p += (bytes + 255) & ~(size_t)255;
        return (void*)q;
    };
    O.keys[0] = (unsigned long long*)take(sizeof(unsigned long long) * cap);
    O.keys[1] = (unsigned long long*)take(sizeof(unsigned long long) * cap);
    O.vals[0] = (uint32_t*)take(sizeof(uint32_t) * cap);
    O.vals[1] = (uint32_t*)take(sizeof(uint32_t) * cap);
    // fixed layout (independent of the pass count of the call): the histogram
    // must stay at the same, zeroed, address from one call to the next
    O.status = (uint32_t*)take(sizeof(uint32_t) * (size_t)(kOsMaxPasses + 1) * O.ntiles_cap * 256);
    O.gstatus = (uint32_t*)take(sizeof(uint32_t) * ((size_t)cap / kOsGatherTile + 1));
    O.hist = (uint32_t*)take(sizeof(uint32_t) * kOsMaxPasses * 256);
    O.base = (uint32_t*)take(sizeof(uint32_t) * kOsMaxPasses * 256);
    O.tile_ctr = (uint32_t*)take(sizeof(uint32_t) * (kOsMaxPasses + 2));
    O.tile_tot = (uint32_t*)take(sizeof(uint32_t) * kOrderSmallBlocks);
    return O;
}

cudaError_t launch_order_gather(const Bufs& b, const OrderBufs& O, bool sort, const double* segs,
                                const uint32_t* nseg, int32_t* pairs_out, uint32_t* job_out, double* segs_out,
                                int32_t* segpair_out, const HostOut& host, bool want_segments, const LaunchCfg& cfg,
                                cudaStream_t st)
{
    const unsigned tiles = O.ntiles_cap ? O.ntiles_cap : 1u;
    OrderBufs o = O;
    if (!sort) o.passes = 0;
    k_os_hist<<<cfg.sms * 2, kOsThreads, 0, st>>>(b, o);
    note_launches(1);
    if (sort) {
        for (int p = 0; p < o.passes; p++) {
            k_os_scatter<<<tiles, kOsThreads, 0, st>>>(b, o, p);
            note_launches(1);
        }
    }
    const unsigned gtiles = O.ntiles_cap * (kOsTile / kOsGatherTile);
    k_os_gather<<<gtiles, kOsGatherTile, 0, st>>>(b, o, segs, nseg, pairs_out, job_out, segs_out, segpair_out,
                                                  host, want_segments ? 1 : 0, sort ? 1 : 0);
    note_launches(1);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Small-count ordering (up to kOrderSmallMax results) in cooperative launches:
// one, or a rank launch and a place launch when the segments are built on
// another stream in between.
//
// At a few thousand to a few tens of thousands of results the radix passes
// above are bound by launch and look-back latency, not by bytes.  Here each of
// kOrderSmallBlocks blocks sorts one run of kOrderSmallRun keys, one key per
// thread, with a bitonic network whose partner distances below 32 are warp
// shuffles (only the longer ones go through shared memory).  The (job, a, b)
// keys are unique, so the final position of a key is its rank in its own run
// plus its lower bound in every other run: each block copies all sorted runs
// into shared memory and searches them there.  A third phase gathers the pairs
// and places the segments (block scan + the preceding runs' totals).  The
// phases are separated by grid barriers; the launch is cooperative, so all
// blocks are co-resident, and every barrier wait is bounded all the same.
// ---------------------------------------------------------------------------
constexpr int kOrderSmallThreads = kOrderSmallRun;  // one key per thread
constexpr size_t kOrderSmallDyn = sizeof(unsigned long long) * kOrderSmallMax;  // all runs, phase 2

// Arrive at grid barrier `k` (1-based) of the launch; waits bounded.  On a spent
// wait the error bit is set and later barriers of the block no longer wait.
__device__ __forceinline__ void grid_barrier(unsigned* ctr, unsigned k, unsigned* err, unsigned* s_ok)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(ctr, 1u);
        const unsigned target = k * gridDim.x;
        unsigned long long spins = 0;
        while (*s_ok && ld_vol(ctr) < target) {
            if (++spins > kLookbackSpins) {
                atomicOr(err, kErrTimeout);
                *s_ok = 0u;
                break;
            }
            __nanosleep(64);
        }
        __threadfence();
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kOrderSmallThreads, 1)
    k_order_small(Bufs B, OrderBufs O, const double* __restrict__ segs, const uint32_t* __restrict__ nseg,
                  int32_t* pairs_out, uint32_t* job_out, double* segs_out, int32_t* segpair_out, int want_segments,
                  int sorted, unsigned phases, unsigned bar0)
{
    extern __shared__ unsigned long long allk[];  // every sorted run (phase 2)
    __shared__ unsigned long long sk[kOrderSmallRun];
    __shared__ uint32_t sv[kOrderSmallRun];
    __shared__ uint32_t sw[33];
    __shared__ unsigned s_ok, s_base;
    Counters* C = B.cnt;
    const unsigned n = res_count(B);
    if (n > kOrderSmallMax) {  // same decision in every block: no barrier is reached
        if (blockIdx.x == 0 && threadIdx.x == 0) C->order_redo = kRedoCount;
        return;
    }
    if (threadIdx.x == 0) s_ok = 1u;
    const unsigned tid = threadIdx.x;
    const unsigned nruns = (n + kOrderSmallRun - 1) / kOrderSmallRun;
    const unsigned t = blockIdx.x;
    const unsigned base = t * kOrderSmallRun;
    const unsigned len = t < nruns ? min((unsigned)kOrderSmallRun, n - base) : 0u;
    uint32_t* perm = O.vals[1];
    unsigned bar = bar0;  // grid barriers already passed by an earlier launch of this call
    if (sorted && (phases & kOrderRank)) {
        // ---- phase 1: sort this block's run (padding keys sort last) ----
        unsigned long long key = tid < len ? order_key(__ldcg(B.res + base + tid), O) : ~0ull;
        uint32_t val = tid < len ? base + tid : 0xffffffffu;
        if (len > 1) {  // uniform in the block
            for (unsigned k = 2; k <= (unsigned)kOrderSmallRun; k <<= 1)
                for (unsigned j = k >> 1; j > 0; j >>= 1) {
                    unsigned long long pk;
                    uint32_t pv;
                    if (j >= 32u) {
                        __syncthreads();  // the previous stage's reads are done
                        sk[tid] = key;
                        sv[tid] = val;
                        __syncthreads();
                        pk = sk[tid ^ j];
                        pv = sv[tid ^ j];
                    } else {
                        pk = __shfl_xor_sync(0xffffffffu, key, j);
                        pv = __shfl_xor_sync(0xffffffffu, val, j);
                    }
                    // the lower index of an ascending pair (or the upper of a
                    // descending one) keeps the smaller key
                    const bool keep_min = ((tid & j) == 0u) == ((tid & k) == 0u);
                    if (keep_min ? (pk < key) : (pk > key)) {
                        key = pk;
                        val = pv;
                    }
                }
        }
        if (tid < len) O.keys[0][base + tid] = key;
        grid_barrier(&C->obar, ++bar, &C->err, &s_ok);
        // ---- phase 2: final position = own rank + lower bounds in the other runs ----
        // all runs into shared memory: every copy is issued before any is
        // waited for (asynchronous 16-byte copies through L2 only: the key
        // buffer is rewritten by every call, so no L1 copy of it may be used;
        // an odd last key is loaded the same way, through L2)
        for (unsigned c = tid; c < n / 2u; c += kOrderSmallThreads) {
            const unsigned dst = (unsigned)__cvta_generic_to_shared(allk + 2u * c);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(O.keys[0] + 2u * c)
                         : "memory");
        }
        if ((n & 1u) && tid == 0) allk[n - 1u] = __ldcg(O.keys[0] + (n - 1u));
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        // A warp's keys are consecutive in its sorted run, so in another run
        // their lower bounds lie between those of its first and its last key.
        // Two lanes per run find that bracket (four runs at once); every lane
        // then counts the keys below its own inside the bracket, held in the
        // warp's registers and searched with shuffles, or (a bracket wider
        // than two chunks) with its own search of the bracket.
        const unsigned lane = tid & 31u, wbase = tid & ~31u;
        if (wbase < len) {  // warp-uniform
            const unsigned wlast = min(len - wbase, 32u) - 1u;  // the warp's last key
            const unsigned long long kf = __shfl_sync(0xffffffffu, key, 0);
            const unsigned long long kl = __shfl_sync(0xffffffffu, key, wlast);
            unsigned pos = tid;
            for (unsigned s0 = 0; s0 < nruns; s0 += 4) {
                // lanes 2r and 2r + 1: lower bounds of the first and last key in run s0 + r
                unsigned a = 0, b = 0;
                if (lane < 8u) {
                    const unsigned sr = s0 + (lane >> 1);
                    if (sr < nruns && sr != t) {
                        a = sr * kOrderSmallRun;
                        b = a + min((unsigned)kOrderSmallRun, n - a);
                    }
                    const unsigned long long q = (lane & 1u) ? kl : kf;
                    while (a < b) {
                        const unsigned mid = (a + b) >> 1;
                        if (allk[mid] < q) a = mid + 1u;
                        else b = mid;
                    }
                }
#pragma unroll
                for (unsigned r = 0; r < 4u; r++) {
                    const unsigned sr = s0 + r;
                    if (sr >= nruns || sr == t) continue;  // warp-uniform
                    const unsigned L = sr * kOrderSmallRun;
                    const unsigned lo = __shfl_sync(0xffffffffu, a, 2u * r);
                    const unsigned hi = __shfl_sync(0xffffffffu, a, 2u * r + 1u);
                    unsigned c = 0;
                    if (hi - lo <= 64u) {
                        for (unsigned w0 = lo; w0 < hi; w0 += 32u) {
                            const unsigned cnt = min(32u, hi - w0);
                            const unsigned long long v = lane < cnt ? allk[w0 + lane] : ~0ull;
                            unsigned first = 0, count = cnt;  // lower bound of key among v[0 .. cnt)
                            for (int st = 0; st < 6; st++) {  // 2^5 < 32 + 1 <= 2^6
                                const unsigned half = count >> 1;
                                const unsigned long long vm = __shfl_sync(0xffffffffu, v, (first + half) & 31u);
                                if (count > 0u) {
                                    if (vm < key) {
                                        first += half + 1u;
                                        count -= half + 1u;
                                    } else {
                                        count = half;
                                    }
                                }
                            }
                            c += first;
                        }
                    } else {
                        unsigned x = lo, y = hi;
                        while (x < y) {
                            const unsigned mid = (x + y) >> 1;
                            if (allk[mid] < key) x = mid + 1u;
                            else y = mid;
                        }
                        c = x - lo;
                    }
                    pos += lo - L + c;
                }
            }
            if (lane <= wlast && pos < n) perm[pos] = val;
        }
        // the placing phase reads every block's perm entries; a separate
        // placing launch is ordered after this one by the kernel boundary
        if (phases & kOrderPlace) grid_barrier(&C->obar, ++bar, &C->err, &s_ok);
    }
    if (!(phases & kOrderPlace)) return;
    // ---- phase 3: gather pairs, place segments (one sorted position per thread) ----
    const unsigned k = base + tid;
    const bool ok = tid < len;
    unsigned src = ok ? (sorted ? __ldcg(perm + k) : k) : 0u;
    if (src >= n) src = 0u;
    const unsigned cnt = (ok && want_segments) ? __ldcg(nseg + src) : 0u;
    const uint4 rr = ok ? __ldcg(B.res + src) : make_uint4(0u, 0u, 0u, 0u);
    unsigned tot;
    const unsigned ex = block_exclusive_scan(cnt, sw, &tot);
    if (tid == 0) O.tile_tot[t] = tot;
    grid_barrier(&C->obar, ++bar, &C->err, &s_ok);
    if (tid < 32u) {
        // the preceding blocks' totals, loaded by one warp at once and summed by shuffles
        static_assert(kOrderSmallBlocks <= 32, "one warp sums the block totals");
        unsigned v = tid < t ? __ldcg(O.tile_tot + tid) : 0u;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (tid == 0) {
            s_base = v;
            if (nruns && t == nruns - 1) C->nseg = v + tot;
        }
    }
    __syncthreads();
    if (!ok) return;
    pairs_out[2 * (size_t)k] = (int32_t)rr.y;
    pairs_out[2 * (size_t)k + 1] = (int32_t)rr.z;
    job_out[k] = rr.x;
    const unsigned off = s_base + ex;
    for (unsigned e = 0; e < cnt; e++) {
        const double2* sp = reinterpret_cast<const double2*>(segs + 18 * (size_t)src + 6 * e);
        double2* dp = reinterpret_cast<double2*>(segs_out + 6 * (size_t)(off + e));
        dp[0] = __ldcg(sp);
        dp[1] = __ldcg(sp + 1);
        dp[2] = __ldcg(sp + 2);
        segpair_out[off + e] = (int32_t)k;
    }
}

cudaError_t launch_order_small(const Bufs& b, const OrderBufs& O, bool sort, const double* segs,
                               const uint32_t* nseg, int32_t* pairs_out, uint32_t* job_out, double* segs_out,
                               int32_t* segpair_out, bool want_segments, cudaStream_t st)
{
    return launch_order_small_phases(b, O, sort, segs, nseg, pairs_out, job_out, segs_out, segpair_out,
                                     want_segments, kOrderRank | kOrderPlace, st);
}

cudaError_t launch_order_small_phases(const Bufs& b, const OrderBufs& O, bool sort, const double* segs,
                                      const uint32_t* nseg, int32_t* pairs_out, uint32_t* job_out, double* segs_out,
                                      int32_t* segpair_out, bool want_segments, unsigned phases, cudaStream_t st)
{
    if (!sort) phases &= ~kOrderRank;  // nothing to rank: results keep their order
    if (!phases) return cudaSuccess;
    const size_t dyn = (phases & kOrderRank) ? kOrderSmallDyn : 0;
    // the shared-memory opt-in is a per-device function attribute: set it once per device
    static std::atomic<uint64_t> attr_done{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? (1ull << dev) : 0ull;
    if (!bit || !(attr_done.load(std::memory_order_acquire) & bit)) {
        e = cudaFuncSetAttribute((const void*)k_order_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kOrderSmallDyn);
        if (e != cudaSuccess) return e;
        attr_done.fetch_or(bit, std::memory_order_acq_rel);
    }
    Bufs bb = b;
    OrderBufs oo = O;
    const double* a_segs = segs;
    const uint32_t* a_nseg = nseg;
    int ws = want_segments ? 1 : 0, so = sort ? 1 : 0;
    // a ranking launch without the placing phase passes one grid barrier; a
    // placing launch that follows it in the same call counts its barrier after it
    unsigned ph = phases, b0 = (sort && !(phases & kOrderRank)) ? 1u : 0u;
    void* args[] = {&bb, &oo, &a_segs, &a_nseg, &pairs_out, &job_out, &segs_out, &segpair_out, &ws, &so, &ph, &b0};
    e = cudaLaunchCooperativeKernel((const void*)k_order_small, dim3(kOrderSmallBlocks), dim3(kOrderSmallThreads),
                                    args, dyn, st);
    note_launches(1);
    return e;
}

// ===========================================================================
// Post-traversal work of a call in one launch (sorted output, up to kFinMax
// results, keys of at most 63 bits).  The traversal has put every result's key
// into its partition (fin_insert), so the partition counts are complete when
// the launch begins and no block waits for another:
//   phase 0  only when pairs were escalated: the exact stage, whose results join
//            their partitions, and a grid barrier;
//   phase 1  a block owns a run of consecutive sorted positions.  It scans all
//            partition counts (16 KB, every block by itself: cheaper than a
//            barrier), gathers the partitions that meet its run and ranks their
//            keys (counting the smaller ones; a partition over kFinRank keys is
//            sorted in shared memory);
//   phase 2  two adjacent threads construct each result's two endpoints, and the
//            run's pairs and segments go out in order, as whole lines, straight
//            into the caller's pinned result block (device memory when the
//            result outgrew it).  The last block copies the counters there too.
// It is cooperative for the barrier of phase 0 and a programmatic dependent of
// the traversal: it waits for that grid (griddepcontrol.wait) before anything
// else.  The counters and partition counts of the next call are cleared here
// (each call uses the other one of two sets), so a call needs no memset and no
// device-to-host copy.  A call over kFinMax results or with a partition over
// kFinBig keys is refused (Counters::order_redo, decided alike in every block).
//
// What bounds it: latency, the chain of one block's scan, gather, ranking and one
// result's construction (about 1,400 instructions an endpoint) with barriers
// between (at 12 k results 23 stalled warps per issue at barriers, issue 9 % and
// FP64 pipe 5 % busy), and, for larger results, the PCIe writes.  Its predecessor inserted the keys itself (a barrier, one block's scan,
// a release; partitions over 32 keys searched a common overflow list) and five
// copies followed it.  Launch to end: 868 results 14.5 -> 10.1 us, 12,245 results
// clustered in index 33 -> 24 us with their 735 KB written to the host; the whole
// call of two UV spheres of 1,216 triangles 81 -> 58 us, of two 1.3M-triangle
// meshes 153 -> 115 us.
// ===========================================================================
constexpr int kFinThreads = 256;
constexpr unsigned kFinRun = 1024;  // most positions of a block (two blocks per SM fit with it)
constexpr unsigned kFinPart = 256;  // results constructed and written at a time
constexpr unsigned kFinRank = 256;  // keys of a partition ranked by counting; larger ones are sorted
constexpr unsigned kFinKeys = kFinRun + 2 * kFinBig;  // a run meets at most two partitions that it does not fill
static_assert(kFinParts == 16 * kFinThreads, "a thread scans 16 partitions");
static_assert(kFinMax <= (1u << 20) && kFinParts <= (1 << 12), "slot and partition share a word");
static_assert(kFinMax <= (1u << 30), "a bucket value holds the result index below bit 30");

struct FinShared {
    uint32_t koff[kFinParts + 4];  // key offsets of the partitions
    uint32_t soff[kFinParts + 4];  // segments beyond one per key before them (only with odd results)
    union {
        struct {
            unsigned long long key[kFinKeys];
            uint32_t val[kFinKeys];
        } g;                                  // gathered keys
        double seg[kFinPart * 3 * 6];         // segments on their way out, in order
    } u;
    unsigned long long skey[kFinRun];  // the run's keys in order, their values and segment offsets
    uint32_t sval[kFinRun];
    uint32_t sseg[kFinRun];
    uint32_t warp[2][kFinThreads / 32];
    uint32_t big[32];
    unsigned nbig, ok, last;
};

__device__ __forceinline__ void fin_stamp(Counters* C, int k)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) C->fin_ns[k] = globaltimer_ns();
}

// Block end: the last block to end stamps the launch's end and copies the
// counters to the host.
__device__ __forceinline__ void fin_end(Counters* C, Counters* host, FinShared& s)
{
    __syncthreads();
    if (threadIdx.x == 0) s.last = arrive_acq_rel(&C->fin_done) == gridDim.x - 1u ? 1u : 0u;
    __syncthreads();
    if (!s.last) return;
    if (threadIdx.x == 0) C->fin_ns[4] = globaltimer_ns();
    __syncthreads();
    for (unsigned w = threadIdx.x; w < sizeof(Counters) / 4u; w += kFinThreads)
        reinterpret_cast<unsigned*>(host)[w] = __ldcg(reinterpret_cast<const unsigned*>(C) + w);
}

// Exclusive scan of the partition counts c (16 per thread) into `out`; returns
// the total.
__device__ __forceinline__ uint32_t fin_scan(const uint4 (&c)[4], uint32_t* out, uint32_t* warp)
{
    const unsigned tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    uint32_t v[16] = {c[0].x, c[0].y, c[0].z, c[0].w, c[1].x, c[1].y, c[1].z, c[1].w,
                      c[2].x, c[2].y, c[2].z, c[2].w, c[3].x, c[3].y, c[3].z, c[3].w};
    uint32_t sum = 0;
#pragma unroll
    for (int q = 0; q < 16; q++) {
        const uint32_t t = v[q];
        v[q] = sum;
        sum += t;
    }
    uint32_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (unsigned)o) inc += y;
    }
    if (lane == 31u) warp[w] = inc;
    __syncthreads();
    uint32_t before = inc - sum, total = 0;
#pragma unroll
    for (unsigned q = 0; q < kFinThreads / 32; q++) {
        if (q < w) before += warp[q];
        total += warp[q];
    }
    uint4* o4 = reinterpret_cast<uint4*>(out + 16 * tid);
#pragma unroll
    for (int q = 0; q < 4; q++)
        o4[q] = make_uint4(before + v[4 * q], before + v[4 * q + 1], before + v[4 * q + 2], before + v[4 * q + 3]);
    if (tid == 0) out[kFinParts] = total;
    __syncthreads();
    return total;
}

// The partition that holds sorted position x (koff[p] <= x < koff[p + 1]).
__device__ __forceinline__ unsigned fin_part(const uint32_t* koff, unsigned x)
{
    unsigned lo = 0, hi = kFinParts;  // koff[lo] <= x < koff[hi]
#pragma unroll
    for (int k = 0; k < kFinPartBits; k++) {
        const unsigned mid = (lo + hi) >> 1;
        if (koff[mid] <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

template <bool MULTI>
__global__ void __launch_bounds__(kFinThreads, 2) k_finish(const __grid_constant__ Bufs B, const __grid_constant__ FinArgs F)
{
    wait_prior_grid();  // the traversal's results are complete and visible
    extern __shared__ __align__(16) unsigned char fin_dyn[];
    FinShared& s = *reinterpret_cast<FinShared*>(fin_dyn);
    Counters* C = B.cnt;
    const unsigned tid = threadIdx.x;
    const unsigned gtid = blockIdx.x * kFinThreads + tid, nth = gridDim.x * kFinThreads;
    if (tid == 0) {
        s.ok = 1u;
        s.nbig = 0u;
    }
    fin_stamp(C, 0);
    // the next call's counters and partition counts
    for (unsigned w = gtid; w < 2u * kFinParts / 4u; w += nth) reinterpret_cast<uint4*>(F.next_count)[w] = make_uint4(0u, 0u, 0u, 0u);
    if (gtid < sizeof(Counters) / 8u) reinterpret_cast<unsigned long long*>(F.next_cnt)[gtid] = 0ull;
    // everything the scan needs, at once; final unless pairs were escalated
    const uint4* const count4 = reinterpret_cast<const uint4*>(B.fin.count) + 4 * tid;
    uint4 c4[4];
#pragma unroll
    for (int q = 0; q < 4; q++) c4[q] = __ldcg(count4 + q);
    unsigned n = ld_cg_u32(&C->res), over = ld_cg_u32(&C->fin_over);
    const unsigned esc = ld_cg_u32(&C->esc);
    // the traversal's overflows, final at launch: the call reruns with larger buffers.
    // (Not the exact stage's: a block that began late would see another block's,
    // leave here and be missed at the barrier below.)
    if (ld_cg_u32(&C->overflow) & ~kOvfResExact) {
        fin_end(C, F.host_cnt, s);
        return;
    }
    bool odd = false;
    // ---- phase 0: exact stage ----
    if (esc) {
        exact_stage<MULTI>(B, gtid, nth);
        grid_barrier(&C->obar, 1u, &C->err, &s.ok);
        if (ld_cg_u32(&C->overflow)) {  // read after the barrier: alike in every block
            fin_end(C, F.host_cnt, s);
            return;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) c4[q] = __ldcg(count4 + q);
        n = ld_cg_u32(&C->res);
        over = ld_cg_u32(&C->fin_over);
        odd = ld_cg_u32(&C->odd) != 0u;
    }
    fin_stamp(C, 1);
    if (n > kFinMax || n > kFinRun * gridDim.x) {
        if (blockIdx.x == 0 && tid == 0) C->order_redo = kRedoCount;
        fin_end(C, F.host_cnt, s);
        return;
    }
    // ---- phase 1: this block's run of sorted positions [lo, hi) ----
    // runs of at least 16 results (one warp's, two lanes each)
    const unsigned run = max(16u, (n + gridDim.x - 1u) / gridDim.x);
    const unsigned lo = blockIdx.x * run, hi = min(n, lo + run);
    if (lo >= n && blockIdx.x != 0u) {
        fin_end(C, F.host_cnt, s);
        return;
    }
    unsigned most = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) most = max(most, max(max(c4[q].x, c4[q].y), max(c4[q].z, c4[q].w)));
    const bool crowded = __syncthreads_or(most > (unsigned)kFinBig);
    if (crowded || over > (unsigned)kFinOverflow) {
        if (blockIdx.x == 0 && tid == 0) C->order_redo = crowded ? kRedoCrowded : kRedoSpilled;
        fin_end(C, F.host_cnt, s);
        return;
    }
    const uint32_t have = fin_scan(c4, s.koff, s.warp[0]);
    uint32_t nseg = F.want_segments ? have : 0u;
    if (odd) {
        const uint4* const extra4 = reinterpret_cast<const uint4*>(B.fin.extra) + 4 * tid;
        uint4 e4[4];
#pragma unroll
        for (int q = 0; q < 4; q++) e4[q] = __ldcg(extra4 + q);
        nseg += fin_scan(e4, s.soff, s.warp[1]);
    }
    // into the caller's block where it fits, else into device memory
    const bool fits = n <= F.host_pairs && nseg <= F.host_segs;
    if (blockIdx.x == 0u && tid == 0) C->nseg = nseg;
    if (lo >= n || have != n || (!fits && n > F.cap)) {  // no result; or (after a spent wait only) inconsistent counts
        fin_end(C, F.host_cnt, s);
        return;
    }
    const unsigned p0 = fin_part(s.koff, lo), p1 = fin_part(s.koff, hi - 1u) + 1u;
    const unsigned base = s.koff[p0], m = min(s.koff[p1] - base, kFinKeys);
    bool spill = false;
    for (unsigned t = tid; t < m; t += kFinThreads) {
        const unsigned part = fin_part(s.koff, base + t), slot = base + t - s.koff[part];
        if (slot < (unsigned)B.fin.bucket) {
            s.u.g.key[t] = __ldcg(B.fin.bkey + (size_t)part * B.fin.bucket + slot);
            s.u.g.val[t] = __ldcg(B.fin.bval + (size_t)part * B.fin.bucket + slot);
        } else {
            spill = true;
        }
        if (slot == kFinRank) {  // one of its keys lists a partition that is sorted
            const unsigned at = atomicAdd(&s.nbig, 1u);
            if (at < 32u) s.big[at] = part;
        }
    }
    if (__syncthreads_or(spill)) {
        // keys beyond a bucket: found on the overflow list, their slots with them
        for (unsigned t = tid; t < over; t += kFinThreads) {
            const unsigned long long key = __ldcg(B.fin.okey + t);
            const uint2 v = __ldcg(B.fin.oval + t);
            const unsigned part = v.y >> 20;
            if (part >= p0 && part < p1) {
                const unsigned at = s.koff[part] - base + (v.y & 0xfffffu);
                if (at < m) {
                    s.u.g.key[at] = key;
                    s.u.g.val[at] = v.x;
                }
            }
        }
        __syncthreads();
    }
    if (s.nbig) {
        const unsigned nbig = min(s.nbig, 32u);
        for (unsigned q = 0; q < nbig; q++) {
            // bitonic sort of one partition, every comparison ascending (the first
            // step of a merge mirrors), so keys past its end need not exist
            const unsigned part = s.big[q], off = s.koff[part] - base;
            const unsigned c = min(s.koff[part + 1u] - s.koff[part], m - off);
            unsigned long long* const kk = s.u.g.key + off;
            uint32_t* const vv = s.u.g.val + off;
            unsigned pow = 1;
            while (pow < c) pow <<= 1;
            for (unsigned w = 2; w <= pow; w <<= 1)
                for (unsigned j = w >> 1; j > 0; j >>= 1) {
                    for (unsigned t = tid; t < pow; t += kFinThreads) {
                        const unsigned u = j == (w >> 1) ? (t ^ (w - 1u)) : (t ^ j);
                        if (u > t && u < c && kk[t] > kk[u]) {
                            const unsigned long long x = kk[t];
                            kk[t] = kk[u];
                            kk[u] = x;
                            const uint32_t y = vv[t];
                            vv[t] = vv[u];
                            vv[u] = y;
                        }
                    }
                    __syncthreads();
                }
        }
    }
    // ranks: the keys of the run to their places
    for (unsigned t = tid; t < m; t += kFinThreads) {
        const unsigned part = fin_part(s.koff, base + t), off = s.koff[part] - base;
        const unsigned c = min(s.koff[part + 1u] - s.koff[part], m - off);
        const unsigned long long key = s.u.g.key[t];
        const uint32_t val = s.u.g.val[t];
        unsigned rank = 0, pre = 0;
        if (c > kFinRank) {  // sorted above
            rank = t - off;
            if (odd)
                for (unsigned q = 0; q < rank; q++) pre += s.u.g.val[off + q] >> 30;
        } else if (odd) {
            for (unsigned q = 0; q < c; q++)
                if (s.u.g.key[off + q] < key) {
                    rank++;
                    pre += s.u.g.val[off + q] >> 30;
                }
        } else {
            for (unsigned q = 0; q < c; q++) rank += s.u.g.key[off + q] < key ? 1u : 0u;
        }
        const unsigned pos = base + off + rank;
        if (pos >= lo && pos < hi) {
            s.skey[pos - lo] = key;
            s.sval[pos - lo] = val;
            s.sseg[pos - lo] = odd ? s.koff[part] + s.soff[part] + pre : pos;
        }
    }
    __syncthreads();  // the gathered keys are done with: their place takes the segments
    fin_stamp(C, 2);
    // ---- phase 2: constructions, and the run out in order ----
    const unsigned cnt = hi - lo;
    const unsigned idx_mask = (1u << 30) - 1u;
    int32_t* const pairs = fits ? F.h_pairs : F.pairs_out;
    {
        const unsigned long long ma = (1ull << B.fin.bits_a) - 1ull, mb = (1ull << B.fin.bits_b) - 1ull;
        for (unsigned j = tid; j < cnt; j += kFinThreads) {
            const unsigned long long key = s.skey[j];
            reinterpret_cast<int2*>(pairs)[lo + j] = make_int2((int)((key >> B.fin.bits_b) & ma), (int)(key & mb));
            if constexpr (MULTI) (fits ? F.h_job : F.job_out)[lo + j] = (uint32_t)(key >> (B.fin.bits_a + B.fin.bits_b));
        }
    }
    if (F.want_segments) {
        int32_t* const segpair = fits ? F.h_segpair : F.segpair_out;
        for (unsigned q = 0; q < cnt; q += kFinPart) {
            const unsigned end = min(cnt, q + kFinPart), s0 = s.sseg[q];
            for (unsigned j = q + (tid >> 1); j < end; j += kFinThreads / 2) {
                const uint32_t v = s.sval[j], ns = v >> 30;
                const unsigned so = s.sseg[j];
                if (!ns) continue;
                const uint4 rr = __ldcg(B.res + (v & idx_mask));
                result_segments<MULTI>(B, rr, s.u.seg + 6u * (so - s0), tid & 1u, 2u);
                for (unsigned e = tid & 1u; e < ns; e += 2u) {
                    if (fits && F.h_segpair64) F.h_segpair64[so + e] = (int64_t)(lo + j);
                    else segpair[so + e] = (int32_t)(lo + j);
                }
            }
            __syncthreads();
            const unsigned s1 = s.sseg[end - 1u] + (s.sval[end - 1u] >> 30);
            double2* const out = reinterpret_cast<double2*>((fits ? F.h_segs : F.segs_out) + 6 * (size_t)s0);
            const double2* const in = reinterpret_cast<const double2*>(s.u.seg);
            for (unsigned t = tid; t < 3u * (s1 - s0); t += kFinThreads) out[t] = in[t];
            __syncthreads();  // read before the next part's segments take its place
        }
    }
    fin_stamp(C, 3);
    fin_end(C, F.host_cnt, s);
}

// Layout of the partition memory: two sets of counts (keys, extra segments),
// then the buckets and the overflow list, which both sets share (a call's are
// done with when the next begins).
size_t fin_scratch_bytes(int bucket)
{
    return sizeof(uint32_t) * 4 * kFinParts + (sizeof(unsigned long long) + sizeof(uint32_t)) * (size_t)kFinParts * bucket +
           (sizeof(unsigned long long) + sizeof(uint2)) * kFinOverflow;
}
uint32_t* fin_counts(void* mem, int set)
{
    return (uint32_t*)mem + (size_t)set * 2 * kFinParts;
}
FinBufs make_fin_bufs(void* mem, int bucket, int set, int bits_a, int bits_b, uint64_t sum_a, uint64_t max_b)
{
    FinBufs f;
    f.count = fin_counts(mem, set);
    f.extra = f.count + kFinParts;
    f.bkey = (unsigned long long*)((uint32_t*)mem + 4 * kFinParts);
    f.okey = f.bkey + (size_t)kFinParts * bucket;
    f.oval = (uint2*)(f.okey + kFinOverflow);
    f.bval = (uint32_t*)(f.oval + kFinOverflow);
    f.bucket = bucket;
    f.bits_a = bits_a;
    f.bits_b = bits_b;
    // rank * scale / 2^64 < kFinParts for every rank < sum_a * max_b (< 2^63: the keys' bits)
    f.stride = max_b;
    f.scale = (unsigned long long)(((unsigned __int128)kFinParts << 64) / std::max<unsigned __int128>((unsigned __int128)sum_a * max_b, kFinParts + 1));
    f.on = f.segments = 0;
    return f;
}

cudaError_t launch_finish(const Bufs& b, const FinArgs& F, const LaunchCfg& cfg, cudaStream_t st)
{
    note_launches(1);
    const void* kern = b.njobs > 1 ? (const void*)k_finish<true> : (const void*)k_finish<false>;
    Bufs bb = b;
    FinArgs ff = F;
    void* args[] = {&bb, &ff};
    // cooperative, and a programmatic dependent of the traversal launched just
    // before it on the stream: its launch overlaps the traversal's end
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(cfg.fin_per_sm * cfg.sms);
    lc.blockDim = dim3(kFinThreads);
    lc.dynamicSmemBytes = sizeof(FinShared);
    lc.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at;
    lc.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelExC(&lc, kern, args);
    if (e == cudaSuccess) return e;
    (void)cudaGetLastError();  // refused: launch it the plain cooperative way
    return cudaLaunchCooperativeKernel(kern, lc.gridDim, lc.blockDim, args, lc.dynamicSmemBytes, st);
}

// ===========================================================================
// Launchers
// ===========================================================================

cudaError_t query_launch(int device, LaunchCfg* cfg)
{
    cudaDeviceProp prop;
    GI_TRY(cudaGetDeviceProperties(&prop, device));
    cfg->sms = prop.multiProcessorCount;
    int nr[2][2] = {};
    cfg->blk_dyn[0][0] = sizeof(BlockShared<false, false>);
    cfg->blk_dyn[0][1] = sizeof(BlockShared<false, true>);
    cfg->blk_dyn[1][0] = sizeof(BlockShared<true, false>);
    cfg->blk_dyn[1][1] = sizeof(BlockShared<true, true>);
    const void* const kb[2][2] = {{(const void*)k_traverse_blocks<false, false>, (const void*)k_traverse_blocks<false, true>},
                                  {(const void*)k_traverse_blocks<true, false>, (const void*)k_traverse_blocks<true, true>}};
    for (int a = 0; a < 2; a++)
        for (int m = 0; m < 2; m++) {
            GI_TRY(cudaFuncSetAttribute(kb[a][m], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg->blk_dyn[a][m]));
            GI_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nr[a][m], kb[a][m], kBlkThreads, cfg->blk_dyn[a][m]));
        }
    for (int a = 0; a < 2; a++)
        for (int m = 0; m < 2; m++) cfg->blocks_per_sm[a][m] = nr[a][m] < 1 ? 1 : nr[a][m];
    int nf = 0, nm = 0;
    GI_TRY(cudaFuncSetAttribute(k_finish<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FinShared)));
    GI_TRY(cudaFuncSetAttribute(k_finish<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FinShared)));
    GI_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nf, k_finish<false>, kFinThreads, sizeof(FinShared)));
    GI_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nm, k_finish<true>, kFinThreads, sizeof(FinShared)));
    nf = nf < nm ? nf : nm;
    cfg->fin_per_sm = nf < 1 ? 1 : (nf > 2 ? 2 : nf);
    return cudaSuccess;
}

cudaError_t launch_traverse(const Bufs& b, const LaunchCfg& cfg, int precision, TravShape shape, cudaStream_t st)
{
    note_launches(1);
    const int f64 = precision == 1 ? 1 : 0, m = b.njobs > 1 ? 1 : 0;
    // cooperative: a block that waits needs every other resident
    const int grid = (shape.one_per_sm ? 1 : cfg.blocks_per_sm[f64][m]) * cfg.sms;
    Bufs bb = b;
    bb.keep = shape.give_half ? kBlkUnits / 2u : kBlkUnits;
    void* args[] = {&bb};
    const void* kern = f64 ? (m ? (const void*)k_traverse_blocks<true, true> : (const void*)k_traverse_blocks<true, false>)
                           : (m ? (const void*)k_traverse_blocks<false, true> : (const void*)k_traverse_blocks<false, false>);
    return cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(kBlkThreads), args, cfg.blk_dyn[f64][m], st);
}

cudaError_t launch_exact(const Bufs& b, const LaunchCfg& cfg, cudaStream_t st)
{
    k_exact<<<cfg.sms * 4, 128, 0, st>>>(b);
    note_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_segments(const Bufs& b, double* segs, uint32_t* nseg, const LaunchCfg& cfg, cudaStream_t st)
{
    k_segments<<<cfg.sms * 8, 128, 0, st>>>(b, segs, nseg);
    note_launches(1);
    return cudaGetLastError();
}

}  // namespace gi
