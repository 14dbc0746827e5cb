// gi_sort.cuh -- block scan, decoupled look-back and LSD radix sort (10-bit digits, stable).
//
// Used by the BVH build (30-bit Morton keys, replaces the reference's CUB
// DeviceRadixSort in include/third-party/cubql/level_cut_builder.h:345-347)
// and by output ordering (64-bit (job, a, b) keys).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "gi_internal.cuh"

namespace gi {

// counts kernel launches made by this library (for gi_stats.launches)
void note_launches(unsigned n);

// Programmatic dependent launch of the build's kernels.  A kernel launched by
// launch_dep may be scheduled while the kernel before it in the stream is still
// finishing; at its first statement (pdl_enter) it waits for that kernel's
// completion and memory (griddepcontrol.wait), then lets its own successor be
// scheduled (griddepcontrol.launch_dependents).  Because the wait comes first
// in every such kernel, each one starts its work after all earlier kernels of
// the stream have completed, as in a plain launch; only the launch latency of
// the next kernel overlaps the tail of the current one.  In a plain launch both
// instructions are no-ops.
__device__ __forceinline__ void pdl_enter()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launches k(args...) with programmatic stream serialisation; a launch the
// driver refuses is repeated as a plain launch.
template <class... KArgs, class... Args>
inline void launch_dep(void (*k)(KArgs...), unsigned grid, unsigned block, cudaStream_t st, Args... args)
{
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(grid);
    lc.blockDim = dim3(block);
    lc.dynamicSmemBytes = 0;
    lc.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    if (cudaLaunchKernelEx(&lc, k, args...) != cudaSuccess) {
        (void)cudaGetLastError();
        k<<<grid, block, 0, st>>>(args...);
    }
}

// block-wide exclusive scan of per-thread sums; returns the block total
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* smem_warp, uint32_t* total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) smem_warp[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint32_t w = lane < nw ? smem_warp[lane] : 0u;
        uint32_t s = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < nw) smem_warp[lane] = s - w;
        if (lane == nw - 1) smem_warp[32] = s;
    }
    __syncthreads();
    uint32_t r = smem_warp[wid] + x - v;
    *total = smem_warp[32];
    __syncthreads();
    return r;
}

// ---------------------------------------------------------------------------
// Decoupled look-back (tile prefix sums in one pass): a status word per tile
// and slot holds a flag and a count, the tile's own aggregate first, then its
// inclusive prefix.
// ---------------------------------------------------------------------------
constexpr unsigned kFlagAgg = 1u << 30, kFlagInc = 2u << 30, kCountMask = (1u << 30) - 1u;
constexpr unsigned long long kLookbackSpins = 1ull << 22;

// Exclusive prefix of this tile over the preceding tiles, per status slot.
// Returns false if a wait ran out (the error bit is set; results are invalid).
__device__ __forceinline__ bool lookback(unsigned* status, unsigned tile, unsigned stride, unsigned own,
                                         unsigned* excl_out, unsigned* err)
{
    unsigned excl = 0;
    if (tile > 0) {
        // publish the local aggregate first so successors need not wait for our prefix
        atomicExch(status + (size_t)tile * stride, kFlagAgg | (own & kCountMask));
        unsigned t = tile - 1;
        for (;;) {
            volatile unsigned* q = status + (size_t)t * stride;
            unsigned v = *q;
            unsigned long long spins = 0;
            while ((v & ~kCountMask) == 0u) {
                if (++spins > kLookbackSpins) {
                    atomicOr(err, kErrTimeout);
                    *excl_out = 0;
                    return false;
                }
                __nanosleep(32);
                v = *q;
            }
            excl += v & kCountMask;
            if ((v & ~kCountMask) == kFlagInc || t == 0) break;
            t--;
        }
    }
    __threadfence();
    atomicExch(status + (size_t)tile * stride, kFlagInc | ((excl + own) & kCountMask));
    *excl_out = excl;
    return true;
}

// ---------------------------------------------------------------------------
// Radix sort
// ---------------------------------------------------------------------------
// Keys per thread of a tile.  Large sorts: 12, 427 tiles of 3,072 keys for a
// 1.3M-triangle mesh, which keeps more scatter warps resident per SM than
// 4,096-key tiles (build 0.435 -> 0.418 ms on B200; 10 and 14 keys per thread
// gave 0.427 and 0.426 ms, 8 keys 0.436 ms: smaller tiles pay more per-tile
// overhead).  Small sorts: 4, so that they have blocks enough for the SMs.
constexpr int kRsThreads = 256;
constexpr int kRsItems = 12;
constexpr int kRsItemsSmall = 4;
constexpr int kRsWarps = kRsThreads / 32;

template <class K, int BITS, int ITEMS>
__global__ void __launch_bounds__(kRsThreads) k_rs_hist(const K* __restrict__ keys, uint32_t n, int shift,
                                                        uint32_t* __restrict__ counts, uint32_t ntiles)
{
    pdl_enter();
    constexpr uint32_t kDig = 1u << BITS;
    __shared__ uint32_t h[kDig];
    for (uint32_t d = threadIdx.x; d < kDig; d += kRsThreads) h[d] = 0;
    __syncthreads();
    // every load of the tile is issued before the first shared-memory atomic
    // (one round trip to memory per thread instead of one per few keys)
    uint32_t base = blockIdx.x * (kRsThreads * ITEMS);
    K kk[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        const uint32_t i = base + k * kRsThreads + threadIdx.x;
        kk[k] = i < n ? keys[i] : (K)0;
    }
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        const uint32_t i = base + k * kRsThreads + threadIdx.x;
        if (i < n) atomicAdd(&h[(uint32_t)(kk[k] >> shift) & (kDig - 1u)], 1u);
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d < kDig; d += kRsThreads) counts[d * ntiles + blockIdx.x] = h[d];
}

// Exclusive scan of every digit's tile counts, a warp per digit, in place; the
// digit's total to totals[d].  (The counts of all digits as one sequence took
// two launches: tiles of 4,096 counts and their sums.)
template <int BITS>
__global__ void __launch_bounds__(256) k_rs_scan(uint32_t* __restrict__ counts, uint32_t* __restrict__ totals, uint32_t ntiles)
{
    pdl_enter();
    const uint32_t d = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    uint32_t* const c = counts + (size_t)d * ntiles;
    uint32_t run = 0;
    constexpr int kAhead = 4;  // chunks of 32 counts in flight
    for (uint32_t t0 = 0; t0 < ntiles; t0 += 32u * kAhead) {
        uint32_t v[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; q++) {
            const uint32_t t = t0 + 32u * q + lane;
            v[q] = t < ntiles ? c[t] : 0u;
        }
#pragma unroll
        for (int q = 0; q < kAhead; q++) {
            uint32_t x = v[q];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= (uint32_t)o) x += y;
            }
            const uint32_t t = t0 + 32u * q + lane;
            if (t < ntiles) c[t] = run + x - v[q];
            run += __shfl_sync(0xffffffffu, x, 31);
        }
    }
    if (lane == 0) totals[d] = run;
}

template <class K, int BITS, int ITEMS>
__global__ void __launch_bounds__(kRsThreads) k_rs_scatter(const K* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                           K* __restrict__ kout, uint32_t* __restrict__ vout, uint32_t n,
                                                           int shift, const uint32_t* __restrict__ offsets,
                                                           const uint32_t* __restrict__ totals, uint32_t ntiles)
{
    pdl_enter();
    constexpr uint32_t kDig = 1u << BITS;
    __shared__ uint32_t wc[kRsWarps][kDig];
    __shared__ uint32_t tile_off[kDig];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (uint32_t d = lane; d < kDig; d += 32) wc[w][d] = 0;
    {
        // a digit's place: the digits before it (a scan of the totals, four per
        // thread) and its keys in the tiles before this one
        static_assert(kDig == 4u * kRsThreads, "four digits per thread");
        __shared__ uint32_t sw[33];
        const uint4 t4 = __ldg(reinterpret_cast<const uint4*>(totals) + threadIdx.x);
        const uint32_t d = 4u * threadIdx.x;
        uint32_t o4[4];
#pragma unroll
        for (int q = 0; q < 4; q++) o4[q] = offsets[(size_t)(d + q) * ntiles + blockIdx.x];
        uint32_t tot;
        const uint32_t base = block_exclusive_scan(t4.x + t4.y + t4.z + t4.w, sw, &tot);
        tile_off[d] = base + o4[0];
        tile_off[d + 1] = base + t4.x + o4[1];
        tile_off[d + 2] = base + t4.x + t4.y + o4[2];
        tile_off[d + 3] = base + t4.x + t4.y + t4.z + o4[3];
    }
    __syncwarp();
    const uint32_t seg = blockIdx.x * (kRsThreads * ITEMS) + w * 32 * ITEMS;
    K key[ITEMS];
    uint32_t val[ITEMS];
    uint32_t rank[ITEMS];
    uint32_t dig[ITEMS];
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int c = 0; c < ITEMS; c++) {
        uint32_t i = seg + c * 32 + lane;
        bool ok = i < n;
        key[c] = ok ? kin[i] : (K)0;
        val[c] = ok ? vin[i] : 0u;
        uint32_t d = ok ? ((uint32_t)(key[c] >> shift) & (kDig - 1u)) : kDig;
        dig[c] = d;
        unsigned peers = __match_any_sync(0xffffffffu, d);
        uint32_t r = 0;
        if (ok) r = wc[w][d] + __popc(peers & lt);
        rank[c] = r;
        __syncwarp();
        if (ok && (peers & lt) == 0) wc[w][d] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // per digit: exclusive prefix over warps
    for (uint32_t d = threadIdx.x; d < kDig; d += kRsThreads) {
        uint32_t run = 0;
        for (int q = 0; q < kRsWarps; q++) {
            uint32_t t = wc[q][d];
            wc[q][d] = run;
            run += t;
        }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < ITEMS; c++) {
        uint32_t d = dig[c];
        if (d < kDig) {
            uint32_t pos = tile_off[d] + wc[w][d] + rank[c];
            kout[pos] = key[c];
            vout[pos] = val[c];
        }
    }
}

// Sorts (keys, vals) by the low `bits` bits of the key in passes of BITS-bit
// digits.  The passes alternate between the two buffer pairs; on return
// (k0, v0) point to the pair that holds the result and (k1, v1) to the other
// (swapped after an odd number of passes, nothing copied).  Scratch: 2^BITS
// counts per tile of 256 x ITEMS keys, 2^BITS totals.  The producer of the keys
// has already written the first pass's per-tile digit counts into `counts`
// (layout of k_rs_hist: digit-major, one column per tile).
template <class K, int BITS, int ITEMS>
void radix_sort(K*& k0, uint32_t*& v0, K*& k1, uint32_t*& v1, uint32_t n, int bits, uint32_t* counts, uint32_t* totals,
                cudaStream_t st)
{
    if (n <= 1) return;
    const uint32_t tile = kRsThreads * ITEMS, ntiles = (n + tile - 1) / tile;
    int passes = (bits + BITS - 1) / BITS;
    K* ks = k0;
    uint32_t* vs = v0;
    K* kd = k1;
    uint32_t* vd = v1;
    for (int p = 0; p < passes; p++) {
        if (p > 0) {
            launch_dep(k_rs_hist<K, BITS, ITEMS>, ntiles, kRsThreads, st, (const K*)ks, n, BITS * p, counts, ntiles);
            note_launches(1);
        }
        launch_dep(k_rs_scan<BITS>, (1u << BITS) / 8u, 256, st, counts, totals, ntiles);
        launch_dep(k_rs_scatter<K, BITS, ITEMS>, ntiles, kRsThreads, st, (const K*)ks, (const uint32_t*)vs, kd, vd, n,
                   BITS * p, (const uint32_t*)counts, (const uint32_t*)totals, ntiles);
        note_launches(2);
        K* tk = ks;
        ks = kd;
        kd = tk;
        uint32_t* tv = vs;
        vs = vd;
        vd = tv;
    }
    k1 = kd;
    v1 = vd;
    k0 = ks;
    v0 = vs;
}

}  // namespace gi
