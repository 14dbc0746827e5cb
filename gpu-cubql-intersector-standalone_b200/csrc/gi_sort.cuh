// gi_sort.cuh -- block scan, decoupled look-back (output ordering) and the BVH
// build's LSD radix sort (30-bit Morton keys, 10-bit digits, stable; replaces the
// reference's CUB DeviceRadixSort in include/third-party/cubql/level_cut_builder.h:345-347).
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
// FEW: up to kRsFew small tiles, every scatter block adds up the tiles' digit
// counts itself, kept a row per tile, instead of a scan launch before each pass.
// Builds of 1 / 4 / 16 / 20 tiles: 67.5 / 75.0 / 81.2 / 82.8 us with the scans, 59.6 /
// 69.3 / 77.0 / 80.2 without.  Beyond, nothing is to be had: of 22 / 24 / 28 / 32
// tiles 84.1 / 84.8 / 90.9 / 92.8 with and 82.4 / 89.6 / 90.4 / 92.2 without (two
// spheres' build of 32 tiles: 81 and 87).
constexpr uint32_t kRsFew = 20;
// Place of a tile's count of digit d (2^BITS digits).
template <int BITS, bool FEW>
__device__ __forceinline__ uint32_t rs_count_at(uint32_t d, uint32_t tile, uint32_t ntiles)
{
    return FEW ? (tile << BITS) + d : d * ntiles + tile;
}

// Elements are (key << 32 | value): one 8-byte store per element and pass.
typedef unsigned long long RsElem;
template <int BITS>
__device__ __forceinline__ uint32_t rs_digit(RsElem e, int shift)
{
    return (uint32_t)(e >> (32 + shift)) & ((1u << BITS) - 1u);
}

template <int BITS, int ITEMS, bool FEW>
__global__ void __launch_bounds__(kRsThreads) k_rs_hist(const RsElem* __restrict__ in, uint32_t n, int shift,
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
    RsElem kk[ITEMS];
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        const uint32_t i = base + k * kRsThreads + threadIdx.x;
        kk[k] = i < n ? in[i] : 0ull;
    }
#pragma unroll
    for (int k = 0; k < ITEMS; k++) {
        const uint32_t i = base + k * kRsThreads + threadIdx.x;
        if (i < n) atomicAdd(&h[rs_digit<BITS>(kk[k], shift)], 1u);
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d < kDig; d += kRsThreads) counts[rs_count_at<BITS, FEW>(d, blockIdx.x, ntiles)] = h[d];
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

// Lanes of the warp with the same digit (kDig of a lane past the end included):
// a ballot per bit.  __match_any_sync takes a step per distinct value, up to 32:
// 20 us a pass of 1.3M elements against 15, 9.2 against 8.4 of 300k.
template <int BITS>
__device__ __forceinline__ unsigned same_digit(uint32_t d)
{
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b <= BITS; b++) {
        const bool bit = (d >> b) & 1u;
        const unsigned m = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? m : ~m;
    }
    return peers;
}

// Moves a tile's elements to their places; in the last pass (LAST) as separate
// keys and values.  A store instruction costs one memory transaction per sector
// that its lanes touch, and random places touch 32: elements are one word, and
// tiles with several keys per digit (ITEMS > 4) are put in order in shared memory
// first, so that a digit's elements leave as one run.  Passes of 1.3M elements,
// separate arrays and direct stores: 27, 27, 16.4 us; one word: 16.8, 16.8, 18.1;
// staged as well: 15.1, 15.1, 14.9.  Of 300k: 12.3, 12.3, 10.5 to 8.4 each.
template <int BITS, int ITEMS, bool LAST, bool FEW>
__global__ void __launch_bounds__(kRsThreads) k_rs_scatter(const RsElem* __restrict__ in, RsElem* __restrict__ out,
                                                           uint32_t* __restrict__ kout, uint32_t* __restrict__ vout, uint32_t n,
                                                           int shift, const uint32_t* __restrict__ offsets,
                                                           const uint32_t* __restrict__ totals, uint32_t ntiles)
{
    pdl_enter();
    constexpr uint32_t kDig = 1u << BITS;
    constexpr bool kStage = ITEMS > 4;
    static_assert(kDig == 4u * kRsThreads, "four digits per thread");
    static_assert(sizeof(RsElem) * kRsThreads * ITEMS <= sizeof(uint32_t) * kRsWarps * kDig, "a tile fits where its counts were");
    __shared__ __align__(16) uint32_t wc[kRsWarps][kDig];
    __shared__ __align__(16) uint32_t place[kDig];
    __shared__ uint32_t sw[33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t seg = blockIdx.x * (kRsThreads * ITEMS) + w * 32 * ITEMS;
    RsElem e[ITEMS];
#pragma unroll
    for (int c = 0; c < ITEMS; c++) {
        const uint32_t i = seg + c * 32 + lane;
        e[c] = i < n ? in[i] : 0ull;
    }
    // of the thread's four digits: all keys, and the keys of the tiles before this one
    uint4 t4 = make_uint4(0u, 0u, 0u, 0u);
    const uint32_t d0 = 4u * threadIdx.x;
    uint32_t o4[4] = {0u, 0u, 0u, 0u};
    if (FEW) {
#pragma unroll 4
        for (uint32_t t = 0; t < ntiles; t++) {
            const uint4 c = __ldg(reinterpret_cast<const uint4*>(offsets + ((size_t)t << BITS)) + threadIdx.x);
            if (t == blockIdx.x) o4[0] = t4.x, o4[1] = t4.y, o4[2] = t4.z, o4[3] = t4.w;
            t4.x += c.x, t4.y += c.y, t4.z += c.z, t4.w += c.w;
        }
    } else {
        t4 = __ldg(reinterpret_cast<const uint4*>(totals) + threadIdx.x);
#pragma unroll
        for (int q = 0; q < 4; q++) o4[q] = offsets[(size_t)(d0 + q) * ntiles + blockIdx.x];
    }
    for (uint32_t d = lane; d < kDig / 4u; d += 32) reinterpret_cast<uint4*>(wc[w])[d] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    uint32_t rank[ITEMS];
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int c = 0; c < ITEMS; c++) {
        const bool ok = seg + c * 32 + lane < n;
        const uint32_t d = ok ? rs_digit<BITS>(e[c], shift) : kDig;
        const unsigned peers = same_digit<BITS>(d);
        uint32_t r = 0;
        if (ok) r = wc[w][d] + __popc(peers & lt);
        rank[c] = r;
        __syncwarp();
        if (ok && (peers & lt) == 0) wc[w][d] += __popc(peers);
        __syncwarp();
    }
    // a digit's place: the digits before it (a scan of the totals, four per
    // thread) and its keys in the tiles before this one
    uint32_t tot;
    const uint32_t base = block_exclusive_scan(t4.x + t4.y + t4.z + t4.w, sw, &tot);  // (its barriers also complete wc)
    uint4 run = make_uint4(0u, 0u, 0u, 0u);  // the digits' keys in the warps before
    auto prefix = [&](uint4 start) {
        run = start;
#pragma unroll
        for (int q = 0; q < kRsWarps; q++) {
            uint4* const x = reinterpret_cast<uint4*>(wc[q]) + threadIdx.x;
            const uint4 t = *x;
            *x = run;
            run.x += t.x, run.y += t.y, run.z += t.z, run.w += t.w;
        }
    };
    uint4 pl = make_uint4(base + o4[0], base + t4.x + o4[1], base + t4.x + t4.y + o4[2], base + t4.x + t4.y + t4.z + o4[3]);
    if (!kStage) {
        prefix(pl);
        __syncthreads();
#pragma unroll
        for (int c = 0; c < ITEMS; c++) {
            if (seg + c * 32 + lane >= n) continue;
            const uint32_t pos = wc[w][rs_digit<BITS>(e[c], shift)] + rank[c];
            if (LAST) {
                kout[pos] = (uint32_t)(e[c] >> 32);
                vout[pos] = (uint32_t)e[c];
            } else {
                out[pos] = e[c];
            }
        }
        return;
    }
    uint4 mine = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int q = 0; q < kRsWarps; q++) {
        const uint4 t = reinterpret_cast<const uint4*>(wc[q])[threadIdx.x];
        mine.x += t.x, mine.y += t.y, mine.z += t.z, mine.w += t.w;
    }
    const uint32_t first = block_exclusive_scan(mine.x + mine.y + mine.z + mine.w, sw, &tot);
    const uint4 st = make_uint4(first, first + mine.x, first + mine.x + mine.y, first + mine.x + mine.y + mine.z);
    prefix(st);
    // element at position i of the ordered tile: place[digit] + i
    reinterpret_cast<uint4*>(place)[threadIdx.x] = make_uint4(pl.x - st.x, pl.y - st.y, pl.z - st.z, pl.w - st.w);
    __syncthreads();
#pragma unroll
    for (int c = 0; c < ITEMS; c++)
        if (seg + c * 32 + lane < n) rank[c] += wc[w][rs_digit<BITS>(e[c], shift)];
    __syncthreads();
    RsElem* const tile = reinterpret_cast<RsElem*>(&wc[0][0]);
#pragma unroll
    for (int c = 0; c < ITEMS; c++)
        if (seg + c * 32 + lane < n) tile[rank[c]] = e[c];
    __syncthreads();
#pragma unroll
    for (int c = 0; c < ITEMS; c++) {
        const uint32_t i = c * kRsThreads + threadIdx.x;
        if (i >= tot) break;
        const RsElem x = tile[i];
        const uint32_t pos = place[rs_digit<BITS>(x, shift)] + i;
        if (LAST) {
            kout[pos] = (uint32_t)(x >> 32);
            vout[pos] = (uint32_t)x;
        } else {
            out[pos] = x;
        }
    }
}

// Sorts elements in `a` by the low `bits` bits of their keys in passes of BITS-bit
// digits, between a and b; the last pass writes keys and vals.  Scratch: 2^BITS
// counts per tile of 256 x ITEMS elements, 2^BITS totals.  The producer of the
// elements has already written the first pass's per-tile digit counts into
// `counts` (at rs_count_at, as k_rs_hist).
template <int BITS, int ITEMS, bool FEW>
void radix_sort(RsElem* a, RsElem* b, uint32_t* keys, uint32_t* vals, uint32_t n, int bits, uint32_t* counts, uint32_t* totals,
                cudaStream_t st)
{
    const uint32_t tile = kRsThreads * ITEMS, ntiles = (n + tile - 1) / tile;
    const int passes = (bits + BITS - 1) / BITS;
    for (int p = 0; p < passes; p++) {
        if (p > 0) {
            launch_dep(k_rs_hist<BITS, ITEMS, FEW>, ntiles, kRsThreads, st, (const RsElem*)a, n, BITS * p, counts, ntiles);
            note_launches(1);
        }
        if (!FEW) {
            launch_dep(k_rs_scan<BITS>, (1u << BITS) / 8u, 256, st, counts, totals, ntiles);
            note_launches(1);
        }
        launch_dep(p + 1 < passes ? k_rs_scatter<BITS, ITEMS, false, FEW> : k_rs_scatter<BITS, ITEMS, true, FEW>, ntiles, kRsThreads, st,
                   (const RsElem*)a, b, keys, vals, n, BITS * p, (const uint32_t*)counts, (const uint32_t*)totals, ntiles);
        note_launches(1);
        RsElem* const t = a;
        a = b;
        b = t;
    }
}

}  // namespace gi
