// gi_launch.h -- host-side launchers of the kernels in gi_kernels.cu.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "gi_internal.cuh"

namespace gi {

// Device arrays owned by one resident mesh.
struct MeshBuffers {
    void* arena = nullptr;  // holds verts, tris, leafTri, leafBox, cutRef, cutBox, ncuts
    double* verts = nullptr;
    uint32_t* tris = nullptr;
    uint4* leafTri = nullptr;
    float* leafBox = nullptr;
    WNode* nodes = nullptr;
    double* leafBox64 = nullptr;
    WNode64* nodes64 = nullptr;
    uint32_t* cutRef = nullptr;
    uint32_t* ncuts = nullptr;  // device: sizes of the depth-3 and depth-4 cuts
    float* cutBox = nullptr;
    double* cutBox64 = nullptr;
    uint32_t* cutRef64 = nullptr;
    uint32_t nv = 0, nt = 0, nnodes = 0, root = 0;
    size_t bytes = 0;
};

// Stream-ordered allocation from the context's own pool (the device's default
// pool when none is given).
inline cudaError_t pool_alloc(void** p, size_t bytes, cudaMemPool_t pool, cudaStream_t st)
{
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, st) : cudaMallocAsync(p, bytes, st);
}
template <class T>
inline cudaError_t pool_alloc(T** p, size_t bytes, cudaMemPool_t pool, cudaStream_t st)
{
    return pool_alloc(reinterpret_cast<void**>(p), bytes, pool, st);
}

// A mesh's arrays of known size (all but the nodes) in one piece of device
// memory: sets their pointers and returns the bytes used.
size_t mesh_arena(MeshBuffers& m, void* mem);
size_t mesh_arena_bytes(uint32_t nv, uint32_t nt);

// Validates the input (error bit 1: bad index, 2: out of domain) and builds the
// 4-wide BVH (FP32 boxes) or, with fp64 = true, the FP64 node copy.  Queues
// everything on st, the copy of the build's header to h_words (kBuildWords
// pinned words) last.  With exact_nodes the node array has its exact size, for
// which the call waits once in between.
// After the stream has been synchronised, build_result reads the header: the
// node count and the error bits (4: the wide tree came out inconsistent, not
// expected; the kernels then skip the bad links).
constexpr int kBuildWords = 8;
bool build_wants_exact(uint32_t nt);  // true: a mesh of this size is built so in any case
cudaError_t build_bvh(MeshBuffers& m, bool fp64, bool exact_nodes, unsigned* h_words, cudaMemPool_t pool, cudaStream_t st);
unsigned build_result(MeshBuffers& m, bool fp64, const unsigned* h_words);

// Intersect launch configuration.
struct LaunchCfg {
    int sms = 0;
    int blocks_per_sm[2][2] = {};  // resident blocks of the block traversal, [FP64][batch]
    size_t blk_dyn[2][2] = {};     // ... and their shared memory
    int fin_per_sm = 1;            // resident blocks of the post-traversal launch (at most 2)
};

// Traversal shapes (GI_FLAG_SHAPE; every shape gives the same results): bit 0
// one block per SM instead of all resident ones, bit 1 blocks hand over what
// they hold beyond half an iteration's node pairs instead of beyond a whole
// one's.  The default has neither: the other forms measured slower or equal at
// every size (two 1.3 M-triangle meshes: 55 us of traversal against 60 with
// bit 1 and 78 with bit 0).  Bit 2 has no effect; the default has it set because
// gi_stats.traverse_shape has named the default so.
struct TravShape {
    bool one_per_sm = false;
    bool give_half = false;
};
constexpr int kDefaultShape = 4;
inline TravShape trav_shape(int k)
{
    TravShape t;
    t.one_per_sm = (k & 1) != 0;
    t.give_half = (k & 2) != 0;
    return t;
}
cudaError_t query_launch(int device, LaunchCfg* cfg);

// Traversal + first filter stage (persistent), then the exact stage.
cudaError_t launch_traverse(const Bufs& b, const LaunchCfg& cfg, int precision, TravShape shape, cudaStream_t st);
cudaError_t launch_exact(const Bufs& b, const LaunchCfg& cfg, cudaStream_t st);
// Segments of every result (count from the device counters):
// segs[18*i ..] (up to 3 segments), nseg[i].
cudaError_t launch_segments(const Bufs& b, double* segs, uint32_t* nseg, const LaunchCfg& cfg, cudaStream_t st);

// Output ordering (radix sort by (job, a, b), sizes from the device counters)
// and the gather of pairs / jobs / segments in that order.
constexpr int kOsMaxPasses = 8;
struct OrderBufs {
    unsigned long long* keys[2];
    uint32_t* vals[2];
    uint32_t* status;    // look-back status: (passes + 1) x ntiles_cap x 256
    uint32_t* gstatus;   // look-back status of the gather tiles
    uint32_t* hist;      // kOsMaxPasses x 256 (kept zero between calls)
    uint32_t* base;      // kOsMaxPasses x 256
    uint32_t* tile_ctr;  // kOsMaxPasses + 2 (per pass, the gather, the histogram blocks)
    uint32_t* tile_tot;  // kOrderSmallBlocks: segment totals per run (small-count path)
    uint32_t ntiles_cap;
    int passes;
    int bits_a, bits_b;
};
size_t order_scratch_bytes(uint32_t cap, int passes);
OrderBufs make_order_bufs(void* scratch, uint32_t cap, int bits_a, int bits_b, int bits_job);
// Pinned host arrays for the first pairs_cap pairs and segs_cap segments of the
// ordered result (job null: not wanted); the device arrays get all of it.
struct HostOut {
    int32_t* pairs;
    uint32_t* job;
    double* segs;
    int32_t* segpair;
    uint32_t pairs_cap, segs_cap;
};
cudaError_t launch_order_gather(const Bufs& b, const OrderBufs& O, bool sort, const double* segs,
                                const uint32_t* nseg, int32_t* pairs_out, uint32_t* job_out, double* segs_out,
                                int32_t* segpair_out, const HostOut& host, bool want_segments, const LaunchCfg& cfg,
                                cudaStream_t st);
// Small-count ordering: a cooperative launch of kOrderSmallBlocks blocks,
// each sorting a run of kOrderSmallRun keys, for up to kOrderSmallMax results.
// If the call produced more, the kernel only sets Counters::order_redo and the
// caller reruns with launch_order_gather.  Keys must fit in 63 bits.
constexpr int kOrderSmallRun = 1024;
constexpr int kOrderSmallBlocks = 24;
constexpr uint32_t kOrderSmallMax = (uint32_t)kOrderSmallRun * kOrderSmallBlocks;
cudaError_t launch_order_small(const Bufs& b, const OrderBufs& O, bool sort, const double* segs,
                               const uint32_t* nseg, int32_t* pairs_out, uint32_t* job_out, double* segs_out,
                               int32_t* segpair_out, bool want_segments, cudaStream_t st);
// The same in two launches: kOrderRank (sort the runs, rank every key) needs
// only the final result list; kOrderPlace (gather the pairs, place the
// segments) needs the segments too, so the ranking can run while the segments
// are built on another stream.
constexpr unsigned kOrderRank = 1u, kOrderPlace = 2u;
cudaError_t launch_order_small_phases(const Bufs& b, const OrderBufs& O, bool sort, const double* segs,
                                      const uint32_t* nseg, int32_t* pairs_out, uint32_t* job_out, double* segs_out,
                                      int32_t* segpair_out, bool want_segments, unsigned phases, cudaStream_t st);
// Everything after the traversal in one launch, for sorted output of up to
// kFinMax results with keys of at most 63 bits: the exact stage (when pairs were
// escalated), the segments, and the ordering by the kFinParts partitions that
// the results were put into as they were found (FinBufs).  A call over those
// limits, or with a partition over kFinBig keys, makes the kernel set only Counters::order_redo; the caller then reruns
// on the general path (launch_exact, launch_segments, launch_order_gather).
constexpr int kFinBig = 2048;
constexpr uint32_t kFinMax = 1u << 18;
struct FinArgs {
    // results in pinned host memory: for host_pairs pairs and host_segs segments
    int32_t* h_pairs;
    uint32_t* h_job;  // batches only
    double* h_segs;
    int32_t* h_segpair;
    int64_t* h_segpair64;  // not null: pair indices in this form instead
    uint32_t host_pairs, host_segs;
    // ... or, when they do not fit, in device memory (cap pairs, 3 segments each)
    int32_t* pairs_out;
    uint32_t* job_out;
    double* segs_out;
    int32_t* segpair_out;
    uint32_t cap;
    int want_segments;
    Counters* host_cnt;    // pinned: the counters when the launch ends
    Counters* next_cnt;    // cleared for the next call
    uint32_t* next_count;  // 2 x kFinParts, cleared for the next call
};
size_t fin_scratch_bytes(int bucket);
uint32_t* fin_counts(void* mem, int set);
FinBufs make_fin_bufs(void* mem, int bucket, int set, int bits_a, int bits_b, uint64_t sum_a, uint64_t max_b);
// Launched right after the traversal on the same stream, with no other stream
// work between them (programmatic dependent launch).
cudaError_t launch_finish(const Bufs& b, const FinArgs& F, const LaunchCfg& cfg, cudaStream_t st);

// Number of kernels launched by the launchers of this library (monotonic).
unsigned long long launch_count();
void note_launches(unsigned n);


}  // namespace gi
