// gi_internal.cuh -- device-side data layout shared by the kernels of libgi.
//
// HBM layout of one resident mesh (built once by gi_mesh_upload):
//   verts     double[3*nv]            input vertices (mesh-local frame)
//   tris      uint32[3*nt]            input triangles (original order)
//   leafTri   uint4[nt]               per Morton-sorted leaf: v0, v1, v2, original id
//   leafBox   float[6*nt]             per sorted leaf: FP32 box rounded outward
//   nodes     WNode[nnodes]           4-wide BVH, 128 B per node (one cache line)
//   leafBox64 / nodes64               FP64 copies for the plain-FP64 form (built lazily)
// Traversal runs in the world frame: node boxes are mapped through the pose on
// the fly (conservatively), so a new pose needs no rebuild or refit.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace gi {

constexpr uint32_t kLeaf = 0x80000000u;   // child ref: sorted leaf position
constexpr uint32_t kEmpty = 0xFFFFFFFFu;  // unused child slot

// 4-wide BVH node: a child's box and reference lie together, so that lane k of a
// quad reads child k with two 16-byte loads (field by field it took seven
// 4-byte ones, each of which touched the lines of all eight quads of a warp)
// and the collapse writes it with two stores.
struct __align__(32) WKid {
    float lo[3];
    uint32_t ref;
    float hi[3];
    uint32_t pad;
};
struct __align__(128) WNode {
    WKid kid[4];
};
static_assert(sizeof(WNode) == 128, "WNode is one 128-byte line");

struct __align__(64) WKid64 {
    double lo[3], hi[3];
    uint32_t ref, pad[3];
};
struct __align__(256) WNode64 {
    WKid64 kid[4];
};
static_assert(sizeof(WNode64) == 256, "WNode64 is two 128-byte lines");

// Pose on the device.
//  exact vertex map: world = ((R*(v - C)) + C) + T in FP64, left to right, no FMA
//  box map (FP32):  world = R*v + b, padded by rho*(|R|(|c|+h) + padm)
struct __align__(16) BoxMap {
    float4 row[3];  // R's row r, and b[r]
    float padm[3];
    int use;  // 0: the map is the identity (forward) or must not be used (inverse)
};
static_assert(sizeof(BoxMap) == 64, "four 16-byte loads");
struct __align__(16) DevPose {
    BoxMap fw;   // local -> world
    BoxMap inv;  // world -> local (inverse map, near-orthonormal R only: use = inv_ok)
    double R[9], C[3], T[3];
    double b64[3];     // C + T - R*C (FP64), for FP64 node boxes
    double padm64[3];  // |C| + |T| + |R||C| (FP64), magnitude term of the pad
    int identity;
    // world -> local (inverse) map for a near-orthonormal R: local = Ri*w + bi
    // with Ri = R^T; inv_ok = 0 when R is not orthonormal within 2^-30
    int inv_ok;
    double inv_eta;    // max |R^T R - I| entry: error of R^T as the inverse
    double Ri64[9], bi64[3], padmi64[3];
};

struct MeshDev {
    const double* verts;
    const uint32_t* tris;
    const uint4* leafTri;
    const float* leafBox;
    const double* leafBox64;
    const WNode* nodes;
    const WNode64* nodes64;
    // cuts: node / leaf refs whose subtrees cover all leaves, the depth-3 cut in
    // entries [0, kCutMax) and the depth-4 cut in [kCutMax, kCutMax + kCut4Max)
    const uint32_t* cutRef;
    const uint32_t* cutRef64;  // the same for nodes64 (the two trees number their nodes apart)
    const float* cutBox;     // their boxes (6 floats each)
    const double* cutBox64;  // FP64 boxes of the same cuts (FP64 form)
    uint32_t root;  // wide node index, or kLeaf | leaf position when nt == 1
    uint32_t nv, nt, nnodes;
    const uint32_t* ncuts;  // device: entries of the depth-3 and the depth-4 cut (null for an empty mesh)
};

constexpr int kCutMax = 64;    // 4^3
constexpr int kCut4Max = 256;  // 4^4
constexpr int kCutCap = kCutMax + kCut4Max;

struct __align__(16) JobDev {
    MeshDev A, B;
    unsigned long long a0;  // triangles of A in the jobs before this one
    unsigned long long pad_;
    DevPose pa, pb;
};

// Device counters of one intersect launch sequence: zero when it begins (the
// one-launch finish clears the next call's, the host's memset does otherwise).
struct Counters {
    // hot counters, each on its own 128-byte line (polled and updated by every block)
    // pool of the traversal: slots given out (low half), and blocks at work plus
    // slots not yet taken, less the grid's blocks (high half)
    unsigned long long pool;
    unsigned int pad0[30];
    unsigned int q_head;  // tickets taken by blocks out of node pairs
    unsigned int pad1[31];
    unsigned int res;     // intersecting pairs
    unsigned int esc;     // escalated candidate indices
    unsigned int overflow;  // kOvf* bits
    unsigned int err;       // kErr* bits
    unsigned int levels;    // most iterations of a traversal block
    unsigned int nseg;      // total segments after ordering
    unsigned int obar;      // grid barrier of the small-count ordering kernel
    unsigned int order_redo;  // small-count ordering refused (too many results): rerun on the radix path
    unsigned int starved;   // iterations that kept node pairs others waited for, the pool being nearly used up
    unsigned long long node_pairs;
    unsigned long long filter_decided;
    unsigned long long exact_signs;
    unsigned long long exact_points;
    unsigned long long tested;  // candidates run through the first filter stage
    // post-traversal launch (k_finish): globaltimer at its start, after the exact
    // stage, when block 0 had its run ranked and when it had it written, and when
    // the last block ended
    unsigned long long fin_ns[5];
    unsigned long long t_start;  // globaltimer when the traversal's first block began
    unsigned fin_done;  // blocks of k_finish that have ended
    unsigned fin_over;  // results whose partition's bucket was full (may exceed the overflow list)
    unsigned odd;       // 1: some result has other than one segment
    unsigned pad2;
};

// (kOvfResExact: the exact stage's results did not fit; a bit of its own, because
// the traversal's are final when k_finish begins and this one is not)
constexpr unsigned kOvfFrontier = 1u, kOvfRes = 4u, kOvfEsc = 8u, kOvfResExact = 16u;
constexpr unsigned kErrTimeout = 1u, kErrExactCapacity = 2u;
// Counters::order_redo: the small-count ordering or the one-launch finish
// refused; the finish because of a key partition over its limit (kRedoCrowded) or
// of more keys beyond their buckets than the overflow list holds (kRedoSpilled)
constexpr unsigned kRedoCount = 1u, kRedoCrowded = 2u, kRedoSpilled = 3u;

// Results by key partition, for the one-launch finish: filled where results are
// found, read by k_finish.
constexpr int kFinPartBits = 12;
constexpr int kFinParts = 1 << kFinPartBits;
constexpr int kFinOverflow = 1 << 16;
// keys of a partition's bucket: up to 65,536 expected results, and beyond (a
// partition then holds 16 to 64 keys on average, but results cluster in index)
constexpr int kFinBucketSmall = 256, kFinBucketLarge = 1024;
struct FinBufs {
    uint32_t* count;  // kFinParts key counts (zero when a call begins)
    uint32_t* extra;  // kFinParts: segments beyond one per key, modulo 2^32 (zero when a call begins)
    unsigned long long* bkey;  // kFinParts x bucket: each partition's first keys
    uint32_t* bval;            // ... and their result index | segment count << 30
    unsigned long long* okey;  // kFinOverflow: the keys beyond a bucket
    uint2* oval;               // ... their value, and their slot in the partition | partition << 20
    int bucket;
    int bits_a, bits_b;
    // partition of a result: its rank among all conceivable pairs, ((A triangles of
    // the earlier jobs + a) * stride + b), times scale / 2^64
    unsigned long long stride, scale;
    int on;                    // 1: results are inserted
    int segments;              // the call wants segments
};

// Per-call buffers handed to the kernels.
struct Bufs {
    const JobDev* jobs;
    uint32_t njobs;
    uint4* queue;     // pool slots of 64 node pairs: job, node/leaf ref A, node/leaf ref B, entries of the slot
    unsigned* qflag;  // per pool slot: tag of the call that published it
    uint32_t cap_queue;  // node pairs the pool holds
    uint4* res;       // job, triA, triB (original triangle ids), construction code
    uint32_t cap_res;
    uint4* esc;       // escalated candidates: job, leaf posA, leaf posB, 0
    uint32_t cap_esc;
    Counters* cnt;
    unsigned tag;     // nonzero, different for every launch on the context
    int precision;    // 0 FP32 cascade, 1 FP64
    int two_frame;    // also test child boxes in B's own frame (fewer pairs, more work per pair)
    unsigned keep;          // block traversal: node pairs that a block does not hand over
    FinBufs fin;
    JobDev job0;            // the job of a call with one (njobs == 1), read from the kernel's parameters
};

}  // namespace gi
