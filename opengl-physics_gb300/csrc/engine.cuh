// engine.cuh -- device data layout and kernel launchers of the GB300
// Barnes-Hut engine (internal; the public surface is include/ngrav_gpu.h).
//
// Layout in HBM (all particle arrays in the current tree order, i.e. sorted
// by 63-bit octant-path key; `id` maps a slot back to the caller's index):
//   pos   float4 (x_hi, y_hi, z_hi, m)     the state (FP32, or the high half)
//   plo   float4 (x_lo, y_lo, z_lo, 0)     low half of double-float positions (SPLIT)
//   vel   float4 (vx, vy, vz, 0)
//   acc   float4 (ax, ay, az, 0)           G included
//   src   float4 (ox, oy, oz, m)           walk input: offset from the own leaf's
//                                           centre (SPLIT) or absolute (PLAIN)
//   id    int
// Nodes (one record per node, breadth-first by level; children of a node are
// contiguous and in ascending octant order):
//   start/count/first_child/parent/level/nchild, centre (FP64), FP64 moments,
//   and four float4 walk records (see NodeWalk below).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ngrav {

constexpr int kKeyLevels = 21;          // 63-bit keys: 3 bits per level
constexpr int kRsDigitBits = 9;         // radix sort digit: 7 passes over the 63-bit keys
constexpr int kRsBins = 1 << kRsDigitBits;
constexpr int kRsPasses = (3 * kKeyLevels + kRsDigitBits - 1) / kRsDigitBits;
constexpr int kMaxLevels = kKeyLevels + 1;

// Device status word bits (sticky within one force evaluation).
enum : unsigned {
    kStNodeOverflow = 1u,
    kStStackOverflow = 2u,
    kStDepthLimit = 4u,     // warning: a depth-21 leaf holds more than leaf_capacity
    kStNonFinite = 8u,
    kStTimeout = 16u,
    kStListOverflow = 32u,  // per-warp list staging or the final list pool
    kStCorrupt = 64u,       // walk visit limit breached
    kStPendOverflow = 128u, // learned walk: deferred-pair pool exhausted
    kStSortDepth = 256u,    // a node at the deepest sorted key level still needs splitting
    kStFatal = kStNodeOverflow | kStStackOverflow | kStNonFinite | kStTimeout | kStListOverflow | kStCorrupt |
               kStPendOverflow | kStSortDepth,
};

// Per-evaluation device counters (zeroed before each force evaluation).
struct Counters {
    unsigned long long p2p_pairs;
    unsigned long long p2c_terms;
    unsigned long long mac_tests;
    unsigned long long mac_retests;
    unsigned long long groups;
    unsigned long long bbox_min[3];   // order-preserving encoded FP64
    unsigned long long bbox_max[3];
    unsigned status;
    int next_free;                    // node allocator
    int level_begin[kMaxLevels + 2];
    int nleaves;
    int max_leaf_count;
    int depth_limited;
    int work_next;                    // dynamic group scheduler (walk)
    int stack_max;
    int levels_used;
    int eval_next;                    // dynamic pass scheduler (evaluation)
    double root_center[3];
    double root_half;
    unsigned long long far_total;     // list entries written (far, near)
    unsigned long long near_total;
    int list_max;                     // longest per-group list seen
    int far_chunks;                   // chunk allocators (may exceed the pool: then
    int near_chunks;                  //   they count what a retry needs)
    int extra_passes;                 // evaluation passes past each group's first (ListBuffers::passes)
    // learned opening test: pairs handed to the network, accepted by it, and
    // decided by the geometric fallback (low confidence); tensor-core flushes
    unsigned long long lm_queries;
    unsigned long long lm_accepts;
    unsigned long long lm_fallbacks;
    unsigned long long lm_flushes;
    unsigned long long lm_screened;   // band pairs the error bound accepted without the network
    unsigned long long targets;       // particles whose acceleration a block-step evaluation refreshed
};

// Targets per pass of the evaluation (eval.cu).  A pass (of one group) is the
// unit of work of a warp.  A pass of more targets loads the group's lists fewer
// times, so the largest is taken where the groups alone fill the GPU's 152 x 16
// warps four times over, and smaller ones below that, where idle warps and
// long units cost more.  Evaluation kernel, leaf capacity 64: 2,500 bodies
// (spline) 356 us before, 121 at 20 targets a pass, 46 at 5; 150,000 bodies
// 2.97 ms before, 3.54 with a group's passes on one warp, 2.37 as units.  The
// choice changes no sum.
constexpr int kPassMax = 20, kPassMid = 10, kPassMin = 5;
constexpr int kEvalWave = 152 * 16;
__host__ __device__ inline int pass_targets(int groups) {
    return groups >= 4 * kEvalWave ? kPassMax : (groups >= kEvalWave ? kPassMid : kPassMin);
}

// Per-group interaction lists written by the walk, read by the evaluation.
// Each list is a chain of kListChunk-entry chunks taken from a pool with one
// atomic per chunk; next[c] links chunk c to the following one.
constexpr int kListChunk = 128;
struct ListBuffers {
    int far_chunk_cap = 0, near_chunk_cap = 0;
    int* far = nullptr;               // far node ids, far_chunk_cap * kListChunk
    int* near = nullptr;              // near leaf ids
    int* far_next = nullptr;          // chunk links
    int* near_next = nullptr;
    int4* ginfo = nullptr;            // per group: far first chunk, near first chunk, far count, near count
    int2* passes = nullptr;           // evaluation passes past each group's first: group, pass (n / kPassMin entries)
    int* stack = nullptr;             // per walking warp traversal stack
    int stack_cap = 0;
    int nwarps = 0;                   // resident walking warps
};

// Scratch of the topology build, and the leaves it lists in key order.
struct TreeBuffers {
    unsigned short* runs = nullptr;   // per particle: the levels of the nodes that begin at it
    int* counts = nullptr;            // nodes per level and leaves, per segment of the particles; their totals
    int* leaf_list = nullptr;
    unsigned* leaf_before = nullptr;  // per particle: the leaves that begin before it,
    unsigned* leaf_start = nullptr;   // and whether one begins at it
};

struct NodeArrays {
    int cap = 0;
    int* start = nullptr;
    int* count = nullptr;
    int* first_child = nullptr;       // -1 for leaves
    int* parent = nullptr;
    unsigned char* nchild = nullptr;
    unsigned char* level = nullptr;
    double* cx = nullptr;             // geometric centre (FP64 recurrence of the reference)
    double* cy = nullptr;
    double* cz = nullptr;
    double* half = nullptr;           // half size (0 on the system-id levels of an ensemble)
    int* sysroot = nullptr;           // root node of the node's system (0 for a single system)
    // FP64 moments
    double* mass = nullptr;
    double* comx = nullptr;
    double* comy = nullptr;
    double* comz = nullptr;
    double* maxr = nullptr;
    double* quad = nullptr;           // 5 per node
    float* amin = nullptr;            // leaves: min |a| over the members (learned opening test)
    // FP32 walk records
    float4* wA = nullptr;             // com_hi.xyz, mass
    float4* wB = nullptr;             // Qxx, Qyy, Qxy, Qxz
    float4* wC = nullptr;             // maxR (rounded up), 2h, link (int bits), meta (int bits)
    float4* wD = nullptr;             // com_lo.xyz, Qyz
    float4* chi = nullptr;            // leaves: centre hi, first slot (int bits)
    float4* clo = nullptr;            // leaves: centre lo, particle count (int bits)
};

// wC.w meta: bit 31 leaf flag; bits 0..23 count (leaf) or nchild (internal);
// bits 24..28 level.
__host__ __device__ inline int meta_pack(bool leaf, int count_or_nchild, int level) {
    return (leaf ? (int)0x80000000u : 0) | ((level & 31) << 24) | (count_or_nchild & 0xFFFFFF);
}

struct Particles {
    long long cap = 0;
    float4* pos = nullptr;
    float4* plo = nullptr;
    float4* vel = nullptr;
    float4* vlo = nullptr;            // velocity low halves (SPLIT): kicks accumulate ~48 bits
    float4* acc = nullptr;
    float4* src = nullptr;
    int* id = nullptr;
    // ping-pong partners for the permutation
    float4* pos2 = nullptr;
    float4* plo2 = nullptr;
    float4* vel2 = nullptr;
    float4* vlo2 = nullptr;
    float4* acc2 = nullptr;
    int* id2 = nullptr;
};

struct SortBuffers {
    long long cap = 0;
    unsigned long long* keys = nullptr;
    unsigned long long* keys_alt = nullptr;
    unsigned* vals = nullptr;
    unsigned* vals_alt = nullptr;
    unsigned* hist = nullptr;         // kRsBins x blocks
    long long hist_cap = 0;
    float4* frame = nullptr;          // key frame of a single system (kFrame)
};

struct WalkParams {
    float eps2;
    float theta;
    float theta2;
    float G;
    double theta2_d;
    double eps2_d;
    int quadrupole;
    int split;
    int retest;
    int kick;                         // apply closing half-kick v += hdt * a
    float hdt;
    int stack_cap;
    int node_limit;                   // visits per group beyond this mean a corrupt tree
    int global_stack;                 // walk stack in global memory (fallback for deep frontiers)
    int smem_stack;                   // per-warp shared-memory walk stack: 1024, 2048 or 4096 entries
    int soft;                         // kSoftPlummer or kSoftSpline (softening.cuh)
    float ih;                         // spline: 1 / h (h = eps)
    int p2p_tile;                     // sources per near batch of the evaluation (64 or 128; 256 and 0: as many as fit)
    // learned opening test (walk_lmac_kernel)
    int learned;
    float lm_log2b;                   // log2 of the per-target error budget
    float lm_gate;                    // |logit| below which the geometric test decides
    float lm_rho_lo, lm_rho_hi;       // band of 2h/worst handed to the network
    float lm_mu[8], lm_isd[8];        // feature standardisation of the network
    float lm_screen;                  // accept unasked when the error bound <= lm_screen * budget (0: off)
    float lm_budget;                  // the budget itself
};

// A root cube in the form the keys are computed from, kFrame float4 per system:
// centre high parts, tolerance; centre low parts, scale; scale's low part.
constexpr int kFrame = 3;

// A forest of independent systems in one particle set (ensemble).  System s
// holds slots [off[s], off[s+1]) in every tree order; its id occupies the top
// sys_levels key digits, the remaining 21 - sys_levels digits are the octant
// path from its own root cube (the reference's BuildRoot on its particles).
// The system-id levels are virtual: they always split and carry no geometry.
// A single system is sys_levels = 0, nsys = 1, off = nullptr.
struct Forest {
    int nsys = 1;
    int sys_levels = 0;
    const long long* off = nullptr;   // nsys + 1 slot offsets
    double* root = nullptr;           // per system: centre x, y, z, half (4 doubles)
    unsigned long long* bbox = nullptr;  // per system: encoded min x, y, z, max x, y, z
    float4* frame = nullptr;          // per system: its key frame (kFrame)
};

// Packed FP32 pair arithmetic (two lanes of one register pair per op).
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }

// Error-free steps.  Every rounding is asked for by name: an operand may be a
// product after inlining, and one fused into the sum, but not into its error,
// would be counted twice.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

__device__ __forceinline__ void fast_two_sum(float a, float b, float& s, float& e) {
    s = __fadd_rn(a, b);
    e = __fsub_rn(b, __fsub_rn(s, a));
}

// Offset of a double-float coordinate (h + l) from a double-float centre
// (ch + cl), as a normalised double-float pair.
__device__ __forceinline__ void df_offset(float h, float l, float ch, float cl, float& oh, float& ol) {
    float s, e;
    two_sum(h, -ch, s, e);
    fast_two_sum(s, __fadd_rn(e, __fsub_rn(l, cl)), oh, ol);
}

// (h, l) += m (oh + ol) for a double-float pair, the product of the high parts exact.
__device__ __forceinline__ void df_add_prod(float& h, float& l, float m, float oh, float ol) {
    const float p = __fmul_rn(m, oh);
    const float pe = __fmaf_rn(m, ol, __fmaf_rn(m, oh, -p));
    float t, e;
    two_sum(h, p, t, e);
    fast_two_sum(t, __fadd_rn(l, __fadd_rn(e, pe)), h, l);
}

// Bounding box of double-float coordinates, compared as pairs: the high part is
// the rounded value, so it orders the values, and the low part does where the
// high parts are equal.  (FP64 minima and maxima cost a particle a dozen
// instructions of a pipe 64 times narrower.)
struct DfBox {
    float2 lo[3], hi[3];  // (high, low)
};

__device__ __forceinline__ bool df_less(const float2& a, const float2& b) {
    return a.x < b.x || (a.x == b.x && a.y < b.y);
}

__device__ __forceinline__ DfBox empty_box() {
    DfBox b;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        b.lo[k] = make_float2(1.f / 0.f, 0.f);
        b.hi[k] = make_float2(-1.f / 0.f, 0.f);
    }
    return b;
}

__device__ __forceinline__ void box_take(DfBox& b, int k, const float2& lo, const float2& hi) {
    if (df_less(lo, b.lo[k])) b.lo[k] = lo;
    if (df_less(b.hi[k], hi)) b.hi[k] = hi;
}

__device__ __forceinline__ void box_add(DfBox& b, const float4& p, const float4& l) {
    const float2 x = make_float2(p.x, l.x), y = make_float2(p.y, l.y), z = make_float2(p.z, l.z);
    box_take(b, 0, x, x);
    box_take(b, 1, y, y);
    box_take(b, 2, z, z);
}

__device__ __forceinline__ void box_warp(DfBox& b) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            float2 lo, hi;
            lo.x = __shfl_xor_sync(0xffffffffu, b.lo[k].x, o);
            lo.y = __shfl_xor_sync(0xffffffffu, b.lo[k].y, o);
            hi.x = __shfl_xor_sync(0xffffffffu, b.hi[k].x, o);
            hi.y = __shfl_xor_sync(0xffffffffu, b.hi[k].y, o);
            box_take(b, k, lo, hi);
        }
    }
}

// Order-preserving integer image of a double, for atomics.
__device__ __forceinline__ unsigned long long enc_f64(double d) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(d);
    return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}

__device__ __forceinline__ unsigned long long enc_df(const float2& v) { return enc_f64((double)v.x + (double)v.y); }

// The block's box into the counters (all threads call; 256 threads).
__device__ __forceinline__ void box_publish(DfBox& b, bool bad, Counters* C) {
    __shared__ float2 s_lo[3][8], s_hi[3][8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    box_warp(b);
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            s_lo[k][w] = b.lo[k];
            s_hi[k][w] = b.hi[k];
        }
    }
    bad = __syncthreads_or(bad);
    if (threadIdx.x < 3) {
        float2 lo = s_lo[threadIdx.x][0], hi = s_hi[threadIdx.x][0];
        for (int j = 1; j < 8; ++j) {
            if (df_less(s_lo[threadIdx.x][j], lo)) lo = s_lo[threadIdx.x][j];
            if (df_less(hi, s_hi[threadIdx.x][j])) hi = s_hi[threadIdx.x][j];
        }
        atomicMin(&C->bbox_min[threadIdx.x], enc_df(lo));
        atomicMax(&C->bbox_max[threadIdx.x], enc_df(hi));
    }
    if (threadIdx.x == 0 && bad) atomicOr(&C->status, kStNonFinite);
}

// Closing or opening half-kick of one particle: v += h a, as a double-float
// pair when vl is given (split precision), else in FP32.
__device__ __forceinline__ void kick_v(float4& v, float4* vl, float h, const float4& a) {
    if (vl) {
        df_add_prod(v.x, vl->x, h, a.x, 0.f);
        df_add_prod(v.y, vl->y, h, a.y, 0.f);
        df_add_prod(v.z, vl->z, h, a.z, 0.f);
    } else {
        v.x = fmaf(h, a.x, v.x);
        v.y = fmaf(h, a.y, v.y);
        v.z = fmaf(h, a.z, v.z);
    }
}

// System of a slot (binary search over the offsets).
__device__ __forceinline__ int forest_system(const Forest& F, long long k) {
    int lo = 0, hi = F.nsys - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (F.off[mid] <= k)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// ---- launchers (each enqueues on `s`; no host synchronisation) ----
void launch_bbox(const float4* pos, const float4* plo, long long n, Counters* C, cudaStream_t s);
void launch_root(Counters* C, long long n, float4* frame, cudaStream_t s);
// Ensemble: per-system bounding boxes and root cubes (F.nsys > 1).
void launch_forest_bbox(const float4* pos, const float4* plo, long long n, const Forest& F, Counters* C,
                        cudaStream_t s);
void launch_forest_root(const Forest& F, cudaStream_t s);
void launch_collapse_split(float4* pos, float4* plo, long long n, cudaStream_t s);
// Keys of the current order (vals = 0 .. n-1), in the frames that the root
// kernels wrote.
void launch_keys(const float4* pos, const float4* plo, long long n, Counters* C, const Forest& F, const float4* frame,
                 unsigned long long* keys, unsigned* vals, cudaStream_t s);
// Stable LSD radix sort over bits [shift0, shift0 + kRsDigitBits*passes) of the
// pairs in (keys, vals), or in (keys_alt, vals_alt) where sort_from_alt says so;
// the result ends in (keys, vals).  Returns the number of launches.
bool sort_from_alt(long long n, int passes);
int radix_sort_pairs(SortBuffers& sb, long long n, int passes, int shift0, cudaStream_t s);
// Entries of SortBuffers::hist for n keys: the tile histograms, then the
// digit totals.
long long radix_hist_size(long long n);
void launch_permute(const Particles& P, const unsigned* perm, long long n, bool split, cudaStream_t s);
// Builds the nodes down to level `levels` (keys sorted on their top `levels`
// digits; a node there that would still split sets kStSortDepth) and the leaf
// list; with leaf_scan also B.leaf_before and B.leaf_start.  Returns the number
// of launches.
int launch_tree(NodeArrays& T, Counters* C, const unsigned long long* keys, long long n, int leaf_cap, int max_depth,
                const Forest& F, int levels, const TreeBuffers& B, bool leaf_scan, cudaStream_t s);
// Entries of TreeBuffers::counts.
long long tree_counts_size();
// Leaf and internal moments; also the evaluation's pass list (LB.passes).
// Returns the number of launches.
int launch_moments(NodeArrays& T, Counters* C, const Particles& P, const int* leaf_list, const ListBuffers& LB,
                   long long n, int max_leaves, int leaf_cap, bool split, bool quadrupole, int levels, cudaStream_t s);
void launch_walk(const NodeArrays& T, Counters* C, const int* leaf_list, const WalkParams& wp,
                 const ListBuffers& LB, cudaStream_t s);
void launch_eval(const NodeArrays& T, Counters* C, const Particles& P, const int* leaf_list, const WalkParams& wp,
                 const ListBuffers& LB, int nwarps, cudaStream_t s);
void launch_kick_drift(const Particles& P, long long n, float hdt, float dt, bool split, Counters* C,
                       cudaStream_t s);
void launch_scatter_accel(const Particles& P, long long n, double* ax, double* ay, double* az, cudaStream_t s);

}  // namespace ngrav
