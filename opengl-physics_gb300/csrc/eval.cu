// eval.cu -- force evaluation from the walk's interaction lists: P2C over
// each group's far list, P2P over its near list, and the closing half-kick.
//
// Arithmetic restates the reference (projects/nbody_core/src/Solvers.cpp):
//   P2P  a += G m d / (|d|^2 + eps^2)^(3/2)                 (AccumPairPlummer, :19-38)
//   P2C  the same softened monopole of the node's mass at its COM, plus the
//        unsoftened traceless quadrupole
//        a += -G Q.d / r^5 + 2.5 G (d.Q.d) d / r^7       (AddQuadrupole, :147-179)
// with the group's own members included as a near leaf (the self term is
// zero for eps > 0 and masked for eps == 0).
//
// GB300 mapping.  One warp per pass of a group (dynamic scheduling; a pass is
// up to kTargets of its targets, all for most groups), lane = source: a
// window of list entries sits in registers, two to a packed FP32 operand (add
// / mul / fma .f32x2), and the warp runs down up to kTargets targets, each
// read from shared memory by broadcast, its running sums kept there per lane
// (one conflict-free row of 32 floats per component).  Every lane works on
// every target, whatever the group's size, and a source is loaded once per
// kTargets targets.  The layout before this, lane = target x source slice over
// staged tiles, read every source from shared memory for every pair of
// targets and was bound by that: 86 % of the LSU data pipe at 5 targets a
// group (1M Plummer, leaf capacity 16), 46 % of the FMA pipe.
//  * Near windows: a batch of 64 leaves is laid end to end; a slot finds its
//    leaf from a bit mask of the leaves' first slots and loads its source
//    from global memory into the group's frame.  256 sources a window (four
//    pairs a lane); what a list's end leaves over goes 128 or 64 at a time,
//    and sources that do not fill a window start the next batch.  The next
//    batch's node ids load with this one's first sources, its leaf records
//    (cp.async) while those are evaluated.
//  * Far windows: a list chunk of 128 records (two pairs a lane); node ids are
//    loaded a window ahead, the records gathered.
//  * Sums: each lane sums a window's pairs from zero and adds the result to
//    the target's running sum; these are added across lanes every
//    flush_windows() windows of 64, and in SPLIT precision join the target's
//    total with Kahan compensation.
// What bounds it: the FP32 pipe's operand reads.  A packed step with two
// distinct register operands takes 2 cycles, with three 3 (measured), so a
// pair of sources costs 24 to 27 cycles per target (12 steps, 24 FMA-pipe
// cycles) and a pair of far records about 83 (34 steps); mixing in scalar
// FP32 steps costs more than packed ones (an FFMA beside packed steps: 2
// cycles).  Marginal cost, from running each loop twice: 8.1 ms for the 18.3 G
// pairs and 5.5 ms for the 4.6 G far terms of the 4M galaxy at theta 0.63,
// where the whole kernel took 16.1 ms (groups then still one unit each).
// Measured before -> after, evaluation kernel: 1M Plummer, leaf 16, PLAIN
// 7.87 -> 6.4 ms; 131,071, leaf 16 1.30 -> 0.91; 64-system ensemble, leaf 32
// 4.56 -> 3.8; 4M galaxy, leaf 40 17.7 -> 15.7, learned test, leaf 48 6.98 ->
// 6.6; 16.8M ball, leaf 32 28.6 -> 26.7; 20,011, leaf 8, spline 0.46 -> 0.28.
// Tried: sums in registers, targets unrolled: the loops outgrew the SM's
// instruction cache (95 % of the instruction path's request rate; 22.2 ms on
// the 4M galaxy).  Scalar FFMA sums 17.2 ms, 8, 16, 24 and 32 targets a pass
// 18.8, 16.3, 16.5 and 17.8, a prefetched target 16.7, 128-source windows
// 17.9, 96 registers (5 CTAs) 17.3.  Groups handed out in key-order ranges per
// SM, for L1 reuse: 1 to 3 % slower, most of shared memory being in use.
#include "engine.cuh"
#include "softening.cuh"
#include "walk_common.cuh"

namespace ngrav {

constexpr int kEvalWarps = 4;
constexpr int kEvalThreads = kEvalWarps * 32;
constexpr int kEvalMinBlocks = 4;             // CTAs per SM (128 registers per thread)
constexpr int kTargets = kPassMax;            // targets per pass at most
constexpr int kBatch = 64;                    // leaves per near batch, and the sources
constexpr int kSlots = 1024;                  //   one batch may cover
constexpr int kWide = 4;                      // source pairs per lane in a wide near window
// Windows of 64 between flushes of the lanes' sums.  SPLIT compensates at every
// flush; at 16, with one between the far and the near field, its rounding
// error against FP64 sums over the same lists is at or below that of the
// earlier chunk-wise compensation (Plummer and galaxy, leaves of 8 to 64:
// rms 6.4e-8 to 7.6e-8 against 6.4e-8 to 8.0e-8; at 32 up to 1.6 % above it
// at leaf capacity 40, 1.4 % faster).  PLAIN only adds the flushes up, so
// fewer of them are better (rms 6.7e-8 to 8.9e-8 at 32, 9.2e-8 to 1.3e-7
// before).
constexpr int flush_windows(bool split) { return split ? 16 : 32; }
constexpr float kFarPad = 1e18f;              // position of the massless source that pads a window

static_assert(kSlots == 1024, "one word of start bits per lane");

struct __align__(16) EvalSmem {
    float sum[3 * kTargets][33];              // running sums: row 3 t + axis, one float per lane (and a pad)
    float4 nhi[kBatch];                       // next near batch's leaf records (cp.async): centre hi, start
    float4 nlo[kBatch];                       //   centre lo, count
    float4 leaf[kBatch];                      // batch: frame shift, source index minus slot (int bits)
    unsigned starts[kSlots / 32];             // bit per slot of the batch: a leaf starts there
    float4 txy[kTargets];                     // targets, negated and duplicated: -x -x -y -y
    float2 tz[kTargets];                      //   -z -z
    unsigned long long npairs, nterms;        // interaction counters of this warp
};

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Two sources against target t: the reference's softened pair
// (Solvers.cpp:19-38, AccumPairPlummer) for each, FP32.
// SOFT: 0 Plummer, 1 Plummer with eps = 0 (the self pair gives 0), 2 spline.
struct NearPair {
    float2 x, y, z, m;
};

// FIRST starts the window's sums a, else it adds to them.
template <int SOFT, bool FIRST>
__device__ __forceinline__ void p2p_pair2(const NearPair& q, const float4& xy, const float2& tz, float2 e2, float ih,
                                          float2& ax, float2& ay, float2& az) {
    const float2 dx = add2(q.x, make_float2(xy.x, xy.y));
    const float2 dy = add2(q.y, make_float2(xy.z, xy.w));
    const float2 dz = add2(q.z, tz);
    float2 f;
    if (SOFT == 2) {
        const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
        f = make_float2(pair_factor<kSoftSpline>(r2.x, q.m.x, 0.f, ih), pair_factor<kSoftSpline>(r2.y, q.m.y, 0.f, ih));
    } else {
        const float2 r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, e2)));
        const float2 ir = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
        f = mul2(q.m, mul2(mul2(ir, ir), ir));
        if (SOFT == 1) {
            f.x = r2.x > 0.f ? f.x : 0.f;
            f.y = r2.y > 0.f ? f.y : 0.f;
        }
    }
    ax = FIRST ? mul2(f, dx) : fma2(f, dx, ax);
    ay = FIRST ? mul2(f, dy) : fma2(f, dy, ay);
    az = FIRST ? mul2(f, dz) : fma2(f, dz, az);
}

// Adds a window's sums to the target's running ones: one rounding at the
// running sum's size per window, whatever the window's width.
__device__ __forceinline__ void add_window(EvalSmem& sm, int t, int lane, float2 ax, float2 ay, float2 az) {
    sm.sum[3 * t][lane] += ax.x + ax.y;
    sm.sum[3 * t + 1][lane] += ay.x + ay.y;
    sm.sum[3 * t + 2][lane] += az.x + az.y;
}

// A near window of N pairs per lane against the pass's targets.
template <int SOFT, int N>
__device__ __forceinline__ void p2p_window(EvalSmem& sm, int nt, const NearPair (&q)[N], float2 e2, float ih,
                                           int lane) {
#pragma unroll 1
    for (int t = 0; t < nt; ++t) {
        const float4 xy = sm.txy[t];
        const float2 tz = sm.tz[t];
        float2 ax, ay, az;
        p2p_pair2<SOFT, true>(q[0], xy, tz, e2, ih, ax, ay, az);
#pragma unroll
        for (int k = 1; k < N; ++k) p2p_pair2<SOFT, false>(q[k], xy, tz, e2, ih, ax, ay, az);
        add_window(sm, t, lane, ax, ay, az);
    }
}

// Two far records against target t: the softened monopole of each node's
// mass at its COM plus the unsoftened quadrupole (Solvers.cpp:147-179,
// AddQuadrupole).  The quadrupole is held negated, so that neither of its
// terms needs a sign change (packed operands have no free negation), and the
// monopole and the radial quadrupole term share one multiplier of the offset.
struct FarPair {
    float2 x, y, z, m;
    float2 qxx, qyy, qzz, qxy, qxz, qyz;  // -Q
};

template <bool QUAD, int SOFT, bool FIRST>
__device__ __forceinline__ void p2c_pair2(const FarPair& q, const float4& xy, const float2& tz, float2 e2, float ih,
                                          float2& ax, float2& ay, float2& az) {
    const float2 dx = add2(q.x, make_float2(xy.x, xy.y));
    const float2 dy = add2(q.y, make_float2(xy.z, xy.w));
    const float2 dz = add2(q.z, tz);
    const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
    float2 fm;
    if (SOFT == 2) {
        fm = make_float2(pair_factor<kSoftSpline>(r2.x, q.m.x, e2.x, ih),
                         pair_factor<kSoftSpline>(r2.y, q.m.y, e2.x, ih));
    } else {
        const float2 re = add2(r2, e2);
        const float2 is = make_float2(rsqrtf(re.x), rsqrtf(re.y));
        fm = mul2(q.m, mul2(mul2(is, is), is));
    }
    if (QUAD) {
        // operands shared by neighbouring steps: dz, then dy, then dx
        float2 qdx = mul2(q.qxz, dz), qdy = mul2(q.qyz, dz), qdz = mul2(q.qzz, dz);
        qdx = fma2(q.qxy, dy, qdx);
        qdy = fma2(q.qyy, dy, qdy);
        qdz = fma2(q.qyz, dy, qdz);
        qdx = fma2(q.qxx, dx, qdx);
        qdy = fma2(q.qxy, dx, qdy);
        qdz = fma2(q.qxz, dx, qdz);
        const float2 qd2 = fma2(dx, qdx, fma2(dy, qdy, mul2(dz, qdz)));
        const float2 ir = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
        const float2 ir2 = mul2(ir, ir);
        const float2 ir5 = mul2(mul2(ir2, ir2), ir);
        fm = fma2(mul2(dup2(-2.5f), qd2), mul2(ir5, ir2), fm);
        ax = FIRST ? mul2(ir5, qdx) : fma2(ir5, qdx, ax);
        ay = FIRST ? mul2(ir5, qdy) : fma2(ir5, qdy, ay);
        az = FIRST ? mul2(ir5, qdz) : fma2(ir5, qdz, az);
    }
    ax = FIRST && !QUAD ? mul2(fm, dx) : fma2(fm, dx, ax);
    ay = FIRST && !QUAD ? mul2(fm, dy) : fma2(fm, dy, ay);
    az = FIRST && !QUAD ? mul2(fm, dz) : fma2(fm, dz, az);
}

// A far window of N record pairs per lane against the pass's targets.
template <bool QUAD, int SOFT, int N>
__device__ __forceinline__ void p2c_window(EvalSmem& sm, int nt, const FarPair (&q)[N], float2 e2, float ih,
                                           int lane) {
#pragma unroll 1
    for (int t = 0; t < nt; ++t) {
        const float4 xy = sm.txy[t];
        const float2 tz = sm.tz[t];
        float2 ax, ay, az;
        p2c_pair2<QUAD, SOFT, true>(q[0], xy, tz, e2, ih, ax, ay, az);
#pragma unroll
        for (int k = 1; k < N; ++k) p2c_pair2<QUAD, SOFT, false>(q[k], xy, tz, e2, ih, ax, ay, az);
        add_window(sm, t, lane, ax, ay, az);
    }
}

// One far record in the group's frame (node < 0, unless FULL: the massless pad).
struct FarRec {
    float x, y, z, m, qxx, qyy, qzz, qxy, qxz, qyz;
};

template <bool SPLIT, bool QUAD, bool FULL>
__device__ __forceinline__ FarRec far_record(const NodeArrays& T, int node, const float4& gh, const float4& gl) {
    FarRec r = {kFarPad, kFarPad, kFarPad, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (FULL || node >= 0) {
        const float4 A = T.wA[node], D = T.wD[node];
        r.x = A.x;
        r.y = A.y;
        r.z = A.z;
        if (SPLIT) {
            r.x = (A.x - gh.x) + (D.x - gl.x);
            r.y = (A.y - gh.y) + (D.y - gl.y);
            r.z = (A.z - gh.z) + (D.z - gl.z);
        }
        r.m = A.w;
        if (QUAD) {
            const float4 B = T.wB[node];
            r.qxx = -B.x;
            r.qyy = -B.y;
            r.qzz = B.x + B.y;  // traceless
            r.qxy = -B.z;
            r.qxz = -B.w;
            r.qyz = -D.w;
        }
    }
    return r;
}

template <bool SPLIT, bool QUAD, bool FULL>
__device__ __forceinline__ FarPair far_pair(const NodeArrays& T, int n0, int n1, const float4& gh, const float4& gl) {
    const FarRec a = far_record<SPLIT, QUAD, FULL>(T, n0, gh, gl), b = far_record<SPLIT, QUAD, FULL>(T, n1, gh, gl);
    return {make_float2(a.x, b.x),     make_float2(a.y, b.y),     make_float2(a.z, b.z),     make_float2(a.m, b.m),
            make_float2(a.qxx, b.qxx), make_float2(a.qyy, b.qyy), make_float2(a.qzz, b.qzz), make_float2(a.qxy, b.qxy),
            make_float2(a.qxz, b.qxz), make_float2(a.qyz, b.qyz)};
}

__device__ __forceinline__ void kahan_add(float& s, float& c, float v) {
    const float y = v - c, t = s + y;
    c = (t - s) - y;
    s = t;
}

// Totals of a pass: lane l holds rows l, l + 32, .. (row = 3 target + axis).
constexpr int kRowsPerLane = (3 * kTargets + 31) / 32;
struct Total {
    float s[kRowsPerLane] = {}, c[kRowsPerLane] = {};
};

// Adds every row's 32 lane sums into its total (and clears them): eight chains
// of four, then a tree, in the same order whatever the row, so a target's sum
// does not depend on its place in the pass.  The pad keeps the 32 rows read
// together clear of each other's banks.
template <bool SPLIT>
__device__ __forceinline__ void flush(EvalSmem& sm, int nt, Total& g, int lane, bool clear = true) {
    __syncwarp();
#pragma unroll
    for (int h = 0; h < kRowsPerLane; ++h) {
        const int row = 32 * h + lane;
        if (row < 3 * nt) {
            float v[8];
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                const float x = sm.sum[row][k];
                v[k & 7] = k < 8 ? x : v[k & 7] + x;
            }
            const float t = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
            if (SPLIT)
                kahan_add(g.s[h], g.c[h], t);
            else
                g.s[h] += t;
        }
    }
    __syncwarp();
    if (clear)
        for (int r = 0; r < 3 * nt; ++r) sm.sum[r][lane] = 0.f;
}

// One axis of a target's acceleration: stored, and the closing half-kick.
template <bool SPLIT>
__device__ __forceinline__ void finish_row(const Total& g, int h, int row, int first, const WalkParams& wp,
                                           float4* __restrict__ acc, float4* __restrict__ vel,
                                           float4* __restrict__ vlo) {
    const int slot = first + row / 3, axis = row % 3;
    const float a = wp.G * g.s[h];
    float* out = reinterpret_cast<float*>(acc + slot);
    out[axis] = a;
    if (axis == 0) out[3] = 0.f;
    if (wp.kick) {
        float* v = reinterpret_cast<float*>(vel + slot) + axis;
        if (SPLIT) {
            float* l = reinterpret_cast<float*>(vlo + slot) + axis;
            float vh = *v, vl = *l;
            df_add_prod(vh, vl, wp.hdt, a, 0.f);
            *v = vh;
            *l = vl;
        } else {
            *v = fmaf(wp.hdt, a, *v);
        }
    }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// A near list being read: the next entry and the chunks that hold entries
// pos .. pos + kBatch - 1 (ca holds pos, cb is the one after).
struct NearCursor {
    int pos, ca, cb;
};

__device__ __forceinline__ NearCursor near_begin(const ListBuffers& LB, int first, int nnear) {
    return {0, first, nnear > kListChunk ? LB.near_next[first] : -1};
}

__device__ __forceinline__ void near_advance(const ListBuffers& LB, NearCursor& W, int nb, int nnear) {
    const int np = W.pos + nb;  // nb <= kBatch < kListChunk: at most one chunk further
    if ((np >> 7) != (W.pos >> 7)) {
        W.ca = W.cb;
        W.cb = ((np >> 7) + 1) * kListChunk < nnear ? LB.near_next[W.ca] : -1;
    }
    W.pos = np;
}

// Node ids of the batch at the cursor (lane: entries pos + lane and pos + 32 +
// lane; -1 past the list).
__device__ __forceinline__ int2 near_ids(const ListBuffers& LB, const NearCursor& W, int nnear, int lane) {
    int id[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int e = W.pos + 32 * h + lane;
        const int c = (e >> 7) == (W.pos >> 7) ? W.ca : W.cb;
        id[h] = e < nnear ? __ldg(LB.near + (long long)c * kListChunk + (e & (kListChunk - 1))) : -1;
    }
    return make_int2(id[0], id[1]);
}

// Their leaf records copied into shared memory by cp.async, so they cost no
// registers while the batch before is evaluated.  Past the list: count 0.
__device__ __forceinline__ void prefetch_near(EvalSmem& sm, const NodeArrays& T, int2 ids, int lane) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int node = h ? ids.y : ids.x;
        if (node >= 0) {
            cp_async16(&sm.nhi[32 * h + lane], &T.chi[node]);
            cp_async16(&sm.nlo[32 * h + lane], &T.clo[node]);
        } else {
            sm.nlo[32 * h + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

__device__ __forceinline__ void prefetch_wait() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
}

// N source pairs per lane from the batch's slots base .. base + 64 N, in the
// group's frame (unless FULL, slots past `used` are massless pads far away);
// all loads in flight together.  A slot's leaf is the number of leaves that
// start up to it, less one: those before the window (`before`) plus the start
// bits up to the slot.
template <bool SPLIT, int N, bool FULL>
__device__ __forceinline__ void near_load(const EvalSmem& sm, const float4* __restrict__ src, int base, int used,
                                          int& before, int lane, NearPair (&q)[N]) {
    const unsigned upto = 0xffffffffu >> (31 - lane);
    float4 v[2 * N];
    int rank[2 * N];
#pragma unroll
    for (int k = 0; k < 2 * N; ++k) {
        const int slot = base + 32 * k + lane;
        const unsigned starts = sm.starts[(base >> 5) + k];
        rank[k] = before + __popc(starts & upto);
        before += __popc(starts);
        if (!FULL) v[k] = make_float4(kFarPad, kFarPad, kFarPad, 0.f);
        if (FULL || slot < used) v[k] = __ldg(src + (slot + __float_as_int(sm.leaf[rank[k]].w)));
    }
    if (SPLIT) {
#pragma unroll
        for (int k = 0; k < 2 * N; ++k) {
            const float4 sh = sm.leaf[rank[k]];
            v[k].x += sh.x;
            v[k].y += sh.y;
            v[k].z += sh.z;
        }
    }
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const float4 a = v[2 * k], b = v[2 * k + 1];
        q[k] = {make_float2(a.x, b.x), make_float2(a.y, b.y), make_float2(a.z, b.z), make_float2(a.w, b.w)};
    }
}

template <bool SPLIT, bool QUAD, int SOFT>
__global__ void __launch_bounds__(kEvalThreads, kEvalMinBlocks) eval_kernel(NodeArrays T, Counters* C,
                                                            const float4* __restrict__ src,
                                                            float4* __restrict__ acc, float4* __restrict__ vel,
                                                            float4* __restrict__ vlo,
                                                            const int* __restrict__ leaf_list, WalkParams wp,
                                                            ListBuffers LB) {
    __shared__ EvalSmem smem[kEvalWarps];
    const int lane = threadIdx.x & 31;
    EvalSmem& sm = smem[threadIdx.x >> 5];
    if (C->status & kStFatal) return;
    if (lane == 0) sm.npairs = sm.nterms = 0ull;
    // Sources per near batch at most: the tuned tile, 256 or 0 for all there is room for.
    const int tile = wp.p2p_tile > 0 && wp.p2p_tile < 256 ? (wp.p2p_tile + 63) & ~63 : kSlots;
    const float2 e2 = dup2(wp.eps2);

    // Units of work: the passes past each group's first (they belong to the
    // largest groups), then every group's first.
    const int extra = C->extra_passes, units = extra + C->nleaves;
    const int pass = pass_targets(C->nleaves);
    int next = 0;
    if (lane == 0) next = atomicAdd(&C->eval_next, 1);
    for (;;) {
        const int unit = __shfl_sync(0xffffffffu, next, 0);
        if (unit >= units) break;
        if (lane == 0) next = atomicAdd(&C->eval_next, 1);  // the next unit's index arrives while this one runs
        const int2 gp = unit < extra ? LB.passes[unit] : make_int2(unit - extra, 0);
        const int leaf = leaf_list[gp.x];
        const int4 gin = LB.ginfo[gp.x];
        const int far_first = gin.x, near_first = gin.y, nfar = gin.z, nnear = gin.w;
        const float4 gh = T.chi[leaf], gl = T.clo[leaf];
        // even passes: the first gcount % passes of them take one target more
        const int gcount = __float_as_int(gl.w), passes = (gcount + pass - 1) / pass;
        const int each = gcount / passes, odd = gcount % passes;
        const int nt = each + (gp.y < odd ? 1 : 0);
        const int first = __float_as_int(gh.w) + gp.y * each + min(gp.y, odd);  // first target's slot
        NearCursor W = near_begin(LB, near_first, nnear);
        const int2 ids0 = near_ids(LB, W, nnear, lane);
        int id[4];                                     // the first far window's ids
#pragma unroll
        for (int k = 0; k < 4; ++k)
            id[k] = 32 * k + lane < nfar ? LB.far[(long long)far_first * kListChunk + 32 * k + lane] : -1;
        __syncwarp();
        static_assert(kTargets <= 32, "one target per lane");
        if (lane < nt) {
            const float4 t = src[first + lane];
            sm.txy[lane] = make_float4(-t.x, -t.x, -t.y, -t.y);
            sm.tz[lane] = make_float2(-t.z, -t.z);
        }
        prefetch_near(sm, T, ids0, lane);
        __syncwarp();
        for (int r = 0; r < 3 * nt; ++r) sm.sum[r][lane] = 0.f;
        Total total;
        int windows = 0;

        // ---- far field: a chunk of 128 records a window, or its last 64 ----
        for (int b = 0, cur = far_first; b < nfar; b += kListChunk) {
            int n[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                n[k] = id[k];
                id[k] = -1;
            }
            const int e = b + kListChunk;  // the next window's ids
            if (e < nfar) {
                cur = LB.far_next[cur];
                const int* ids = LB.far + (long long)cur * kListChunk + lane;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (e + 32 * k + lane < nfar) id[k] = ids[32 * k];
            }
            if (nfar - b > 64) {
                FarPair q[2];
                q[0] = far_pair<SPLIT, QUAD, true>(T, n[0], n[1], gh, gl);
                q[1] = far_pair<SPLIT, QUAD, false>(T, n[2], n[3], gh, gl);
                p2c_window<QUAD, SOFT, 2>(sm, nt, q, e2, wp.ih, lane);
                windows += 2;
            } else {
                const FarPair q[1] = {far_pair<SPLIT, QUAD, false>(T, n[0], n[1], gh, gl)};
                p2c_window<QUAD, SOFT, 1>(sm, nt, q, e2, wp.ih, lane);
                ++windows;
            }
            if (windows >= flush_windows(SPLIT)) {
                flush<SPLIT>(sm, nt, total, lane);
                windows = 0;
            }
        }

        if (SPLIT && windows > 0) {
            flush<SPLIT>(sm, nt, total, lane);
            windows = 0;
        }

        // ---- near field: batches of up to kBatch leaves ----
        int skip = 0;                                  // sources of the batch's first leaf already taken
        long long staged = 0;
        while (W.pos < nnear) {
            prefetch_wait();
            sm.starts[lane] = 0u;
            // lane: leaves 2 lane and 2 lane + 1 of the batch, so one scan orders both
            int start[2], cnt[2];
            float3 sh[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float4 hi = sm.nhi[2 * lane + h], lo = sm.nlo[2 * lane + h];
                start[h] = __float_as_int(hi.w);
                cnt[h] = __float_as_int(lo.w);
                sh[h] = make_float3(0.f, 0.f, 0.f);
                if (SPLIT)
                    sh[h] = make_float3((hi.x - gh.x) + (lo.x - gl.x), (hi.y - gh.y) + (lo.y - gl.y),
                                        (hi.z - gh.z) + (lo.z - gl.z));
            }
            if (lane == 0) {
                start[0] += skip;
                cnt[0] -= skip;
            }
            __syncwarp();
            int tot;
            const int ex0 = warp_excl_scan(cnt[0] + cnt[1], lane, tot), ex1 = ex0 + cnt[0];
            // whole windows, the wide ones if there is one, unless this is
            // the end of the list (or the batch does not fill one)
            const bool last = W.pos + kBatch >= nnear;
            const int whole = tot >= 64 * kWide ? tot & ~(64 * kWide - 1) : (tot >= 64 ? tot & ~63 : tot);
            const int used = min(last ? tot : whole, tile);
            // leaves consumed whole (a prefix), and where the next one begins
            const int nb = min(nnear - W.pos, __popc(__ballot_sync(0xffffffffu, ex1 <= used)) +
                                                  __popc(__ballot_sync(0xffffffffu, ex1 + cnt[1] <= used)));
            const int ex_even = __shfl_sync(0xffffffffu, ex0, nb >> 1);
            const int ex_odd = __shfl_sync(0xffffffffu, ex1, nb >> 1);
            skip = nb == 0 ? skip + used : (nb < kBatch ? used - (nb & 1 ? ex_odd : ex_even) : 0);
            // by rank among the non-empty leaves
            const unsigned has0 = __ballot_sync(0xffffffffu, cnt[0] > 0);
            const unsigned has1 = __ballot_sync(0xffffffffu, cnt[1] > 0);
            const unsigned below = (1u << lane) - 1u;
            const int r0 = __popc(has0 & below) + __popc(has1 & below);
            if (cnt[0] > 0) sm.leaf[r0] = make_float4(sh[0].x, sh[0].y, sh[0].z, __int_as_float(start[0] - ex0));
            if (cnt[1] > 0)
                sm.leaf[r0 + (cnt[0] > 0)] = make_float4(sh[1].x, sh[1].y, sh[1].z, __int_as_float(start[1] - ex1));
            if (cnt[0] > 0 && ex0 < kSlots) atomicOr(&sm.starts[ex0 >> 5], 1u << (ex0 & 31));
            if (cnt[1] > 0 && ex1 < kSlots) atomicOr(&sm.starts[ex1 >> 5], 1u << (ex1 & 31));
            near_advance(LB, W, nb, nnear);
            __syncwarp();
            staged += used;
            // the next batch's ids load with this one's first sources,
            // its leaf records while those are evaluated
            const bool more = W.pos < nnear;
            int2 ids = make_int2(-1, -1);
            if (more) ids = near_ids(LB, W, nnear, lane);
            int before = -1;
            bool ahead = more;
#pragma unroll 1
            for (int base = 0; base < used;) {
                const int left = used - base;
                if (left >= 64 * kWide) {
                    NearPair q[kWide];
                    near_load<SPLIT, kWide, true>(sm, src, base, used, before, lane, q);
                    if (ahead) prefetch_near(sm, T, ids, lane);
                    p2p_window<SOFT, kWide>(sm, nt, q, e2, wp.ih, lane);
                    base += 64 * kWide;
                    windows += kWide;
                } else if (left > 64) {
                    NearPair q[2];
                    near_load<SPLIT, 2, false>(sm, src, base, used, before, lane, q);
                    if (ahead) prefetch_near(sm, T, ids, lane);
                    p2p_window<SOFT, 2>(sm, nt, q, e2, wp.ih, lane);
                    base += 128;
                    windows += 2;
                } else {
                    NearPair q[1];
                    near_load<SPLIT, 1, false>(sm, src, base, used, before, lane, q);
                    if (ahead) prefetch_near(sm, T, ids, lane);
                    p2p_window<SOFT, 1>(sm, nt, q, e2, wp.ih, lane);
                    base += 64;
                    ++windows;
                }
                ahead = false;
                if (windows >= flush_windows(SPLIT)) {
                    flush<SPLIT>(sm, nt, total, lane);
                    windows = 0;
                }
            }
            __syncwarp();
        }
        flush<SPLIT>(sm, nt, total, lane, false);
        if (lane == 0) {
            sm.nterms += (unsigned long long)nt * (unsigned long long)nfar;
            sm.npairs += (unsigned long long)nt * (unsigned long long)staged - (unsigned long long)nt;
        }

        // ---- write a, closing kick ----
#pragma unroll
        for (int h = 0; h < kRowsPerLane; ++h)
            if (32 * h + lane < 3 * nt) finish_row<SPLIT>(total, h, 32 * h + lane, first, wp, acc, vel, vlo);
    }
    __syncwarp();
    if (lane == 0) {
        atomicAdd(&C->p2p_pairs, sm.npairs);
        atomicAdd(&C->p2c_terms, sm.nterms);
    }
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------

int eval_warps_per_block() { return kEvalWarps; }

#define NGRAV_EVAL_INSTANCES(X)                                                       \
    X(true, true, 0) X(true, true, 1) X(true, true, 2) X(true, false, 0) X(true, false, 1) \
    X(true, false, 2) X(false, true, 0) X(false, true, 1) X(false, true, 2) X(false, false, 0) \
    X(false, false, 1) X(false, false, 2)

int eval_blocks_per_sm() {
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, eval_kernel<true, true, 0>, kEvalThreads, 0);
    return nb > 0 ? nb : 1;
}

void launch_eval(const NodeArrays& T, Counters* C, const Particles& P, const int* leaf_list, const WalkParams& wp,
                 const ListBuffers& LB, int nwarps, cudaStream_t s) {
    const int blocks = (nwarps + kEvalWarps - 1) / kEvalWarps;
    const int soft = wp.soft == kSoftSpline ? 2 : (!(wp.eps2 > 0.f) ? 1 : 0);
#define NGRAV_LAUNCH(SP, Q, Z)                                                                             \
    if (wp.split == (SP) && (wp.quadrupole != 0) == (Q) && soft == (Z))                                   \
        eval_kernel<SP, Q, Z><<<blocks, kEvalThreads, 0, s>>>(T, C, P.src, P.acc, P.vel, P.vlo, leaf_list, wp, LB);
    NGRAV_EVAL_INSTANCES(NGRAV_LAUNCH)
#undef NGRAV_LAUNCH
}

}  // namespace ngrav
