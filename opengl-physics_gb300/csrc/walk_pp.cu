// walk_pp.cu -- the per-particle walk of the reference (WalkBH,
// projects/nbody_core/src/Solvers.cpp:181-227), used by the relative
// (GADGET-2) opening test (ComputeAccelBarnesHutPerParticle, :359-382) and by
// the block-timestep integrator's target subsets (ComputeAccelBarnesHutTargets,
// :384-405).
//
// Every target decides every node on its own path:
//   leaf:      exact pairs with each member but itself;
//   internal:  accepted (softened monopole + unsoftened quadrupole) iff
//              geometric: (2h)^2 < theta^2 d^2, d = |com - x_target|;
//              relative:  M (2h)^2 < alpha |a_old| d^4 / G when |a_old| > 0,
//                         the geometric test otherwise (Mac.hpp:31-42);
//              otherwise its children are visited.
// GPU mapping: one warp per slice of kPpTargets consecutive particles
// (key order, so neighbours in space), the active ones of them its members,
// lane = node or source.  The warp walks the union of the members' paths; each
// stack entry carries the mask of members still on that path, so a member that
// accepts a node stops there while the others descend, and the result of every
// member is exactly its own walk.  32 entries are taken off the stack at once,
// one per lane: the lane decides its node for every member in turn (members
// broadcast from shared memory), and the node's accepting members, its reached
// leaf or its opened children go to three buffers.  Far nodes are evaluated 64
// at a time, leaves' particles 64 at a time, two per lane on the packed FP32
// pipe, each with its mask of members.  (The layout before this, one leaf a
// warp, lane = member, node after node, left all but the leaf's members idle,
// 2.8 of 32 lanes at leaf capacity 8, and ran the particles of every reached
// leaf one after another on dependent loads.)  Sums are FP32 with error
// compensation, per window and across lanes; differences use the double-float
// positions; a test within a relative 1e-5 of its threshold is re-taken in
// FP64 on the FP64 moments.
// Latency-bound (16 warps an SM).  Measured before -> after: relative test,
// 49,999 bodies, leaf capacity 8 9.56 -> 1.16 ms, 16,384 at leaf capacity 64
// 6.88 -> 0.57; block substep of 4,096 bodies 0.78 -> 0.09.  Four members, with
// their sums in registers, are the best slice: with 16 and the sums in shared
// memory 49,999 bodies took 2.5 ms, a leaf a warp 2.0, eight members 2.1, two
// 1.01 (but 2.68 against 2.14 at leaf capacity 64).
#include "engine.cuh"
#include "softening.cuh"
#include "walk_common.cuh"

namespace ngrav {

constexpr int kPpWarps = 4;
constexpr int kPpThreads = kPpWarps * 32;
constexpr int kPpTargets = 4;     // particles per slice: members walked together at most
constexpr int kPpStack = 1024;    // union of the members' paths
// Entries kept free for a walk that takes one node at a time: it leaves at most
// seven siblings waiting per level.  Full up to here, the walk goes on so until
// it is below again, and no tree outgrows the stack.  (A full stack cannot end
// the walk: the slices done by then have had their closing kick.)  49,999 bodies
// at leaf capacity 8, relative test, and substeps of 4,096: as fast as without.
constexpr int kPpReserve = 7 * kMaxLevels;
constexpr int kPpBuffer = 128;    // far nodes / near leaves waiting: 64 make a window or batch
constexpr float kPpPad = 1e18f;   // position of the masked source that pads a window

struct PpParams {
    int relative;                     // relative MAC (else geometric)
    float alpha;                      // relative MAC tolerance
    double alpha_d;
    int n;                            // particles
    const unsigned* before;           // per slot: leaves that start before it
    const unsigned* starts;           // per slot: 1 if a leaf starts there
    // block timesteps (System::BlockStep): only particles whose rung step
    // (rung in vel.w) ends at finest substep `sub` + 1, each closing with its
    // own half-kick 0.5 base / 2^rung
    int block, sub, rmax;
    double base;
};

struct __align__(16) PpSmem {
    float4 hi[kPpTargets];            // member: position, alpha |a_old| (< 0: the geometric test)
    float4 lo[kPpTargets];            //   low halves, |a_old|
    int slot[kPpTargets];
    float hdt[kPpTargets];            // closing half-kick
    int snode[kPpStack];              // walk stack: node and members on its path
    unsigned char smask[kPpStack];
    int fnode[kPpBuffer];             // accepted nodes and the members that accepted them
    unsigned char fmask[kPpBuffer];
    int nstart[kPpBuffer], ncount[kPpBuffer];  // reached leaves and the members that reached them
    unsigned char nmask[kPpBuffer];
    int delta[64];                    // batch of leaves: source index minus slot
    unsigned char bmask[64];
};

// Two sources or node centres (double-float) of one lane, and their members.
struct PpPair {
    float2 x, y, z, m;
    float2 lx, ly, lz;
    unsigned ma, mb;
};

// Offsets to member t: (hi - hi) + (lo - lo).
template <bool SPLIT>
__device__ __forceinline__ void pp_offset(const PpSmem& sm, int t, const PpPair& q, float2& dx, float2& dy, float2& dz) {
    const float4 h = sm.hi[t];
    dx = add2(q.x, dup2(-h.x));
    dy = add2(q.y, dup2(-h.y));
    dz = add2(q.z, dup2(-h.z));
    if (SPLIT) {
        const float4 l = sm.lo[t];
        dx = add2(dx, add2(q.lx, dup2(-l.x)));
        dy = add2(dy, add2(q.ly, dup2(-l.y)));
        dz = add2(dz, add2(q.lz, dup2(-l.z)));
    }
}

// A lane's running force on one member, with what it rounded off.
struct PpSum {
    float s[3], low[3];
    __device__ __forceinline__ void add(const float v[3]) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            float t, e;
            two_sum(s[k], v[k], t, e);
            s[k] = t;
            low[k] += e;
        }
    }
};

template <bool SPLIT, bool QUAD, int SOFT>
struct PpWalk {
    PpSmem& sm;
    const NodeArrays& T;
    const Particles& P;
    const WalkParams& wp;
    const int lane;
    int nt;                           // members
    PpSum sum[kPpTargets];            // this lane's share of their forces

    // The first `n` <= 64 buffered far nodes: softened monopole plus unsoftened
    // quadrupole (AddQuadrupole, Solvers.cpp:147-179) for the members that
    // accepted them.
    __device__ __forceinline__ void far_window(int n) {
        PpPair q;
        float4 A[2], B[2], D[2];
        unsigned m[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int e = 32 * h + lane;
            A[h] = make_float4(kPpPad, kPpPad, kPpPad, 0.f);
            B[h] = D[h] = make_float4(0.f, 0.f, 0.f, 0.f);
            m[h] = 0u;
            if (e < n) {
                const int node = sm.fnode[e];
                m[h] = sm.fmask[e];
                A[h] = T.wA[node];
                D[h] = T.wD[node];
                if (QUAD) B[h] = T.wB[node];
            }
        }
        q.x = make_float2(A[0].x, A[1].x);
        q.y = make_float2(A[0].y, A[1].y);
        q.z = make_float2(A[0].z, A[1].z);
        q.m = make_float2(A[0].w, A[1].w);
        q.lx = make_float2(D[0].x, D[1].x);
        q.ly = make_float2(D[0].y, D[1].y);
        q.lz = make_float2(D[0].z, D[1].z);
        const float2 qxx = make_float2(-B[0].x, -B[1].x), qyy = make_float2(-B[0].y, -B[1].y);
        const float2 qxy = make_float2(-B[0].z, -B[1].z), qxz = make_float2(-B[0].w, -B[1].w);
        const float2 qyz = make_float2(-D[0].w, -D[1].w);
        const float2 qzz = make_float2(B[0].x + B[0].y, B[1].x + B[1].y);  // traceless
#pragma unroll
        for (int t = 0; t < kPpTargets; ++t) {
            if (t >= nt) break;
            const bool a = (m[0] >> t) & 1u, b = (m[1] >> t) & 1u;
            float2 dx, dy, dz;
            pp_offset<true>(sm, t, q, dx, dy, dz);
            const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
            float2 f = make_float2(pair_factor<SOFT>(r2.x, q.m.x, wp.eps2, wp.ih),
                                   pair_factor<SOFT>(r2.y, q.m.y, wp.eps2, wp.ih));
            float2 ir5 = dup2(0.f), qdx = ir5, qdy = ir5, qdz = ir5;
            if (QUAD) {
                qdx = fma2(qxx, dx, fma2(qxy, dy, mul2(qxz, dz)));
                qdy = fma2(qxy, dx, fma2(qyy, dy, mul2(qyz, dz)));
                qdz = fma2(qxz, dx, fma2(qyz, dy, mul2(qzz, dz)));
                const float2 qd2 = fma2(dx, qdx, fma2(dy, qdy, mul2(dz, qdz)));
                const float2 ir = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
                const float2 ir2 = mul2(ir, ir);
                ir5 = mul2(mul2(ir2, ir2), ir);
                f = fma2(mul2(dup2(-2.5f), qd2), mul2(ir5, ir2), f);
                ir5.x = a ? ir5.x : 0.f;
                ir5.y = b ? ir5.y : 0.f;
            }
            f.x = a ? f.x : 0.f;
            f.y = b ? f.y : 0.f;
            const auto force = [&](float2 d, float2 qd) {
                const float first = QUAD ? fmaf(f.x, d.x, ir5.x * qd.x) : f.x * d.x;
                return fmaf(f.y, d.y, QUAD ? fmaf(ir5.y, qd.y, first) : first);
            };
            const float v[3] = {force(dx, qdx), force(dy, qdy), force(dz, qdz)};
            sum[t].add(v);
        }
    }

    // The first `n` <= 64 buffered leaves: exact softened pairs of their
    // particles with the members that reached them, each member's own self
    // excluded (`own`: the slice's first slot, `active` its members' bits).
    __device__ __forceinline__ void near_batch(int n, int own, unsigned active) {
        int cnt[2], first[2], tot0, tot1;
#pragma unroll
        for (int h = 0; h < 2; ++h) cnt[h] = 32 * h + lane < n ? sm.ncount[32 * h + lane] : 0;
        first[0] = warp_excl_scan(cnt[0], lane, tot0);
        first[1] = warp_excl_scan(cnt[1], lane, tot1) + tot0;
        const int tot = tot0 + tot1;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int e = 32 * h + lane;
            if (e < n) {
                sm.delta[e] = sm.nstart[e] - first[h];
                sm.bmask[e] = sm.nmask[e];
            } else {
                first[h] = 0x7fffffff;
            }
        }
        __syncwarp();
        const unsigned upto = 0xffffffffu >> (31 - lane);
        int before = -1;                      // leaves begun before the window, less one
        for (int base = 0; base < tot; base += 64) {
            float4 p[2], l[2];
            unsigned m[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                // bit i: a leaf starts at slot base + 32 h + i
                const unsigned o0 = (unsigned)(first[0] - base - 32 * h), o1 = (unsigned)(first[1] - base - 32 * h);
                const unsigned starts =
                    __reduce_or_sync(0xffffffffu, (o0 < 32u ? 1u << o0 : 0u) | (o1 < 32u ? 1u << o1 : 0u));
                const int rank = before + __popc(starts & upto);
                before += __popc(starts);
                p[h] = make_float4(kPpPad, kPpPad, kPpPad, 0.f);
                l[h] = make_float4(0.f, 0.f, 0.f, 0.f);
                m[h] = 0u;
                const int at = base + 32 * h + lane;
                if (at < tot) {
                    const int j = at + sm.delta[rank];
                    p[h] = P.pos[j];
                    if (SPLIT) l[h] = P.plo[j];
                    m[h] = sm.bmask[rank];
                    const unsigned k = (unsigned)(j - own);
                    if (k < 32u && ((active >> k) & 1u)) m[h] &= ~(1u << __popc(active & ((1u << k) - 1u)));
                }
            }
            PpPair q;
            q.x = make_float2(p[0].x, p[1].x);
            q.y = make_float2(p[0].y, p[1].y);
            q.z = make_float2(p[0].z, p[1].z);
            q.m = make_float2(p[0].w, p[1].w);
            q.lx = make_float2(l[0].x, l[1].x);
            q.ly = make_float2(l[0].y, l[1].y);
            q.lz = make_float2(l[0].z, l[1].z);
#pragma unroll
            for (int t = 0; t < kPpTargets; ++t) {
                if (t >= nt) break;
                float2 dx, dy, dz;
                pp_offset<SPLIT>(sm, t, q, dx, dy, dz);
                const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
                float2 f = make_float2(pair_factor<SOFT>(r2.x, q.m.x, wp.eps2, wp.ih),
                                       pair_factor<SOFT>(r2.y, q.m.y, wp.eps2, wp.ih));
                f.x = (m[0] >> t) & 1u ? f.x : 0.f;
                f.y = (m[1] >> t) & 1u ? f.y : 0.f;
                const float v[3] = {fmaf(f.y, dx.y, f.x * dx.x), fmaf(f.y, dy.y, f.x * dy.x),
                                    fmaf(f.y, dz.y, f.x * dz.x)};
                sum[t].add(v);
            }
            }
        __syncwarp();
    }
};

// Drops the first 64 entries of a buffer of `size` (the rest move down).
template <class V>
__device__ __forceinline__ void pp_drop(V* buf, int size, int lane) {
    V keep[2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if (64 + 32 * h + lane < size) keep[h] = buf[64 + 32 * h + lane];
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if (64 + 32 * h + lane < size) buf[32 * h + lane] = keep[h];
    __syncwarp();
}

template <bool SPLIT, bool QUAD, int SOFT>
__global__ void __launch_bounds__(kPpThreads, 4) walk_pp_kernel(NodeArrays T, Counters* C, Particles P,
                                                             const int* __restrict__ leaf_list, WalkParams wp,
                                                             PpParams pp) {
    extern __shared__ __align__(16) unsigned char pp_smem[];
    const int lane = threadIdx.x & 31;
    PpSmem& sm = reinterpret_cast<PpSmem*>(pp_smem)[threadIdx.x >> 5];
    if (C->status & kStFatal) return;
    const int nslices = (pp.n + kPpTargets - 1) / kPpTargets;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const unsigned lt_mask = (1u << lane) - 1u;
    unsigned long long pairs = 0, p2c = 0, tests = 0, targets = 0;  // per lane
    unsigned bad = 0;
    for (;;) {
        int si = 0;
        if (lane == 0) si = atomicAdd(&C->work_next, 1);
        si = __shfl_sync(0xffffffffu, si, 0);
        if (si >= nslices) break;
        const int own = si * kPpTargets, slot = own + lane;
        bool mine = lane < kPpTargets && slot < pp.n;
        float hdt_mine = wp.hdt;
        if (mine && pp.block) {
            const int rung = (int)P.vel[slot].w;
            mine = ((pp.sub + 1) % (1 << (pp.rmax - rung))) == 0;
            hdt_mine = (float)(0.5 * pp.base / (double)(1 << rung));
        }
        const unsigned active = __ballot_sync(0xffffffffu, mine);
        if (active == 0) continue;
        const int nt = __popc(active);
        if (pp.block && lane == 0) targets += (unsigned long long)nt;
        __syncwarp();
        int size;
        {
            // the members start at the roots of their systems, one stack entry
            // per root
            const int t = __popc(active & lt_mask);
            int root = -1;
            if (mine) {
                const float4 tp = P.pos[slot], ao = P.acc[slot];
                const float4 tl = SPLIT ? P.plo[slot] : zero;
                root = T.sysroot[leaf_list[pp.before[slot] + pp.starts[slot] - 1u]];
                const float aold = sqrtf(ao.x * ao.x + ao.y * ao.y + ao.z * ao.z);
                sm.hi[t] = make_float4(tp.x, tp.y, tp.z, pp.relative && aold > 0.f ? pp.alpha * aold : -1.f);
                sm.lo[t] = make_float4(tl.x, tl.y, tl.z, aold);
                sm.slot[t] = slot;
                sm.hdt[t] = hdt_mine;
            }
            const unsigned same = __match_any_sync(0xffffffffu, root);
            const bool lead = mine && (same & lt_mask) == 0u;
            const unsigned leads = __ballot_sync(0xffffffffu, lead);
            if (lead) {
                // the members of this root: bits t of the active lanes in `same`
                unsigned m = 0u;
                for (unsigned r = same; r; r &= r - 1u) m |= 1u << __popc(active & ((1u << (__ffs(r) - 1)) - 1u));
                sm.snode[__popc(leads & lt_mask)] = root;
                sm.smask[__popc(leads & lt_mask)] = (unsigned char)m;
            }
            size = __popc(leads);
        }
        __syncwarp();
        PpWalk<SPLIT, QUAD, SOFT> w{sm, T, P, wp, lane, nt, {}};
        int nfar = 0, nnear = 0, visits = 0;
        while (size > 0) {
            // at most eight children per node come back
            const int take = min(min(size, 32), max(1, (kPpStack - kPpReserve - size) / 7));
            size -= take;
            visits += take;
            if (visits > wp.node_limit) {
                bad |= kStCorrupt;
                break;
            }
            const int node = lane < take ? sm.snode[size + lane] : -1;
            unsigned m = lane < take ? sm.smask[size + lane] : 0u;
            __syncwarp();
            float4 A = zero, Cw = zero, D = zero;
            if (node >= 0) {
                A = T.wA[node];
                Cw = T.wC[node];
                D = T.wD[node];
            }
            if (!(A.w > 0.f)) m = 0u;
            const int meta = __float_as_int(Cw.w), link = __float_as_int(Cw.z);
            const bool reached = m != 0u && meta < 0;          // a leaf
            unsigned open = 0u, accepted = 0u;
            if (__any_sync(0xffffffffu, m != 0u && meta >= 0)) {
                const bool inner = m != 0u && meta >= 0;
                tests += inner ? (unsigned long long)__popc(m) : 0ull;
                const float size2 = Cw.y * Cw.y;
#pragma unroll
                for (int t = 0; t < kPpTargets; ++t) {
                    if (t >= nt || !inner || !((m >> t) & 1u)) continue;
                    const float4 h = sm.hi[t], l = sm.lo[t];
                    const float dx = (A.x - h.x) + (D.x - l.x);
                    const float dy = (A.y - h.y) + (D.y - l.y);
                    const float dz = (A.z - h.z) + (D.z - l.z);
                    const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                    const bool rel = h.w >= 0.f;
                    float lhs, rhs;
                    if (rel) {
                        lhs = A.w * Cw.y * Cw.y;
                        rhs = h.w * d2 * d2 / wp.G;
                    } else {
                        lhs = size2;
                        rhs = wp.theta2 * d2;
                    }
                    bool accept = lhs < rhs;
                    if (wp.retest && fabsf(lhs - rhs) <= 1e-5f * (lhs + rhs)) {
                        const double ex = T.comx[node] - ((double)h.x + l.x), ey = T.comy[node] - ((double)h.y + l.y),
                                     ez = T.comz[node] - ((double)h.z + l.z);
                        const double dd2 = ex * ex + ey * ey + ez * ez;
                        const double s2 = 4.0 * T.half[node] * T.half[node];
                        accept = rel ? T.mass[node] * s2 < pp.alpha_d * (double)l.w * dd2 * dd2 / (double)wp.G
                                     : s2 < wp.theta2_d * dd2;
                    }
                    if (accept)
                        accepted |= 1u << t;
                    else
                        open |= 1u << t;
                }
                p2c += (unsigned long long)__popc(accepted);
            }
            {  // opened children, with the members that opened their node
                const int nch = open ? meta & 0xFFFFFF : 0;
                int tot;
                const int off = warp_excl_scan(nch, lane, tot);
                for (int k = 0; k < nch; ++k) {
                    sm.snode[size + off + k] = link + k;
                    sm.smask[size + off + k] = (unsigned char)open;
                }
                size += tot;
            }
            {  // accepted nodes
                const unsigned has = __ballot_sync(0xffffffffu, accepted != 0u);
                if (accepted) {
                    const int i = nfar + __popc(has & lt_mask);
                    sm.fnode[i] = node;
                    sm.fmask[i] = (unsigned char)accepted;
                }
                nfar += __popc(has);
            }
            {  // reached leaves
                const unsigned has = __ballot_sync(0xffffffffu, reached);
                if (reached) {
                    const int i = nnear + __popc(has & lt_mask);
                    const int cnt = meta & 0xFFFFFF;
                    sm.nstart[i] = link;
                    sm.ncount[i] = cnt;
                    sm.nmask[i] = (unsigned char)m;
                    // members on the path, each with every particle of the leaf but itself
                    pairs += (unsigned long long)__popc(m) * (unsigned long long)cnt;
                    const int lo = max(link - own, 0), hi = min(link + cnt - own, kPpTargets);
                    if (lo < hi) {  // members in this leaf: bits of the active slots lo .. hi - 1
                        const unsigned upto_hi = hi >= 32 ? 0xffffffffu : (1u << hi) - 1u;
                        const int a = __popc(active & ((1u << lo) - 1u)), b = __popc(active & upto_hi);
                        pairs -= (unsigned long long)__popc(m & ((1u << b) - (1u << a)));
                    }
                }
                nnear += __popc(has);
            }
            __syncwarp();
            if (nfar >= 64) {
                w.far_window(64);
                pp_drop(sm.fnode, nfar, lane);
                pp_drop(sm.fmask, nfar, lane);
                nfar -= 64;
            }
            if (nnear >= 64) {
                w.near_batch(64, own, active);
                pp_drop(sm.nstart, nnear, lane);
                pp_drop(sm.ncount, nnear, lane);
                pp_drop(sm.nmask, nnear, lane);
                nnear -= 64;
            }
        }
        if (bad) break;
        if (nfar > 0) w.far_window(nfar);
        if (nnear > 0) w.near_batch(nnear, own, active);
        // totals across the lanes, error-free but for the sum of the errors
#pragma unroll
        for (int t = 0; t < kPpTargets; ++t) {
            if (t >= nt) break;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                PpSum other;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    other.s[k] = __shfl_xor_sync(0xffffffffu, w.sum[t].s[k], o);
                    other.low[k] = __shfl_xor_sync(0xffffffffu, w.sum[t].low[k], o);
                    w.sum[t].low[k] += other.low[k];
                }
                w.sum[t].add(other.s);
            }
            if (lane == t) {
                const int at = sm.slot[t];
                const float4 a = make_float4(wp.G * (w.sum[t].s[0] + w.sum[t].low[0]), wp.G * (w.sum[t].s[1] + w.sum[t].low[1]),
                                             wp.G * (w.sum[t].s[2] + w.sum[t].low[2]), 0.f);
                P.acc[at] = a;
                if (wp.kick) {
                    float4 v = P.vel[at];
                    float4 vl = SPLIT ? P.vlo[at] : zero;
                    kick_v(v, SPLIT ? &vl : nullptr, sm.hdt[t], a);
                    P.vel[at] = v;
                    if (SPLIT) P.vlo[at] = vl;
                }
            }
        }
        __syncwarp();
    }
    for (int o = 16; o > 0; o >>= 1) {
        bad |= __shfl_xor_sync(0xffffffffu, bad, o);
        pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
        p2c += __shfl_xor_sync(0xffffffffu, p2c, o);
        tests += __shfl_xor_sync(0xffffffffu, tests, o);
    }
    if (lane == 0) {
        if (bad) atomicOr(&C->status, bad);
        atomicAdd(&C->p2p_pairs, pairs);
        atomicAdd(&C->p2c_terms, p2c);
        atomicAdd(&C->mac_tests, tests);
        if (targets) atomicAdd(&C->targets, targets);
    }
}

#define NGRAV_PP_INSTANCES(X) \
    X(true, true, 0) X(true, true, 1) X(true, false, 0) X(true, false, 1) X(false, true, 0) X(false, true, 1) \
    X(false, false, 0) X(false, false, 1)

void walk_pp_set_attributes() {
#define NGRAV_PP_ATTR(SP, Q, SO)                                                                              \
    cudaFuncSetAttribute(walk_pp_kernel<SP, Q, (SO) ? kSoftSpline : kSoftPlummer>,                           \
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kPpWarps * sizeof(PpSmem)));
    NGRAV_PP_INSTANCES(NGRAV_PP_ATTR)
#undef NGRAV_PP_ATTR
}

void launch_walk_pp(const NodeArrays& T, Counters* C, const Particles& P, const int* leaf_list, const WalkParams& wp,
                    int relative, double alpha, const int* block, double block_base, long long n,
                    const unsigned* before, const unsigned* starts, int nwarps, cudaStream_t s) {
    PpParams pp;
    pp.n = (int)n;
    pp.before = before;
    pp.starts = starts;
    pp.relative = relative;
    pp.alpha = (float)alpha;
    pp.alpha_d = alpha;
    pp.block = block ? 1 : 0;
    pp.sub = block ? block[0] : 0;
    pp.rmax = block ? block[1] : 0;
    pp.base = block_base;
    const int blocks = (nwarps + kPpWarps - 1) / kPpWarps;
    const int soft = wp.soft == kSoftSpline ? 1 : 0;
#define NGRAV_PP_LAUNCH(SP, Q, SO)                                                                  \
    if (wp.split == (SP) && (wp.quadrupole != 0) == (Q) && soft == (SO))                          \
        walk_pp_kernel<SP, Q, (SO) ? kSoftSpline : kSoftPlummer><<<blocks, kPpThreads, kPpWarps * sizeof(PpSmem), s>>>( \
            T, C, P, leaf_list, wp, pp);
    NGRAV_PP_INSTANCES(NGRAV_PP_LAUNCH)
#undef NGRAV_PP_LAUNCH
}

}  // namespace ngrav
