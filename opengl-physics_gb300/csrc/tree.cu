// tree.cu -- linear octree from sorted keys, leaf list, upward moment pass.
//
// Topology rule (restating projects/nbody_core/src/Tree.cpp:114-145): a node
// at level l whose particle count exceeds the leaf capacity (ncrit) and whose
// level is below maxDepth is internal; its children are its non-empty
// octants.  The node set of the reference's insertion build is exactly this
// set, independent of insertion order, so it is read off the sorted keys, all
// levels at once.  Children of a node are contiguous in ascending octant order.
//
// Moments (restating Tree.cpp:119-122 running COM, :179-202 maxRadius,
// :205-254 quadrupoles): leaves sum their members (mass and COM in FP64,
// quadrupole in FP32 on offsets from the COM); internal nodes combine their
// children in FP64 (the top-level moment accumulation), level by level.
#include "engine.cuh"
#include "walk_common.cuh"

#include <algorithm>

namespace ngrav {

__global__ void reset_counters_kernel(Counters* C) {
    if (threadIdx.x == 0) {
        Counters z{};
        for (int a = 0; a < 3; ++a) {
            z.bbox_min[a] = ~0ull;
            z.bbox_max[a] = 0ull;
        }
        *C = z;
    }
}

// ---------------------------------------------------------------------------
// Topology
// ---------------------------------------------------------------------------
//
// Two neighbours in key order say where cells begin, and two particles
// leaf_cap apart whether a cell is too full, so every particle finds by itself
// which nodes begin at it, and the tree needs no descent level by level:
//   a cell of level l begins at particle i if keys i - 1 and i share fewer
//   than l digits; it holds more than leaf_cap particles if keys i and
//   i + leaf_cap share at least l;
//   of the cells that begin at i, c + 1 (one more digit than shared with
//   i - 1) is a node if its parent, which began earlier, splits; the next is
//   one if the cell above it splits, and so on: a run [first, top] of levels,
//   whose last is a leaf.
// Node numbers are by level and, in a level, in key order, which puts the
// children of a node side by side in ascending octant order.  A number is a
// count of runs that reach the level: tree_count counts them per segment of the
// particles (one warp each), tree_scan adds the segments up, tree_fill hands
// the numbers out, and tree_finish adds what a node can say for itself.
//
// Four launches instead of one per level and six for the leaf list; all of it is
// latency at small sizes and a read of the keys at large ones.  Before and now
// (levels and leaf list): 2,048 bodies 92 and 23 us, 1 Mi bodies 217 and 72 us,
// 4 Mi 293 and 144 us, 16.8 M 537 and 431 us.

constexpr int kRows = kMaxLevels + 1;       // counted per segment: nodes of each level, leaves
constexpr int kLeafRow = kMaxLevels;
constexpr int kSegMax = 152 * 48;           // as many warps as stay resident
constexpr unsigned short kNoRun = 0xFFFFu;  // a particle at which no node begins

static_assert(kRows <= 32, "a lane counts a row");

long long tree_counts_size() { return (long long)kRows * kSegMax + 32; }

// Digits that two keys share, at most `levels`.
__device__ __forceinline__ int shared_digits(unsigned long long a, unsigned long long b, int levels) {
    return min((__clzll((long long)(a ^ b)) - 1) / 3, levels);
}

__device__ __forceinline__ bool share(unsigned long long a, unsigned long long b, int digits) {
    return ((a ^ b) >> (3 * (kKeyLevels - digits))) == 0;
}

// Ensemble (sys_levels > 0): levels above sys_levels group systems by id
// digits, always split and carry no geometry; a node of level sys_levels is a
// system root.  max_depth counts from there (depth_cap from the top).
__global__ void __launch_bounds__(256, 6) tree_count_kernel(const unsigned long long* __restrict__ keys, long long n,
                                                           int leaf_cap, int depth_cap, int sys_levels, int levels,
                                                           int nseg, int seglen, unsigned short* __restrict__ runs,
                                                           int* __restrict__ counts, Counters* C) {
    const int lane = threadIdx.x & 31;
    const int seg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (seg >= nseg) return;
    const int deepest = min(depth_cap, levels);
    const long long lo = (long long)seg * seglen, hi = min(n, lo + seglen);
    int count = 0;  // of row `lane`
    for (long long base = lo; base < hi; base += 32) {
        const long long i = base + lane;
        const bool valid = i < hi;
        const unsigned long long key = valid ? keys[i] : 0ull;
        const unsigned long long prev = valid && i > 0 ? keys[i - 1] : 0ull;
        const bool has_on = valid && i + leaf_cap < n, has_back = valid && i >= leaf_cap;
        const unsigned long long on = has_on ? keys[i + leaf_cap] : 0ull;
        const unsigned long long back = has_back ? keys[i - leaf_cap] : 0ull;
        const int c = i > 0 ? shared_digits(prev, key, levels) : -1;
        const int full = has_on ? shared_digits(key, on, levels) : -1;  // cells from i on are too full down to here
        bool node = valid && c < deepest;
        if (node && c >= sys_levels && full < c && !(has_back && share(back, key, c))) {
            // the parent of the first cell: where it begins, and whether that
            // is leaf_cap before a particle that it still holds
            long long a = max(0ll, i - leaf_cap + 1), b = i;
            while (a < b) {
                const long long mid = (a + b) >> 1;
                if (share(keys[mid], key, c))
                    b = mid;
                else
                    a = mid + 1;
            }
            node = a + leaf_cap < n && share(keys[a + leaf_cap], key, c);
        }
        unsigned rows = 0;
        unsigned short run = kNoRun;
        if (node) {
            const int first = c + 1;
            int top = max(first, min(full + 1, deepest));
            if (first <= sys_levels) top = max(top, min(sys_levels, deepest));
            rows = ((2u << top) - (1u << first)) | (1u << kLeafRow);
            run = (unsigned short)(first << 8 | top);
            if (full >= top && top < depth_cap) {
                if (top >= kKeyLevels) {
                    atomicOr(&C->status, kStDepthLimit);
                    atomicAdd(&C->depth_limited, 1);
                } else if (top == levels) {
                    // the keys were sorted on `levels` digits only: this cell
                    // would split on an unsorted digit, so the build is redone
                    // on the full key
                    atomicOr(&C->status, kStSortDepth);
                }
            }
        }
        if (valid) runs[i] = run;
        for (unsigned any = __reduce_or_sync(0xffffffffu, rows); any; any &= any - 1) {
            const int l = __ffs((int)any) - 1;
            const int k = __popc(__ballot_sync(0xffffffffu, (rows >> l) & 1u));
            if (lane == l) count += k;
        }
    }
    if (lane < kRows) counts[lane * nseg + seg] = count;
}

// Row blockIdx.x of the counts: exclusive scan over the segments, in place, and
// the row's total.
__global__ void __launch_bounds__(1024) tree_scan_kernel(int* __restrict__ counts, int nseg, int* __restrict__ totals) {
    __shared__ int warp_sum[32];
    int* row = counts + (long long)blockIdx.x * nseg;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    constexpr int kPer = (kSegMax + 1023) / 1024;
    int v[kPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int at = threadIdx.x * kPer + k;
        v[k] = at < nseg ? row[at] : 0;
        sum += v[k];
    }
    int all;
    int before = warp_excl_scan(sum, lane, all);
    if (lane == 0) warp_sum[w] = all;
    __syncthreads();
    int total;
    const int base = warp_excl_scan(warp_sum[lane], lane, total);
    before += __shfl_sync(0xffffffffu, base, w);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int at = threadIdx.x * kPer + k;
        if (at < nseg) row[at] = before;
        before += v[k];
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = total;
}

// Numbers for the runs: per node its start, level, parent, first child and
// system root, the leaf list, and for a per-particle walk the leaves that begin
// before each particle (leaf_before) and at it (leaf_start).
__global__ void __launch_bounds__(256) tree_fill_kernel(NodeArrays T, Counters* C, long long n, int sys_levels,
                                                        int nseg, int seglen, const unsigned short* __restrict__ runs,
                                                        const int* __restrict__ counts,
                                                        const int* __restrict__ totals, int* __restrict__ leaf_list,
                                                        unsigned* __restrict__ leaf_before,
                                                        unsigned* __restrict__ leaf_start) {
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    const int seg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (seg >= nseg) return;
    const int in_row = lane < kRows ? totals[lane] : 0;
    int nodes;
    const int begin = warp_excl_scan(lane < kMaxLevels ? in_row : 0, lane, nodes);
    const bool fits = nodes <= T.cap;
    if (seg == 0) {
        // A tree too large for the pool is not written: no levels, no leaves;
        // the walk and the evaluation see the status, and the host grows the
        // pool and builds again.
        const unsigned used = __ballot_sync(0xffffffffu, lane < kMaxLevels && in_row > 0);
        if (lane < kMaxLevels + 2) C->level_begin[lane] = fits ? (lane < kMaxLevels ? begin : nodes) : 0;
        if (lane == 0) {
            C->next_free = nodes;
            C->levels_used = 31 - __clz((int)used);
            if (!fits) atomicOr(&C->status, kStNodeOverflow);
        }
        if (lane == kLeafRow) C->nleaves = fits ? in_row : 0;
    }
    if (!fits) return;
    // lane l: the number of the next node of level l (of the next leaf in the list)
    int next = lane < kRows ? (lane < kMaxLevels ? begin : 0) + counts[lane * nseg + seg] : 0;
    const long long lo = (long long)seg * seglen, hi = min(n, lo + seglen);
    for (long long base = lo; base < hi; base += 32) {
        const long long i = base + lane;
        const unsigned short run = i < hi ? runs[i] : kNoRun;
        const bool node = run != kNoRun;
        const int first = run >> 8, top = run & 0xFF;
        const unsigned rows = node ? (2u << top) - (1u << first) : 0u;
        const unsigned leaves = __ballot_sync(0xffffffffu, node);
        const unsigned at_sys = __ballot_sync(0xffffffffu, node && first <= sys_levels);
        const int sys_root = __shfl_sync(0xffffffffu, next, sys_levels) + __popc(at_sys & (lt_mask | 1u << lane)) - 1;
        const int leaf = __shfl_sync(0xffffffffu, next, kLeafRow) + __popc(leaves & lt_mask);
        if (leaf_before && i < hi) {
            leaf_before[i] = (unsigned)leaf;
            leaf_start[i] = node ? 1u : 0u;
        }
        int up = -1;         // this particle's node of the level above
        unsigned at_up = 0;  // the lanes with a node of that level
        int level_up = -1, begun = lane == kLeafRow ? __popc(leaves) : 0;
        for (unsigned any = __reduce_or_sync(0xffffffffu, rows); any; any &= any - 1) {
            const int l = __ffs((int)any) - 1;
            const unsigned at = __ballot_sync(0xffffffffu, (rows >> l) & 1u);
            const int next_up = __shfl_sync(0xffffffffu, next, l > 0 ? l - 1 : 0);
            const int num = __shfl_sync(0xffffffffu, next, l) + __popc(at & lt_mask);
            if ((rows >> l) & 1u) {
                // the parent of the first began earlier: the last of its level so far
                if (l == first) up = l > 0 ? next_up + __popc((level_up == l - 1 ? at_up : 0u) & lt_mask) - 1 : -1;
                T.start[num] = (int)i;
                T.level[num] = (unsigned char)l;
                T.parent[num] = up;
                if (l > first) T.first_child[up] = num;
                T.sysroot[num] = l < sys_levels ? num : sys_root;
                up = num;
            }
            if (lane == l) begun = __popc(at);
            at_up = at;
            level_up = l;
        }
        if (node) {
            T.first_child[up] = -1;
            leaf_list[leaf] = up;
        }
        next += begun;
    }
}

// What a node has by itself: its particle count (the end of its key range),
// child count, centre and size (the reference's recurrence from the root
// cube, rounded in FP64 as NewChild does).
__global__ void __launch_bounds__(256) tree_finish_kernel(NodeArrays T, Counters* C,
                                                         const unsigned long long* __restrict__ keys, long long n,
                                                         int leaf_cap, Forest F) {
    const int nodes = C->next_free;
    if (nodes > T.cap) return;
    int largest = 0;
    for (int node = blockIdx.x * blockDim.x + threadIdx.x; node < nodes; node += gridDim.x * blockDim.x) {
        const int s = T.start[node], l = T.level[node], fc = T.first_child[node];
        const unsigned long long key = keys[s];
        long long a = s, b = n;  // a within, b past the end
        if (l > 0) {
            for (long long step = leaf_cap; a + step < n; step *= 4) {
                if (!share(keys[a + step], key, l)) {
                    b = a + step;
                    break;
                }
                a += step;
            }
            while (b - a > 1) {
                const long long mid = (a + b) >> 1;
                if (share(keys[mid], key, l))
                    a = mid;
                else
                    b = mid;
            }
        }
        const int count = (int)(b - s);
        T.count[node] = count;
        int nch = 0;
        if (fc >= 0) {
#pragma unroll
            for (int k = 0; k < 8; ++k) nch += fc + k < nodes && T.parent[fc + k] == node ? 1 : 0;
        } else {
            largest = max(largest, count);
        }
        T.nchild[node] = (unsigned char)nch;
        double cx = 0.0, cy = 0.0, cz = 0.0, half = 0.0;
        if (l >= F.sys_levels) {
            if (F.sys_levels > 0) {
                const int sys = (int)(key >> (3 * (kKeyLevels - F.sys_levels)));
                cx = F.root[4 * sys];
                cy = F.root[4 * sys + 1];
                cz = F.root[4 * sys + 2];
                half = F.root[4 * sys + 3];
            } else {
                cx = C->root_center[0];
                cy = C->root_center[1];
                cz = C->root_center[2];
                half = C->root_half;
            }
            for (int k = F.sys_levels; k < l; ++k) {
                const unsigned d = (unsigned)(key >> (3 * (kKeyLevels - 1 - k))) & 7u;
                half *= 0.5;
                cx = __dadd_rn(cx, d & 1 ? half : -half);
                cy = __dadd_rn(cy, d & 2 ? half : -half);
                cz = __dadd_rn(cz, d & 4 ? half : -half);
            }
        }
        T.cx[node] = cx;
        T.cy[node] = cy;
        T.cz[node] = cz;
        T.half[node] = half;
    }
    __shared__ int s_largest;
    if (threadIdx.x == 0) s_largest = 0;
    __syncthreads();
    largest = __reduce_max_sync(0xffffffffu, largest);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_largest, largest);
    __syncthreads();
    if (threadIdx.x == 0 && s_largest > 0) atomicMax(&C->max_leaf_count, s_largest);
}

int launch_tree(NodeArrays& T, Counters* C, const unsigned long long* keys, long long n, int leaf_cap, int max_depth,
                const Forest& F, int levels, const TreeBuffers& B, bool leaf_scan, cudaStream_t s) {
    const int seglen = 32 * (int)((n + 32ll * kSegMax - 1) / (32ll * kSegMax));
    const int nseg = (int)((n + seglen - 1) / seglen);
    const unsigned g = (unsigned)((nseg + 7) / 8);
    int* totals = B.counts + (long long)kRows * kSegMax;
    const int depth_cap = max_depth < kMaxLevels ? max_depth + F.sys_levels : kMaxLevels + F.sys_levels;
    tree_count_kernel<<<g, 256, 0, s>>>(keys, n, leaf_cap, depth_cap, F.sys_levels, levels, nseg, seglen, B.runs,
                                        B.counts, C);
    tree_scan_kernel<<<kRows, 1024, 0, s>>>(B.counts, nseg, totals);
    tree_fill_kernel<<<g, 256, 0, s>>>(T, C, n, F.sys_levels, nseg, seglen, B.runs, B.counts, totals, B.leaf_list,
                                       leaf_scan ? B.leaf_before : nullptr, leaf_scan ? B.leaf_start : nullptr);
    long long blocks = ((long long)std::min<long long>(T.cap, 2 * n) + 255) / 256;
    if (blocks > 152 * 8) blocks = 152 * 8;
    tree_finish_kernel<<<(unsigned)blocks, 256, 0, s>>>(T, C, keys, n, leaf_cap, F);
    return 4;
}

// ---------------------------------------------------------------------------
// Upward pass
// ---------------------------------------------------------------------------

__device__ __forceinline__ float round_up_f(double v) {
    float f = (float)v;
    if ((double)f < v) f = nextafterf(f, 3.0e38f);
    return f;
}

__device__ __forceinline__ void write_walk_record(NodeArrays& T, int node, double M, double cx, double cy,
                                                  double cz, const double* Q, double maxr, bool leaf, int link,
                                                  int cnt_or_nch, int level) {
    const float hx = (float)cx, hy = (float)cy, hz = (float)cz;
    T.wA[node] = make_float4(hx, hy, hz, (float)M);
    T.wB[node] = make_float4((float)Q[0], (float)Q[1], (float)Q[2], (float)Q[3]);
    const double size = 2.0 * T.half[node];
    T.wC[node] = make_float4(round_up_f(maxr), (float)size, __int_as_float(link),
                             __int_as_float(meta_pack(leaf, cnt_or_nch, level)));
    T.wD[node] = make_float4((float)(cx - (double)hx), (float)(cy - (double)hy), (float)(cz - (double)hz),
                             (float)Q[4]);
}

// Leaf moments, plus the group acceleration scale amin[leaf] = min over the
// members of |a| from `acc` (the accelerations carried into this tree order;
// zero before the first evaluation) that the learned opening test reads.
//
// GB300's FP64 pipe runs at 1/64 of the FP32 rate, so the per-particle work
// is FP32: each member's offset from the leaf centre is a double-float pair
// (error-free differences of the double-float position and centre), mass
// and first moment are summed as double-float pairs with exact products,
// and only the per-leaf results are FP64.  maxRadius keeps the reference's
// FP64 value: the members within FP32 rounding of the FP32 maximum distance
// are re-measured in FP64 (Tree.cpp:188-201).
//
// A warp takes `lpw` (4 to 32) consecutive leaves, and the FP64 steps run with a
// lane per leaf, as one FP64 instruction occupies the pipe for 16 cycles however
// few of its lanes are wanted.  Only the farthest member is re-measured, unless
// a runner-up is within rounding of it: a re-measurement inside the member loop
// stopped a warp in almost every iteration for one leaf or another.  Members are
// read S lanes to a leaf: eight while there are few leaves, where the latency
// of a leaf counts, one where there are many, which spares the reductions.
// Before and now: 297 k leaves (4 Mi bodies) 278 and 156 us, 462 leaves (2,048
// bodies) 27 and 13 us; eight lanes throughout took 185 us at 297 k leaves.

// (ah, al) += (bh, bl)
__device__ __forceinline__ void df_add(float& ah, float& al, float bh, float bl) {
    float t, e;
    two_sum(ah, bh, t, e);
    fast_two_sum(t, __fadd_rn(al, __fadd_rn(bl, e)), ah, al);
}

__device__ __forceinline__ void df_add_xor(float& h, float& l, int o) {
    const float oh = __shfl_xor_sync(0xffffffffu, h, o), ol = __shfl_xor_sync(0xffffffffu, l, o);
    df_add(h, l, oh, ol);
}

// v of the leaf's lane, for the S lanes that work on leaf 32 / S * r + lane / S
// (and back: the value that those lanes hold, kept by the leaf's lane).
template <int S, typename V>
__device__ __forceinline__ V to_members(V v, int r, int lane) {
    return S == 1 ? v : __shfl_sync(0xffffffffu, v, 32 / S * r + lane / S);
}

template <int S, typename V>
__device__ __forceinline__ void to_leaf(V& keep, V v, int r, int lane) {
    if (S == 1) {
        keep = v;
    } else {
        const V x = __shfl_sync(0xffffffffu, v, lane % (32 / S) * S);
        if (lane / (32 / S) == r) keep = x;
    }
}

constexpr int kMomFew = 16384, kMomWarps = 4;

template <int S>
__device__ __forceinline__ void leaf_moments(NodeArrays& T, Counters* C, const float4* __restrict__ pos,
                                             const float4* __restrict__ plo, float4* __restrict__ src,
                                             const float4* __restrict__ acc, const int* __restrict__ leaf_list,
                                             int2* __restrict__ passes, int split, int quadrupole, int nleaves,
                                             int lpw) {
    const int pass = pass_targets(nleaves);
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const int lane = threadIdx.x & 31, sub = lane % S;
    const int nwarps = gridDim.x * kMomWarps;
    for (long long first = (long long)(blockIdx.x * kMomWarps + (threadIdx.x >> 5)) * lpw; first < nleaves;
         first += (long long)nwarps * lpw) {
        // lane = leaf: the leaf's range and centre
        const int li = (int)first + lane;
        const bool has = lane < lpw && li < nleaves;
        const int leaf = has ? leaf_list[li] : 0;
        const int s = has ? T.start[leaf] : 0, cnt = has ? T.count[leaf] : 0;
        const int more = cnt > pass ? (cnt - 1) / pass : 0;
        int all_more;
        const int before = warp_excl_scan(more, lane, all_more);
        if (all_more > 0) {  // one atomic for the warp's leaves
            int at = 0;
            if (lane == 0) at = atomicAdd(&C->extra_passes, all_more);
            at = __shfl_sync(0xffffffffu, at, 0) + before;
            for (int p = 0; p < more; ++p) passes[at + p] = make_int2(li, p + 1);
        }
        const double ccx = has ? T.cx[leaf] : 0.0, ccy = has ? T.cy[leaf] : 0.0, ccz = has ? T.cz[leaf] : 0.0;
        const float half = has ? (float)T.half[leaf] : 0.f;
        const float chx = (float)ccx, chy = (float)ccy, chz = (float)ccz;
        const float clx = (float)(ccx - (double)chx), cly = (float)(ccy - (double)chy),
                    clz = (float)(ccz - (double)chz);
        // pass 1: mass and first moment about the leaf centre
        float Mh = 0.f, Ml = 0.f, Xh = 0.f, Xl = 0.f, Yh = 0.f, Yl = 0.f, Zh = 0.f, Zl = 0.f;
        for (int r = 0; 32 / S * r < lpw; ++r) {
            const int ms = to_members<S>(s, r, lane), mc = to_members<S>(cnt, r, lane);
            const float hx = to_members<S>(chx, r, lane), hy = to_members<S>(chy, r, lane),
                        hz = to_members<S>(chz, r, lane);
            const float lx = to_members<S>(clx, r, lane), ly = to_members<S>(cly, r, lane),
                        lz = to_members<S>(clz, r, lane);
            float mh = 0.f, ml = 0.f, xh = 0.f, xl = 0.f, yh = 0.f, yl = 0.f, zh = 0.f, zl = 0.f;
#pragma unroll 2
            for (int j = sub; j < mc; j += S) {
                const float4 p = pos[ms + j];
                const float4 q = plo ? plo[ms + j] : zero4;
                float ox, oxl, oy, oyl, oz, ozl;
                df_offset(p.x, q.x, hx, lx, ox, oxl);
                df_offset(p.y, q.y, hy, ly, oy, oyl);
                df_offset(p.z, q.z, hz, lz, oz, ozl);
                df_add(mh, ml, p.w, 0.f);
                df_add_prod(xh, xl, p.w, ox, oxl);
                df_add_prod(yh, yl, p.w, oy, oyl);
                df_add_prod(zh, zl, p.w, oz, ozl);
            }
            __syncwarp();
#pragma unroll
            for (int o = S / 2; o > 0; o >>= 1) {
                df_add_xor(mh, ml, o);
                df_add_xor(xh, xl, o);
                df_add_xor(yh, yl, o);
                df_add_xor(zh, zl, o);
            }
            to_leaf<S>(Mh, mh, r, lane);
            to_leaf<S>(Ml, ml, r, lane);
            to_leaf<S>(Xh, xh, r, lane);
            to_leaf<S>(Xl, xl, r, lane);
            to_leaf<S>(Yh, yh, r, lane);
            to_leaf<S>(Yl, yl, r, lane);
            to_leaf<S>(Zh, zh, r, lane);
            to_leaf<S>(Zl, zl, r, lane);
        }
        const double M = (double)Mh + (double)Ml;
        double ocx = 0.0, ocy = 0.0, ocz = 0.0;  // COM - centre
        if (M > 0.0) {
            const double inv = 1.0 / M;
            ocx = ((double)Xh + (double)Xl) * inv;
            ocy = ((double)Yh + (double)Yl) * inv;
            ocz = ((double)Zh + (double)Zl) * inv;
        }
        const double cx = ccx + ocx, cy = ccy + ocy, cz = ccz + ocz;
        const float ohx = (float)ocx, ohy = (float)ocy, ohz = (float)ocz;
        const float olx = (float)(ocx - (double)ohx), oly = (float)(ocy - (double)ohy),
                    olz = (float)(ocz - (double)ohz);
        // pass 2: FP32 distances from the COM, quadrupole, amin, walk sources,
        // the farthest member and the runner-up's distance
        float Q0 = 0.f, Q1 = 0.f, Q2 = 0.f, Q3 = 0.f, Q4 = 0.f, A2 = 0.f, Cut = 0.f;
        int Far = -1;
        bool several = false;
        for (int r = 0; 32 / S * r < lpw; ++r) {
            const int ms = to_members<S>(s, r, lane), mc = to_members<S>(cnt, r, lane);
            const float hx = to_members<S>(chx, r, lane), hy = to_members<S>(chy, r, lane),
                        hz = to_members<S>(chz, r, lane);
            const float lx = to_members<S>(clx, r, lane), ly = to_members<S>(cly, r, lane),
                        lz = to_members<S>(clz, r, lane);
            const float ux = to_members<S>(ohx, r, lane), uy = to_members<S>(ohy, r, lane),
                        uz = to_members<S>(ohz, r, lane);
            const float vx = to_members<S>(olx, r, lane), vy = to_members<S>(oly, r, lane),
                        vz = to_members<S>(olz, r, lane);
            float maxf = -1.f, second = -1.f, amin2 = 3.0e38f;
            int at = -1;
            float q0 = 0.f, q1 = 0.f, q2 = 0.f, q3 = 0.f, q4 = 0.f;
#pragma unroll 2
            for (int j = sub; j < mc; j += S) {
                const float4 p = pos[ms + j];
                const float4 a = acc[ms + j];
                const float4 l = plo ? plo[ms + j] : zero4;
                amin2 = fminf(amin2, a.x * a.x + a.y * a.y + a.z * a.z);
                float ox, oxl, oy, oyl, oz, ozl;
                df_offset(p.x, l.x, hx, lx, ox, oxl);
                df_offset(p.y, l.y, hy, ly, oy, oyl);
                df_offset(p.z, l.z, hz, lz, oz, ozl);
                const float fx = (ox - ux) + (oxl - vx), fy = (oy - uy) + (oyl - vy), fz = (oz - uz) + (ozl - vz);
                const float d2 = fmaf(fx, fx, fmaf(fy, fy, fz * fz));
                second = fmaxf(second, fminf(maxf, d2));
                at = d2 > maxf ? j : at;
                maxf = fmaxf(maxf, d2);
                if (quadrupole && mc > 1) {
                    const float m = p.w;
                    q0 += m * (3.f * fx * fx - d2);
                    q1 += m * (3.f * fy * fy - d2);
                    q2 += m * 3.f * fx * fy;
                    q3 += m * 3.f * fx * fz;
                    q4 += m * 3.f * fy * fz;
                }
                src[ms + j] = split ? make_float4(ox + oxl, oy + oyl, oz + ozl, p.w) : p;
            }
            __syncwarp();
#pragma unroll
            for (int o = S / 2; o > 0; o >>= 1) {
                q0 += __shfl_xor_sync(0xffffffffu, q0, o);
                q1 += __shfl_xor_sync(0xffffffffu, q1, o);
                q2 += __shfl_xor_sync(0xffffffffu, q2, o);
                q3 += __shfl_xor_sync(0xffffffffu, q3, o);
                q4 += __shfl_xor_sync(0xffffffffu, q4, o);
                amin2 = fminf(amin2, __shfl_xor_sync(0xffffffffu, amin2, o));
                const float m2 = __shfl_xor_sync(0xffffffffu, maxf, o), s2 = __shfl_xor_sync(0xffffffffu, second, o);
                const int at2 = __shfl_xor_sync(0xffffffffu, at, o);
                second = fmaxf(fmaxf(second, s2), fminf(maxf, m2));
                at = m2 > maxf || (m2 == maxf && at2 > at) ? at2 : at;
                maxf = fmaxf(maxf, m2);
            }
            const float rcut = sqrtf(fmaxf(maxf, 0.f)) * (1.f - 4e-6f) - 2e-6f * to_members<S>(half, r, lane);
            const float cut = rcut > 0.f ? rcut * rcut : -0.5f;
            several |= second >= cut;
            to_leaf<S>(Q0, q0, r, lane);
            to_leaf<S>(Q1, q1, r, lane);
            to_leaf<S>(Q2, q2, r, lane);
            to_leaf<S>(Q3, q3, r, lane);
            to_leaf<S>(Q4, q4, r, lane);
            to_leaf<S>(A2, amin2, r, lane);
            to_leaf<S>(Cut, cut, r, lane);
            to_leaf<S>(Far, at, r, lane);
        }
        // pass 3: the FP64 maximum over the members that can hold it.  An FP32
        // distance is within a few ulps of the leaf's half size of the FP64
        // one, so no member farther than the cut can be missed.  That is the
        // farthest alone, unless a leaf of this warp has a runner-up past the
        // cut: then all members are tested again, and the ones past it go to
        // the leaf's lane as a mask per 64.
        double maxr2 = 0.0;
        auto measure = [&](int j) {
            const float4 p = pos[j];
            const float4 l = plo ? plo[j] : zero4;
            const double x = (double)p.x + (double)l.x, y = (double)p.y + (double)l.y, z = (double)p.z + (double)l.z;
            const double dx = x - cx, dy = y - cy, dz = z - cz;
            maxr2 = fmax(maxr2, dx * dx + dy * dy + dz * dz);
        };
        if (!__any_sync(0xffffffffu, several)) {
            if (has && Far >= 0) measure(s + Far);
        } else {
            int most = cnt;
            for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
            for (int m0 = 0; m0 < most; m0 += 64) {
                unsigned long long cand = 0;
                for (int r = 0; 32 / S * r < lpw; ++r) {
                    const int ms = to_members<S>(s, r, lane), mc = min(to_members<S>(cnt, r, lane), m0 + 64);
                    const float hx = to_members<S>(chx, r, lane), hy = to_members<S>(chy, r, lane),
                                hz = to_members<S>(chz, r, lane);
                    const float lx = to_members<S>(clx, r, lane), ly = to_members<S>(cly, r, lane),
                                lz = to_members<S>(clz, r, lane);
                    const float ux = to_members<S>(ohx, r, lane), uy = to_members<S>(ohy, r, lane),
                                uz = to_members<S>(ohz, r, lane);
                    const float vx = to_members<S>(olx, r, lane), vy = to_members<S>(oly, r, lane),
                                vz = to_members<S>(olz, r, lane);
                    const float cut = to_members<S>(Cut, r, lane);
                    unsigned long long mine = 0;  // of this lane's members
                    for (int j = m0 + sub; j < mc; j += S) {
                        const float4 p = pos[ms + j];
                        const float4 l = plo ? plo[ms + j] : zero4;
                        float ox, oxl, oy, oyl, oz, ozl;
                        df_offset(p.x, l.x, hx, lx, ox, oxl);
                        df_offset(p.y, l.y, hy, ly, oy, oyl);
                        df_offset(p.z, l.z, hz, lz, oz, ozl);
                        const float fx = (ox - ux) + (oxl - vx), fy = (oy - uy) + (oyl - vy),
                                    fz = (oz - uz) + (ozl - vz);
                        if (fmaf(fx, fx, fmaf(fy, fy, fz * fz)) >= cut) mine |= 1ull << (j - m0);
                    }
                    __syncwarp();
#pragma unroll
                    for (int o = S / 2; o > 0; o >>= 1) mine |= __shfl_xor_sync(0xffffffffu, mine, o);
                    to_leaf<S>(cand, mine, r, lane);
                }
                while (cand) {
                    measure(s + m0 + __ffsll((long long)cand) - 1);
                    cand &= cand - 1;
                }
                __syncwarp();
            }
        }
        if (has) {
            const double maxr = sqrt(maxr2);
            const double Q[5] = {Q0, Q1, Q2, Q3, Q4};
            T.mass[leaf] = M;
            T.comx[leaf] = cx;
            T.comy[leaf] = cy;
            T.comz[leaf] = cz;
            T.maxr[leaf] = maxr;
            T.amin[leaf] = cnt > 0 ? sqrtf(A2) : 0.f;
            for (int k = 0; k < 5; ++k) T.quad[5 * leaf + k] = Q[k];
            const int level = T.level[leaf];
            write_walk_record(T, leaf, M, cx, cy, cz, Q, maxr, true, s, cnt, level);
            T.chi[leaf] = make_float4(chx, chy, chz, __int_as_float(s));
            T.clo[leaf] = make_float4(clx, cly, clz, __int_as_float(cnt));
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(32 * kMomWarps, 6)
    moments_kernel(NodeArrays T, Counters* C, const float4* __restrict__ pos, const float4* __restrict__ plo,
                   float4* __restrict__ src, const float4* __restrict__ acc, const int* __restrict__ leaf_list,
                   int2* __restrict__ passes, int split, int quadrupole) {
    const int nleaves = C->nleaves;
    if (nleaves <= kMomFew) {
        // as few leaves per warp as four while an SM has few warps
        const int lpw = nleaves <= 4 * 152 * kMomWarps ? 4 : nleaves <= 8 * 152 * kMomWarps ? 8 : 16;
        leaf_moments<8>(T, C, pos, plo, src, acc, leaf_list, passes, split, quadrupole, nleaves, lpw);
    } else {
        leaf_moments<1>(T, C, pos, plo, src, acc, leaf_list, passes, split, quadrupole, nleaves, 32);
    }
}

// Internal nodes of one level, from their (finished) children: mass and COM
// (sum m x / M) in FP64 in child order, as the reference's sequential sums;
// the traceless quadrupole by the parallel-axis shift (Tree.cpp:235-251) and
// maxRadius = max over children of maxR_c + |com_c - com| (Tree.cpp:194-201;
// massless nodes keep 0).  GB300's FP64 pipe is narrow, so the per-child
// work runs on the FP32 pipe from the children's walk records: offsets from
// the double-float parent COM, the quadrupole shift summed in FP32 (the walk
// evaluates quadrupoles in FP32), and maxRadius screened in FP32 with only
// the children within rounding of the FP32 maximum re-measured in FP64.  The
// geometric opening test reads maxRadius of leaves only; the learned one
// reads it for every node.
//
// The re-measured children wait in a mask, so that a warp runs the FP64 square
// root once or twice and not once for each of the eight places (4 Mi bodies, 16
// levels: 280 and 166 us).
//
// A level of the upward pass is a chain of latencies, so the records that the
// FP32 part wants later are asked for with the first loads (all moments at 2,048
// bodies 63 -> 59 us, at 20,011 90 -> 86, with what top_moments_kernel loads early).
__device__ __forceinline__ void ask_for(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

__device__ __forceinline__ void internal_moments(NodeArrays& T, int node, int fc, int nch, int l, int quadrupole) {
    ask_for(T.wA + fc);
    ask_for(T.wA + fc + nch - 1);
    ask_for(T.wD + fc);
    ask_for(T.wD + fc + nch - 1);
    ask_for(T.wC + fc);
    ask_for(T.wC + fc + nch - 1);
    ask_for(T.wB + fc);
    ask_for(T.wB + fc + nch - 1);
    ask_for(T.maxr + fc);
    ask_for(T.maxr + fc + nch - 1);
    // the (at most eight) children unrolled: their loads and the FP64
    // chains of the combination overlap instead of running one child
    // after another
    double mc[8], cxs[8], cys[8], czs[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const bool in = k < nch;
        mc[k] = in ? T.mass[fc + k] : 0.0;
        cxs[k] = in ? T.comx[fc + k] : 0.0;
        cys[k] = in ? T.comy[fc + k] : 0.0;
        czs[k] = in ? T.comz[fc + k] : 0.0;
    }
    double PM = 0.0, px = 0.0, py = 0.0, pz = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {  // in child order, as the sequential sum
        PM += mc[k];
        px = fma(mc[k], cxs[k], px);
        py = fma(mc[k], cys[k], py);
        pz = fma(mc[k], czs[k], pz);
    }
    double pcx = T.cx[node], pcy = T.cy[node], pcz = T.cz[node];
    if (PM > 0.0) {
        const double inv = 1.0 / PM;
        pcx = px * inv;
        pcy = py * inv;
        pcz = pz * inv;
    }
    const float phx = (float)pcx, phy = (float)pcy, phz = (float)pcz;
    const float plx = (float)(pcx - (double)phx), ply = (float)(pcy - (double)phy),
                plz = (float)(pcz - (double)phz);
    float q0 = 0.f, q1 = 0.f, q2 = 0.f, q3 = 0.f, q4 = 0.f;
    float cand[8];
    float best = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        cand[k] = -1.f;
        if (k >= nch) continue;
        const int c = fc + k;
        const float4 A = T.wA[c], D = T.wD[c];
        const float dx = (A.x - phx) + (D.x - plx), dy = (A.y - phy) + (D.y - ply),
                    dz = (A.z - phz) + (D.z - plz);
        const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        if (quadrupole && mc[k] > 0.0) {
            const float4 B = T.wB[c];
            const float m = A.w;
            q0 += B.x + m * (3.f * dx * dx - d2);
            q1 += B.y + m * (3.f * dy * dy - d2);
            q2 += B.z + m * 3.f * dx * dy;
            q3 += B.w + m * 3.f * dx * dz;
            q4 += D.w + m * 3.f * dy * dz;
        }
        cand[k] = T.wC[c].x + sqrtf(d2);  // >= maxR_c (rounded up) + |d| within FP32 rounding
        best = fmaxf(best, cand[k]);
    }
    double mr = 0.0;
    unsigned past = 0;
    if (PM > 0.0) {
        const float cut = best * (1.f - 1e-5f) - 1e-30f;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (k < nch && !(cand[k] < cut)) past |= 1u << k;
    }
    while (past) {
        const int c = fc + __ffs((int)past) - 1;
        past &= past - 1;
        const double dx = T.comx[c] - pcx, dy = T.comy[c] - pcy, dz = T.comz[c] - pcz;
        mr = fmax(mr, T.maxr[c] + sqrt(dx * dx + dy * dy + dz * dz));
    }
    const double PQ[5] = {q0, q1, q2, q3, q4};
    T.mass[node] = PM;
    T.comx[node] = pcx;
    T.comy[node] = pcy;
    T.comz[node] = pcz;
    T.maxr[node] = mr;
    for (int k = 0; k < 5; ++k) T.quad[5 * node + k] = PQ[k];
    write_walk_record(T, node, PM, pcx, pcy, pcz, PQ, mr, false, fc, nch, l);
}

constexpr int kIntThreads = 64;

__global__ void __launch_bounds__(kIntThreads) internal_moments_kernel(NodeArrays T, const Counters* __restrict__ C,
                                                                      int l, int quadrupole) {
    const int end = C->level_begin[l + 1];
    for (int node = C->level_begin[l] + blockIdx.x * blockDim.x + threadIdx.x; node < end;
         node += gridDim.x * blockDim.x) {
        const int fc = T.first_child[node];
        if (fc >= 0) internal_moments(T, node, fc, T.nchild[node], l, quadrupole);
    }
}

// Levels `levels` - 1 down to 0 in one launch: one cluster, its barrier between
// two levels (arrive.release / wait.acquire at cluster scope orders the
// records that its CTAs exchange through global memory).  What does not depend
// on the level below, a thread's node and its children's places, is loaded
// before the barrier.
constexpr int kTopCtas = 8, kTopThreads = 256;

__global__ void __cluster_dims__(kTopCtas, 1, 1) __launch_bounds__(kTopThreads)
    top_moments_kernel(NodeArrays T, const Counters* __restrict__ C, int levels, int quadrupole) {
    __shared__ int begin[kMaxLevels + 2];
    if (threadIdx.x < kMaxLevels + 2) begin[threadIdx.x] = C->level_begin[threadIdx.x];
    __syncthreads();
    // neighbouring nodes go to different SMs by whole warps
    const int tid = ((threadIdx.x >> 5) * kTopCtas + blockIdx.x) * 32 + (threadIdx.x & 31);
    int fc = -1, nch = 0;
    auto look = [&](int l, int node) {
        fc = node < begin[l + 1] ? T.first_child[node] : -1;
        nch = node < begin[l + 1] ? T.nchild[node] : 0;
    };
    look(levels - 1, begin[levels - 1] + tid);
    for (int l = levels - 1; l >= 0; --l) {
        for (int node = begin[l] + tid; node < begin[l + 1]; node += kTopCtas * kTopThreads) {
            if (fc >= 0) internal_moments(T, node, fc, nch, l, quadrupole);
            look(l, node + kTopCtas * kTopThreads);
        }
        if (l > 0) look(l - 1, begin[l - 1] + tid);
        __syncwarp();  // the loop's lanes leave it apart, and the barrier is .aligned
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// The top levels, of at most 8^3 nodes each, go to the cluster, and so do all
// levels of a tree of few nodes: a level is a chain of latencies, some 6 us in the
// cluster (2,048 bodies, 9 levels: 56 us) and 10 in a launch of its own (89 us), but
// a cluster has 8 of the 152 SMs' FP64 pipes.  All of the moments with every level
// in the cluster, and with the top four: 63 and 78 us at 2,048 bodies, 86 and 107
// at 20,011 (leaves of 8), 143 and 131 at 131,071 (leaves of 16).
constexpr int kTopLevels = 4;
constexpr long long kTopTree = 4096;  // bodies per leaf_capacity of a tree of few nodes

int launch_moments(NodeArrays& T, Counters* C, const Particles& P, const int* leaf_list, const ListBuffers& LB,
                    long long n, int max_leaves, int leaf_cap, bool split, bool quadrupole, int levels,
                    cudaStream_t s) {
    long long blocks = ((long long)max_leaves + 4 * kMomWarps - 1) / (4 * kMomWarps);
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (blocks < 1) blocks = 1;
    moments_kernel<<<(unsigned)blocks, 32 * kMomWarps, 0, s>>>(T, C, P.pos, split ? P.plo : nullptr, P.src, P.acc,
                                                               leaf_list, LB.passes, split ? 1 : 0, quadrupole ? 1 : 0);
    const int top = n <= kTopTree * leaf_cap ? levels : std::min(levels, kTopLevels);
    long long b2 = ((long long)T.cap / 4 + kIntThreads - 1) / kIntThreads;
    if (b2 > 152 * 8) b2 = 152 * 8;
    if (b2 < 1) b2 = 1;
    for (int l = levels - 1; l >= top; --l)
        internal_moments_kernel<<<(unsigned)b2, kIntThreads, 0, s>>>(T, C, l, quadrupole ? 1 : 0);
    top_moments_kernel<<<kTopCtas, kTopThreads, 0, s>>>(T, C, top, quadrupole ? 1 : 0);
    return 2 + levels - top;
}

void launch_reset_counters(Counters* C, cudaStream_t s) { reset_counters_kernel<<<1, 32, 0, s>>>(C); }

}  // namespace ngrav
