// walk.cu -- the grouped Barnes-Hut walk: a traversal kernel that applies the
// reference's opening test per leaf group and writes each group's far and
// near interaction lists.
//
// Semantics restate the reference's grouped walk
// (projects/nbody_core/src/Solvers.cpp:248-355):
//  * each leaf is a target group; the group sphere is the leaf COM with
//    radius maxRadius;
//  * an internal node is accepted (far, P2C) iff
//      worst = |com_node - com_group| - maxRadius_group > 0  and
//      (2 half)^2 < theta^2 worst^2                       (:261-271)
//    otherwise its children are visited;
//  * every leaf reached is near (exact P2P), however far away (:256-258);
//  * the group's own members interact exactly, self excluded (:340-348);
//  * nodes with mass <= 0 are skipped (:254).
// P2P: a += G m d / (|d|^2 + eps^2)^(3/2)  (AccumPairPlummer, :19-38).
// P2C: softened monopole plus the unsoftened traceless quadrupole
//      a += -G Q.d / r^5 + 2.5 G (d.Q.d) d / r^7  (AddQuadrupole, :147-179).
//
// Walk: one warp per group, groups taken dynamically in key order.  Each
// iteration takes up to 4 kNPL opened nodes off a per-warp stack and tests
// their children (lane = child, kNPL per lane); near leaves and far nodes are
// appended (ballot + prefix) to the group's lists with coalesced stores, opened
// nodes are pushed.  The
// opening test runs in FP32 on double-float COMs; decisions within a
// relative band of 1e-5 of the threshold are re-taken in FP64 on the FP64
// moments.  Lists are chains of 128-entry chunks taken from a pool with one
// atomic per chunk, so every entry is written once.
//
// The evaluation of the lists lives in eval.cu.
#include "engine.cuh"
#include "walk_common.cuh"

namespace ngrav {

// ---------------------------------------------------------------------------
// Walk
// ---------------------------------------------------------------------------

constexpr int kWalkWarps = 4;
constexpr int kWalkThreads = kWalkWarps * 32;
// Nodes tested per lane per iteration, their loads in flight together.  The
// walk is bound by instruction issue and by the latency of one iteration (the
// records come from the L2), so an iteration's cost is what counts: with a
// stack of opened nodes instead of one of nodes to test, a push is one store per
// opened node without a prefix sum, and siblings are read as whole lines.  1 Mi
// bodies (theta 0.5, plain): 3.50 ms with nodes on the stack, 2.86 ms so; 4 Mi
// (theta 1): 3.72 and 2.86 ms.  One, three and four per lane were all slower.
constexpr int kNPL = 2;

// STACK > 0: a per-warp traversal stack for a frontier of STACK nodes in shared
// memory (STACK / 4 opened nodes; push -> pop never leaves the SM, the size
// trades L1 and occupancy against the frontier it holds, a tuned choice);
// STACK = 0: the global-memory stack, the fallback for trees whose frontier
// outgrows shared memory.
template <int STACK>
__global__ void __launch_bounds__(kWalkThreads) walk_kernel(NodeArrays T, Counters* C,
                                                            const int* __restrict__ leaf_list, WalkParams wp,
                                                            ListBuffers LB) {
    __shared__ int2 s_stack[STACK > 0 ? kWalkWarps * STACK / 4 : 1];
    const int lane = threadIdx.x & 31;
    const int gwarp = blockIdx.x * kWalkWarps + (threadIdx.x >> 5);
    if (C->status & kStFatal) return;
    int2* stack = STACK > 0 ? s_stack + (threadIdx.x >> 5) * (STACK / 4)
                            : reinterpret_cast<int2*>(LB.stack + (long long)gwarp * LB.stack_cap);
    const int stack_cap = STACK > 0 ? STACK / 4 : LB.stack_cap / 2;
    const int nleaves = C->nleaves;
    const unsigned lt_mask = (1u << lane) - 1u;
    unsigned tests = 0, retests = 0;                              // of this lane
    unsigned long long groups = 0;
    int stack_max = 0, list_max = 0;
    unsigned bad = 0;
    int fres_next = 0, fres_end = 0, nres_next = 0, nres_end = 0;  // chunk reservoirs

    for (;;) {
        int gi = 0;
        if (lane == 0) gi = atomicAdd(&C->work_next, 1);
        gi = __shfl_sync(0xffffffffu, gi, 0);
        if (gi >= nleaves) break;
        const int leaf = leaf_list[gi];
        const float4 gA = T.wA[leaf];
        const float4 gC = T.wC[leaf];
        const float4 gD = T.wD[leaf];
        const float gR = gC.x;
        double gcx_d = 0.0, gcy_d = 0.0, gcz_d = 0.0, gr_d = 0.0;
        if (wp.retest) {
            gcx_d = T.comx[leaf];
            gcy_d = T.comy[leaf];
            gcz_d = T.comz[leaf];
            gr_d = T.maxr[leaf];
        }
        ++groups;
        ChunkList far = {-1, -1, 0, 0, fres_next, fres_end}, near = {-1, -1, 0, 0, nres_next, nres_end};
        // own members first (the self term is zero)
        list_append(near, lane == 0, leaf, LB.near, LB.near_next, &C->near_chunks, LB.near_chunk_cap, lane,
                    lt_mask, bad);
        int size = 0, iterations = 0;
        const int root = T.sysroot[leaf];
        if (leaf != root) {
            // The root's test, by every lane at once (the same arithmetic as
            // the loop's, which tests the children of opened nodes).
            const float4 A = T.wA[root], Cw = T.wC[root], D = T.wD[root];
            const int meta = __float_as_int(Cw.w);
            if (A.w > 0.f && meta >= 0) {
                const float dx = (A.x - gA.x) + (D.x - gD.x);
                const float dy = (A.y - gA.y) + (D.y - gD.y);
                const float dz = (A.z - gA.z) + (D.z - gD.z);
                const float dist = sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
                const float worst = dist - gR;
                const float size_n = Cw.y;
                bool accept = worst > 0.f && size_n * size_n < wp.theta2 * worst * worst;
                if (wp.retest) {
                    const float margin = wp.theta * worst - size_n;
                    if (fabsf(margin) <= 1e-5f * (wp.theta * (dist + gR) + size_n)) {
                        if (lane == 0) ++retests;
                        const double ex = T.comx[root] - gcx_d, ey = T.comy[root] - gcy_d,
                                     ez = T.comz[root] - gcz_d;
                        const double d2 = ex * ex + ey * ey + ez * ez;
                        const double sz = 2.0 * T.half[root];
                        const double w = sqrt(d2) - gr_d;
                        accept = w > 0.0 && sz * sz < wp.theta2_d * w * w;
                    }
                }
                if (lane == 0) ++tests;
                if (accept) {
                    list_append(far, lane == 0, root, LB.far, LB.far_next, &C->far_chunks, LB.far_chunk_cap, lane,
                                lt_mask, bad);
                } else {
                    if (lane == 0) stack[0] = make_int2(__float_as_int(Cw.z), meta & 0xFFFFFF);
                    size = 1;
                }
            }
        }
        __syncwarp();
        while (size > 0) {
            const int take = min(size, 4 * kNPL);  // opened nodes; lane = child
            size -= take;
            int node[kNPL];
#pragma unroll
            for (int q = 0; q < kNPL; ++q) {
                const int p = 4 * q + (lane >> 3);
                const int2 e = p < take ? stack[size + p] : make_int2(0, 0);
                // a lane without a child reads the group's own leaf, which the tests skip
                node[q] = (lane & 7) < e.y ? e.x + (lane & 7) : leaf;
            }
            if (++iterations > wp.node_limit) {  // every iteration opens a node of its own
                bad |= kStCorrupt;
                break;
            }
            float4 A[kNPL], Cw[kNPL], Dw[kNPL];
#pragma unroll
            for (int q = 0; q < kNPL; ++q) {  // all record loads in flight together
                A[q] = T.wA[node[q]];
                Cw[q] = T.wC[node[q]];
                Dw[q] = T.wD[node[q]];
            }
            bool near_k[kNPL], far_k[kNPL], open_k[kNPL];
            int nch[kNPL], link[kNPL];
#pragma unroll
            for (int q = 0; q < kNPL; ++q) {
                const int meta = __float_as_int(Cw[q].w);
                link[q] = __float_as_int(Cw[q].z);
                nch[q] = meta & 0xFFFFFF;
                const bool massive = node[q] != leaf && A[q].w > 0.f;
                const bool inner = massive && meta >= 0;
                near_k[q] = massive && meta < 0;
                tests += inner ? 1u : 0u;
                const float4 D = Dw[q];
                const float dx = (A[q].x - gA.x) + (D.x - gD.x);
                const float dy = (A[q].y - gA.y) + (D.y - gD.y);
                const float dz = (A[q].z - gA.z) + (D.z - gD.z);
                const float dist = sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)));
                const float worst = dist - gR;
                const float size_n = Cw[q].y;
                bool accept;
                if (wp.retest) {
                    // outside the band the margin's sign is the test's outcome
                    const float margin = wp.theta * worst - size_n;
                    accept = margin > 0.f;
                    if (inner && fabsf(margin) <= 1e-5f * (wp.theta * (dist + gR) + size_n)) {
                        ++retests;
                        const int nd = node[q];
                        const double ex = T.comx[nd] - gcx_d, ey = T.comy[nd] - gcy_d, ez = T.comz[nd] - gcz_d;
                        const double d2 = ex * ex + ey * ey + ez * ez;
                        const double sz = 2.0 * T.half[nd];
                        const double w = sqrt(d2) - gr_d;
                        accept = w > 0.0 && sz * sz < wp.theta2_d * w * w;
                    }
                } else {
                    accept = worst > 0.f && size_n * size_n < wp.theta2 * worst * worst;
                }
                far_k[q] = inner && accept;
                open_k[q] = inner && !accept;
            }
            list_append_n<kNPL>(near, near_k, node, LB.near, LB.near_next, &C->near_chunks, LB.near_chunk_cap, lane,
                                lt_mask, bad);
            list_append_n<kNPL>(far, far_k, node, LB.far, LB.far_next, &C->far_chunks, LB.far_chunk_cap, lane,
                                lt_mask, bad);
            __syncwarp();  // the entries above were read by every lane
            if (!push_opened<kNPL>(stack, size, stack_cap, open_k, link, nch, lt_mask)) {
                bad |= kStStackOverflow;
                break;
            }
            stack_max = max(stack_max, 4 * size);
            __syncwarp();
        }
        fres_next = far.res_next;
        fres_end = far.res_end;
        nres_next = near.res_next;
        nres_end = near.res_end;
        if (lane == 0) LB.ginfo[gi] = make_int4(far.first, near.first, far.count, near.count);
        list_max = max(list_max, max(far.count, near.count));
        if (bad & (kStStackOverflow | kStCorrupt)) break;
    }
    unsigned long long all_tests = tests, all_retests = retests;
    for (int o = 16; o > 0; o >>= 1) {
        bad |= __shfl_xor_sync(0xffffffffu, bad, o);
        all_tests += __shfl_xor_sync(0xffffffffu, all_tests, o);
        all_retests += __shfl_xor_sync(0xffffffffu, all_retests, o);
    }
    if (lane == 0) {
        if (bad) atomicOr(&C->status, bad);
        atomicAdd(&C->mac_tests, all_tests);
        atomicAdd(&C->groups, groups);
        atomicMax(&C->stack_max, stack_max);
        atomicMax(&C->list_max, list_max);
    }
    if (lane == 0 && all_retests) atomicAdd(&C->mac_retests, all_retests);
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------

int walk_warps_per_block() { return kWalkWarps; }

int walk_blocks_per_sm() {
    int nb = 0, ng = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, walk_kernel<1024>, kWalkThreads, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ng, walk_kernel<0>, kWalkThreads, 0);
    nb = nb > ng ? nb : ng;
    return nb > 0 ? nb : 1;
}

void launch_walk(const NodeArrays& T, Counters* C, const int* leaf_list, const WalkParams& wp,
                 const ListBuffers& LB, cudaStream_t s) {
    const int blocks = (LB.nwarps + kWalkWarps - 1) / kWalkWarps;
    if (wp.global_stack)
        walk_kernel<0><<<blocks, kWalkThreads, 0, s>>>(T, C, leaf_list, wp, LB);
    else if (wp.smem_stack == 1024)
        walk_kernel<1024><<<blocks, kWalkThreads, 0, s>>>(T, C, leaf_list, wp, LB);
    else if (wp.smem_stack == 4096)
        walk_kernel<4096><<<blocks, kWalkThreads, 0, s>>>(T, C, leaf_list, wp, LB);
    else
        walk_kernel<2048><<<blocks, kWalkThreads, 0, s>>>(T, C, leaf_list, wp, LB);
}

}  // namespace ngrav
