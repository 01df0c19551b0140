// keys_sort.cu -- bounding box, 63-bit octant-path keys, stable LSD radix
// sort of (key, slot) pairs and the gather that puts the particle state into
// key order.
//
// Bit-exactness with the reference tree (projects/nbody_core/src/Tree.cpp):
//  * the root cube is the FP64 bounding box of the positions, centre
//    0.5*(lo+hi), half = max half extent (1.0 if <= 1e-12) times 1.001
//    (Tree.cpp:54-88);
//  * at each level the octant bit per axis is (p >= centre) (Tree.cpp:11-20)
//    and the child centre is centre +/- 0.5*half, rounded in FP64 exactly as
//    NewChild does (Tree.cpp:90-112).
// Key digit l (bits 3*(20-l)..+2) is the octant (x:1, y:2, z:4) of the
// particle's level-l ancestor, so ascending keys enumerate leaves in the
// reference's DFS ascending-octant order (Tree.cpp:157-175).
#include "engine.cuh"

#include <utility>

namespace ngrav {

// ---------------------------------------------------------------------------
// FP64 bounding box with order-preserving integer atomics
// ---------------------------------------------------------------------------

__device__ __forceinline__ double dec_f64(unsigned long long u) {
    u = (u & 0x8000000000000000ull) ? (u & 0x7FFFFFFFFFFFFFFFull) : ~u;
    return __longlong_as_double((long long)u);
}

constexpr int kBoxThreads = 256;

__global__ void __launch_bounds__(kBoxThreads) bbox_kernel(const float4* __restrict__ pos,
                                                           const float4* __restrict__ plo, long long n,
                                                           Counters* C) {
    DfBox box = empty_box();
    bool bad = false;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float4 p = pos[i];
        bad |= !(isfinite(p.x) && isfinite(p.y) && isfinite(p.z) && isfinite(p.w));
        box_add(box, p, plo ? plo[i] : make_float4(0.f, 0.f, 0.f, 0.f));
    }
    box_publish(box, bad, C);
}

// The key frame of a root cube: its centre as double-float, the scale
// 2^(digits - 1) / half to cells of the finest level, and how near a cell's face
// (in cells) the arithmetic of axis_cell leaves the side in doubt.  The offset
// from the centre is good to 2^-47 (|centre| + half), its product with the scale
// to 2^-46, and the reference's centres are within 21 roundings of the grid: all
// below 2^-23 (1 + |centre| / half) cells.  A scale whose low part would
// underflow is not used.
__device__ void write_frame(float4* f, double cx, double cy, double cz, double half, int digits) {
    const float hx = (float)cx, hy = (float)cy, hz = (float)cz;
    const double scale = (double)(1 << (digits - 1)) / half;
    const float sh = (float)scale;
    const double far = fmax(fmax(fabs(cx), fabs(cy)), fabs(cz)) / half;
    const float tol = sh > 1e-25f ? (float)(0x1p-20 * (1.0 + far)) : 2.f;
    f[0] = make_float4(hx, hy, hz, tol);
    f[1] = make_float4((float)(cx - (double)hx), (float)(cy - (double)hy), (float)(cz - (double)hz), sh);
    f[2] = make_float4((float)(scale - (double)sh), 0.f, 0.f, 0.f);
}

// Root cube of BuildRoot (Tree.cpp:54-88), once per evaluation.
__global__ void root_kernel(Counters* C, long long n, float4* frame) {
    double lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
        lo[a] = n > 0 ? dec_f64(C->bbox_min[a]) : 0.0;
        hi[a] = n > 0 ? dec_f64(C->bbox_max[a]) : 0.0;
    }
    double half = __dmul_rn(0.5, __dsub_rn(hi[0], lo[0]));
    const double hy = __dmul_rn(0.5, __dsub_rn(hi[1], lo[1]));
    const double hz = __dmul_rn(0.5, __dsub_rn(hi[2], lo[2]));
    if (half < hy) half = hy;
    if (half < hz) half = hz;
    if (!(half > 1e-12)) half = 1.0;
    for (int a = 0; a < 3; ++a) C->root_center[a] = __dmul_rn(0.5, __dadd_rn(lo[a], hi[a]));
    C->root_half = __dmul_rn(half, 1.001);
    write_frame(frame, C->root_center[0], C->root_center[1], C->root_center[2], C->root_half, kKeyLevels);
}

void launch_bbox(const float4* pos, const float4* plo, long long n, Counters* C, cudaStream_t s) {
    long long blocks = (n + kBoxThreads - 1) / kBoxThreads;
    if (blocks > 152 * 8) blocks = 152 * 8;
    if (blocks < 1) blocks = 1;
    bbox_kernel<<<(unsigned)blocks, kBoxThreads, 0, s>>>(pos, plo, n, C);
}

void launch_root(Counters* C, long long n, float4* frame, cudaStream_t s) {
    root_kernel<<<1, 1, 0, s>>>(C, n, frame);
}

// Ensemble: per-system FP64 bounding boxes.  Slots are grouped by system, so a
// warp whose 32 slots share one system reduces in registers first; mixed warps
// fall back to per-lane atomics.
__global__ void __launch_bounds__(kBoxThreads) forest_bbox_kernel(const float4* __restrict__ pos,
                                                                  const float4* __restrict__ plo, long long n,
                                                                  Forest F, Counters* C) {
    const int lane = threadIdx.x & 31;
    bool bad = false;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += stride) {
        const long long i = base + lane;
        const bool has = i < n;
        int sys = has ? forest_system(F, i) : -1;
        DfBox box = empty_box();
        if (has) {
            const float4 p = pos[i];
            bad |= !(isfinite(p.x) && isfinite(p.y) && isfinite(p.z) && isfinite(p.w));
            box_add(box, p, plo ? plo[i] : make_float4(0.f, 0.f, 0.f, 0.f));
        }
        const int s0 = __shfl_sync(0xffffffffu, sys, 0);
        const bool uniform = __all_sync(0xffffffffu, !has || sys == s0);
        if (uniform) {
            box_warp(box);
            sys = s0;
        }
        if (uniform ? lane == 0 : has) {
            for (int a = 0; a < 3; ++a) {
                atomicMin(&F.bbox[6 * sys + a], enc_df(box.lo[a]));
                atomicMax(&F.bbox[6 * sys + 3 + a], enc_df(box.hi[a]));
            }
        }
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&C->status, kStNonFinite);
}

// BuildRoot (Tree.cpp:54-88) of every system; resets the boxes for the next
// evaluation.
__global__ void forest_root_kernel(Forest F) {
    for (int sys = blockIdx.x * blockDim.x + threadIdx.x; sys < F.nsys; sys += gridDim.x * blockDim.x) {
        const bool empty = F.off[sys + 1] <= F.off[sys];
        double lo[3], hi[3];
        for (int a = 0; a < 3; ++a) {
            lo[a] = empty ? 0.0 : dec_f64(F.bbox[6 * sys + a]);
            hi[a] = empty ? 0.0 : dec_f64(F.bbox[6 * sys + 3 + a]);
            F.bbox[6 * sys + a] = ~0ull;
            F.bbox[6 * sys + 3 + a] = 0ull;
        }
        double half = __dmul_rn(0.5, __dsub_rn(hi[0], lo[0]));
        const double hy = __dmul_rn(0.5, __dsub_rn(hi[1], lo[1]));
        const double hz = __dmul_rn(0.5, __dsub_rn(hi[2], lo[2]));
        if (half < hy) half = hy;
        if (half < hz) half = hz;
        if (!(half > 1e-12)) half = 1.0;
        for (int a = 0; a < 3; ++a) F.root[4 * sys + a] = __dmul_rn(0.5, __dadd_rn(lo[a], hi[a]));
        F.root[4 * sys + 3] = __dmul_rn(half, 1.001);
        write_frame(F.frame + kFrame * sys, F.root[4 * sys], F.root[4 * sys + 1], F.root[4 * sys + 2],
                    F.root[4 * sys + 3], kKeyLevels - F.sys_levels);
    }
}

void launch_forest_bbox(const float4* pos, const float4* plo, long long n, const Forest& F, Counters* C,
                        cudaStream_t s) {
    long long blocks = (n + kBoxThreads - 1) / kBoxThreads;
    if (blocks > 152 * 8) blocks = 152 * 8;
    if (blocks < 1) blocks = 1;
    forest_bbox_kernel<<<(unsigned)blocks, kBoxThreads, 0, s>>>(pos, plo, n, F, C);
}

void launch_forest_root(const Forest& F, cudaStream_t s) {
    forest_root_kernel<<<(F.nsys + 127) / 128, 128, 0, s>>>(F);
}

// SPLIT -> PLAIN: fold the low halves into FP32 positions.
__global__ void collapse_split_kernel(float4* __restrict__ pos, float4* __restrict__ plo, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float4 p = pos[i];
        const float4 l = plo[i];
        p.x = (float)((double)p.x + (double)l.x);
        p.y = (float)((double)p.y + (double)l.y);
        p.z = (float)((double)p.z + (double)l.z);
        pos[i] = p;
        plo[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

void launch_collapse_split(float4* pos, float4* plo, long long n, cudaStream_t s) {
    long long blocks = (n + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (blocks < 1) blocks = 1;
    collapse_split_kernel<<<(unsigned)blocks, 256, 0, s>>>(pos, plo, n);
}

// ---------------------------------------------------------------------------
// 63-bit keys by the reference's FP64 centre recurrence
// ---------------------------------------------------------------------------

__device__ __forceinline__ long long ordered_bits(double x) {
    // Integer image of a finite double that orders like the double (-0
    // taken as +0): one 64-bit compare replaces the FP64 comparison.
    long long b = __double_as_longlong(x);
    if (b == (long long)0x8000000000000000ull) b = 0;
    return b ^ ((b >> 63) & 0x7FFFFFFFFFFFFFFFll);
}

template <int LEVELS>
__device__ __forceinline__ unsigned axis_bits(double p, double c, double h) {
    // Returns LEVELS octant bits of one axis, level 0 in the highest bit:
    // bit = p >= c, then h = h / 2 and c = c +- h rounded in FP64 (NewChild).
    // GB300's FP64 pipe is narrow, so only the centre add stays FP64: the
    // comparison is an integer compare of ordered bit images, the halving an
    // exponent decrement (exact: h >= 1e-12 stays normal over 21 levels) and
    // c - h the addition of -h (the same IEEE result).
    const long long op = ordered_bits(p);
    long long hb = __double_as_longlong(h);
    unsigned bits = 0;
#pragma unroll
    for (int l = 0; l < LEVELS; ++l) {
        const bool b = op >= ordered_bits(c);
        bits = (bits << 1) | (b ? 1u : 0u);
        hb -= 1ll << 52;
        c = __dadd_rn(c, __longlong_as_double(b ? hb : (hb | (long long)0x8000000000000000ull)));
    }
    return bits;
}

// Cell of the finest of `digits` levels along one axis, without the FP64 pipe:
// the double-float offset from the root's centre times the scale, split into
// its whole part and fraction.  A cell's bits are the reference's octant bits
// unless a face is within the frame's tolerance, which `doubt` reports; then the
// centre recurrence decides (axis_bits).  In doubt is about one particle in
// 170,000 of a system around its origin.
__device__ __forceinline__ unsigned axis_cell(float h, float l, float ch, float cl, float sh, float sl, float tol,
                                              int digits, bool& doubt) {
    float oh, ol;
    df_offset(h, l, ch, cl, oh, ol);
    const float p = __fmul_rn(oh, sh);
    const float e = fmaf(oh, sh, -p) + fmaf(oh, sl, ol * sh);
    const float whole = floorf(p);
    float f = (p - whole) + e;
    int q = (int)whole + (1 << (digits - 1));
    if (f < 0.f) {
        f += 1.f;
        q -= 1;
    } else if (f >= 1.f) {
        f -= 1.f;
        q += 1;
    }
    doubt |= !(f > tol && f < 1.f - tol) || (unsigned)q >= (1u << digits);
    return (unsigned)q;
}

// Spread 21 bits so bit k lands at 3k.
__device__ __forceinline__ unsigned long long spread3(unsigned v) {
    unsigned long long x = v & 0x1FFFFFull;
    x = (x | (x << 32)) & 0x1F00000000FFFFull;
    x = (x | (x << 16)) & 0x1F0000FF0000FFull;
    x = (x | (x << 8)) & 0x100F00F00F00F00Full;
    x = (x | (x << 4)) & 0x10C30C30C30C30C3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}

// Keys: the system id in the top SYSL digits (none for a single system), then
// 21 - SYSL levels of octant path from the system's root cube.  Reads of the
// positions and writes of the keys bound it; the centre recurrence in FP64 for
// every particle, with the top 17 levels tabulated per build, was bound by the
// FP64 pipe.  Box, root and keys together, before and now: 2,048 bodies 41 and
// 20 us, 4 Mi bodies 347 and 103 us, 16.8 M 1,264 and 332 us, 64 systems of
// 955 k bodies 276 and 119 us.
template <int SYSL>
__global__ void __launch_bounds__(256) keys_kernel(const float4* __restrict__ pos, const float4* __restrict__ plo,
                                                   long long n, const Counters* __restrict__ C, Forest F,
                                                   const float4* __restrict__ frame,
                                                   unsigned long long* __restrict__ keys,
                                                   unsigned* __restrict__ vals) {
    constexpr int L = kKeyLevels - SYSL;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int sys = SYSL > 0 ? forest_system(F, i) : 0;
        const float4 p = pos[i];
        const float4 l = plo ? plo[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 f0 = frame[kFrame * sys], f1 = frame[kFrame * sys + 1];
        const float sl = frame[kFrame * sys + 2].x;
        bool doubt = false;
        unsigned bx = axis_cell(p.x, l.x, f0.x, f1.x, f1.w, sl, f0.w, L, doubt);
        unsigned by = axis_cell(p.y, l.y, f0.y, f1.y, f1.w, sl, f0.w, L, doubt);
        unsigned bz = axis_cell(p.z, l.z, f0.z, f1.z, f1.w, sl, f0.w, L, doubt);
        if (doubt) {
            const double* root = SYSL > 0 ? F.root + 4 * sys : C->root_center;
            const double h0 = SYSL > 0 ? root[3] : C->root_half;
            bx = axis_bits<L>((double)p.x + (double)l.x, root[0], h0);
            by = axis_bits<L>((double)p.y + (double)l.y, root[1], h0);
            bz = axis_bits<L>((double)p.z + (double)l.z, root[2], h0);
        }
        const unsigned long long id = SYSL > 0 ? (unsigned long long)sys << (3 * L % 64) : 0ull;
        keys[i] = id | spread3(bx) | (spread3(by) << 1) | (spread3(bz) << 2);
        vals[i] = (unsigned)i;
    }
}

void launch_keys(const float4* pos, const float4* plo, long long n, Counters* C, const Forest& F, const float4* frame,
                 unsigned long long* keys, unsigned* vals, cudaStream_t s) {
    long long blocks = (n + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (blocks < 1) blocks = 1;
    const unsigned g = (unsigned)blocks;
    switch (F.sys_levels) {
        case 0: keys_kernel<0><<<g, 256, 0, s>>>(pos, plo, n, C, F, frame, keys, vals); break;
        case 1: keys_kernel<1><<<g, 256, 0, s>>>(pos, plo, n, C, F, F.frame, keys, vals); break;
        case 2: keys_kernel<2><<<g, 256, 0, s>>>(pos, plo, n, C, F, F.frame, keys, vals); break;
        case 3: keys_kernel<3><<<g, 256, 0, s>>>(pos, plo, n, C, F, F.frame, keys, vals); break;
        case 4: keys_kernel<4><<<g, 256, 0, s>>>(pos, plo, n, C, F, F.frame, keys, vals); break;
        case 5: keys_kernel<5><<<g, 256, 0, s>>>(pos, plo, n, C, F, F.frame, keys, vals); break;
        default: keys_kernel<6><<<g, 256, 0, s>>>(pos, plo, n, C, F, F.frame, keys, vals); break;
    }
}

// Block-wide exclusive scan of one value per thread; returns the block total.
__device__ __forceinline__ unsigned block_exclusive_scan(unsigned v, unsigned* s_warp, unsigned& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[w] = x;
    __syncthreads();
    if (w == 0) {
        unsigned t = lane < nw ? s_warp[lane] : 0u;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < nw) s_warp[lane] = t;
    }
    __syncthreads();
    total = s_warp[nw - 1];
    const unsigned before = w > 0 ? s_warp[w - 1] : 0u;
    __syncthreads();
    return before + x - v;
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort, 9-bit digits (seven passes cover the 63-bit keys),
// tiles of 4096 keys (512 threads x 8); two or three kernels per pass (tile
// histograms, per-digit scans over the tiles, scatter)
// ---------------------------------------------------------------------------

constexpr int kRsThreads = 512;
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kRsItems = 8;
constexpr int kRsTile = kRsThreads * kRsItems;   // 4096
constexpr int kRsWarpSpan = 32 * kRsItems;       // consecutive keys per warp
constexpr int kRsScatterMinBlocks = 2;
constexpr unsigned kRsMask = kRsBins - 1;
constexpr int kRsDpt = kRsBins / kRsThreads;     // digits per thread in the digit scans
static_assert(kRsDpt * kRsThreads == kRsBins, "whole digits per thread in the digit scans");

// Lanes of the warp holding the same digit as this lane (the invalid lanes of
// a ragged last tile form a group of their own): the AND of one ballot per
// digit bit, cheaper than a warp match.
__device__ __forceinline__ unsigned digit_peers(unsigned d, bool valid) {
    const unsigned vb = __ballot_sync(0xffffffffu, valid);
    unsigned peers = valid ? vb : ~vb;
#pragma unroll
    for (int b = 0; b < kRsDigitBits; ++b) {
        const bool bit = (d >> b) & 1u;
        const unsigned bb = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? bb : ~bb;
    }
    return peers;
}

// Histogram of one digit per tile, digit-major: hist[d * nblocks + b].  All
// keys of a thread are loaded before the first is counted; plain shared
// atomics (a warp match to combine equal digits costs more than the
// conflicts it saves).
__global__ void __launch_bounds__(kRsThreads) rs_hist_kernel(const unsigned long long* __restrict__ keys,
                                                             long long n, int shift, unsigned* __restrict__ hist) {
    __shared__ unsigned h[kRsBins];
#pragma unroll
    for (int j = 0; j < kRsDpt; ++j) h[threadIdx.x + j * kRsThreads] = 0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long base = blockIdx.x * (long long)kRsTile + w * kRsWarpSpan + lane;
    unsigned d[kRsItems];
#pragma unroll
    for (int k = 0; k < kRsItems; ++k) {
        const long long i = base + k * 32;
        d[k] = i < n ? (unsigned)(__ldg(keys + i) >> shift) & kRsMask : (unsigned)kRsBins;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kRsItems; ++k) {
        if (d[k] < (unsigned)kRsBins) atomicAdd(&h[d[k]], 1u);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kRsDpt; ++j)
        hist[(threadIdx.x + j * kRsThreads) * gridDim.x + blockIdx.x] = h[threadIdx.x + j * kRsThreads];
}

// One block per digit d: exclusive scan over the tiles of row d of the
// histogram, in place, and the row's total into totals[d].  The scatter adds
// the digit's own offset (the exclusive scan of the totals) itself.
__global__ void __launch_bounds__(kRsThreads) rs_scan_kernel(unsigned* __restrict__ hist, int nb,
                                                             unsigned* __restrict__ totals) {
    __shared__ unsigned s_warp[32];
    unsigned* row = hist + (long long)blockIdx.x * nb;
    constexpr int kPer = 4;
    unsigned carry = 0;
    for (int c0 = 0; c0 < nb; c0 += kRsThreads * kPer) {
        const int i0 = c0 + threadIdx.x * kPer;
        unsigned v[kPer];
        unsigned sum = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            v[k] = i0 + k < nb ? row[i0 + k] : 0u;
            sum += v[k];
        }
        unsigned total;
        unsigned run = carry + block_exclusive_scan(sum, s_warp, total);
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            if (i0 + k < nb) row[i0 + k] = run;
            run += v[k];
        }
        carry += total;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// The tile's keys are ranked by digit in shared memory and written out in
// digit runs.  The per-warp digit counters share the tile buffer (they are
// dead once every key holds its rank), so a CTA holds 53 KB; at 64 registers
// two CTAs of 512 threads share an SM.
constexpr size_t kRsScatterSmem = (size_t)kRsTile * (sizeof(unsigned long long) + sizeof(unsigned));
static_assert(kRsWarps * kRsBins * sizeof(unsigned) <= kRsScatterSmem, "digit counters fit the tile buffer");

// FEW: the histogram is as rs_hist_kernel left it, and each thread adds its
// digit's row up itself, which for few tiles is quicker than a launch of
// rs_scan_kernel.
template <bool FEW>
__global__ void __launch_bounds__(kRsThreads, kRsScatterMinBlocks)
    rs_scatter_kernel(const unsigned long long* __restrict__ kin,
                      const unsigned* __restrict__ vin,
                      unsigned long long* __restrict__ kout,
                      unsigned* __restrict__ vout, long long n, int shift,
                      const unsigned* __restrict__ hist_scan,
                      const unsigned* __restrict__ totals) {
    extern __shared__ unsigned long long rs_smem[];
    unsigned long long* skeys = rs_smem;                             // kRsTile
    unsigned* svals = reinterpret_cast<unsigned*>(skeys + kRsTile);  // kRsTile
    unsigned (*warp_cnt)[kRsBins] = reinterpret_cast<unsigned (*)[kRsBins]>(rs_smem);  // aliases skeys
    __shared__ unsigned digit_start[kRsBins];   // block-local exclusive prefix over digits
    __shared__ unsigned digit_base[kRsBins];    // global output offset of (digit, block)
    __shared__ unsigned s_warp[32];

    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < kRsWarps * kRsBins; k += kRsThreads) (&warp_cnt[0][0])[k] = 0;

    const long long tile = blockIdx.x * (long long)kRsTile;
    const long long base = tile + w * kRsWarpSpan + lane;
    const unsigned lt_mask = (1u << lane) - 1u;
    unsigned long long key[kRsItems];
    unsigned val[kRsItems];
    unsigned short rank[kRsItems];
#pragma unroll
    for (int k = 0; k < kRsItems; ++k) {
        const long long i = base + k * 32;
        const bool valid = i < n;
        key[k] = valid ? kin[i] : 0ull;
        val[k] = valid ? vin[i] : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kRsItems; ++k) {
        const bool valid = base + k * 32 < n;
        const unsigned d = valid ? (unsigned)(key[k] >> shift) & kRsMask : (unsigned)kRsBins;
        const unsigned peers = digit_peers(d, valid);
        unsigned before = 0;
        if (valid) before = warp_cnt[w][d];
        __syncwarp();
        if (valid) {
            rank[k] = (unsigned short)(before + __popc(peers & lt_mask));
            if ((__ffs(peers) - 1) == lane) warp_cnt[w][d] = before + __popc(peers);
        }
        __syncwarp();
    }
    __syncthreads();
    // Per digit (thread t: digits kRsDpt t ...): exclusive prefix over warps
    // (stable: warp w precedes w+1), then over digits; the digit's global
    // offset is the scan of the digit totals plus this tile's row prefix.
    unsigned run[kRsDpt], tot[kRsDpt], before[kRsDpt];
    unsigned rsum = 0, tsum = 0;
#pragma unroll
    for (int j = 0; j < kRsDpt; ++j) {
        const unsigned d = kRsDpt * threadIdx.x + j;
        run[j] = 0;
#pragma unroll
        for (int ww = 0; ww < kRsWarps; ++ww) {
            const unsigned c = warp_cnt[ww][d];
            warp_cnt[ww][d] = run[j];
            run[j] += c;
        }
        if (FEW) {
            const unsigned* row = hist_scan + d * gridDim.x;
            tot[j] = 0;
            before[j] = 0;
#pragma unroll 8
            for (unsigned b = 0; b < gridDim.x; ++b) {
                const unsigned c = __ldg(row + b);
                before[j] += b < blockIdx.x ? c : 0u;
                tot[j] += c;
            }
        } else {
            tot[j] = __ldg(totals + d);
            before[j] = __ldg(hist_scan + d * gridDim.x + blockIdx.x);
        }
        rsum += run[j];
        tsum += tot[j];
    }
    unsigned total;
    unsigned ds = block_exclusive_scan(rsum, s_warp, total);
    unsigned gs = block_exclusive_scan(tsum, s_warp, total);
#pragma unroll
    for (int j = 0; j < kRsDpt; ++j) {
        const unsigned d = kRsDpt * threadIdx.x + j;
        digit_start[d] = ds;
        digit_base[d] = gs + before[j];
        ds += run[j];
        gs += tot[j];
    }
    __syncthreads();
    // every key's place in the tile, then (counters dead) the tile itself
#pragma unroll
    for (int k = 0; k < kRsItems; ++k) {
        if (base + k * 32 < n) {
            const unsigned dd = (unsigned)(key[k] >> shift) & kRsMask;
            rank[k] = (unsigned short)(digit_start[dd] + warp_cnt[w][dd] + rank[k]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kRsItems; ++k) {
        if (base + k * 32 < n) {
            skeys[rank[k]] = key[k];
            svals[rank[k]] = val[k];
        }
    }
    __syncthreads();
    long long nvalid = n - tile;
    if (nvalid > kRsTile) nvalid = kRsTile;
    for (int j = threadIdx.x; j < nvalid; j += kRsThreads) {
        const unsigned long long kk = skeys[j];
        const unsigned dd = (unsigned)(kk >> shift) & kRsMask;
        const unsigned o = digit_base[dd] + (unsigned)j - digit_start[dd];
        kout[o] = kk;
        vout[o] = svals[j];
    }
}

// All passes of up to THREADS x kRsItems keys in one CTA: the keys stay in
// registers, a pass ranks them as the scatter does and exchanges them through
// shared memory.  Three launches per pass cost a chain of latencies, some
// 16 us a pass at any small size.  THREADS by size: the fewer warps, the
// cheaper the prefix over them.  Sort phase (with the gather), before and now:
// 1,000 bodies (2 passes) 37 and 15 us, 2,048 (3 passes) 64 and 19 us.  More keys
// than one CTA holds take two or three launches a pass.
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1) rs_single_kernel(unsigned long long* __restrict__ keys,
                                                              unsigned* __restrict__ vals, int n, int passes,
                                                              int shift0) {
    constexpr int WARPS = THREADS / 32, TILE = THREADS * kRsItems;
    static_assert(WARPS * kRsBins * sizeof(unsigned) <= TILE * (sizeof(unsigned long long) + sizeof(unsigned)),
                  "digit counters fit the tile buffer");
    static_assert(THREADS >= kRsBins, "a thread per digit");
    extern __shared__ unsigned long long rs_smem[];
    unsigned long long* skeys = rs_smem;
    unsigned* svals = reinterpret_cast<unsigned*>(skeys + TILE);
    unsigned (*warp_cnt)[kRsBins] = reinterpret_cast<unsigned (*)[kRsBins]>(rs_smem);  // aliases skeys
    __shared__ unsigned digit_start[kRsBins];
    __shared__ unsigned s_warp[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int base = w * kRsWarpSpan + lane;
    const unsigned lt_mask = (1u << lane) - 1u;
    unsigned long long key[kRsItems];
    unsigned val[kRsItems];
    unsigned short rank[kRsItems];
#pragma unroll
    for (int k = 0; k < kRsItems; ++k) {
        const int i = base + k * 32;
        key[k] = i < n ? keys[i] : 0ull;
        val[k] = i < n ? vals[i] : 0u;
    }
    for (int p = 0; p < passes; ++p) {
        const int shift = shift0 + kRsDigitBits * p;
        for (int k = threadIdx.x; k < WARPS * kRsBins; k += THREADS) (&warp_cnt[0][0])[k] = 0;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kRsItems; ++k) {
            const bool valid = base + k * 32 < n;
            const unsigned d = valid ? (unsigned)(key[k] >> shift) & kRsMask : (unsigned)kRsBins;
            const unsigned peers = digit_peers(d, valid);
            unsigned before = 0;
            if (valid) before = warp_cnt[w][d];
            __syncwarp();
            if (valid) {
                rank[k] = (unsigned short)(before + __popc(peers & lt_mask));
                if ((__ffs(peers) - 1) == lane) warp_cnt[w][d] = before + __popc(peers);
            }
            __syncwarp();
        }
        __syncthreads();
        unsigned run = 0;
        if (threadIdx.x < kRsBins) {
#pragma unroll
            for (int ww = 0; ww < WARPS; ++ww) {
                const unsigned c = warp_cnt[ww][threadIdx.x];
                warp_cnt[ww][threadIdx.x] = run;
                run += c;
            }
        }
        unsigned total;
        const unsigned ds = block_exclusive_scan(run, s_warp, total);
        if (threadIdx.x < kRsBins) digit_start[threadIdx.x] = ds;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kRsItems; ++k) {
            if (base + k * 32 < n) {
                const unsigned d = (unsigned)(key[k] >> shift) & kRsMask;
                rank[k] = (unsigned short)(digit_start[d] + warp_cnt[w][d] + rank[k]);
            }
        }
        __syncthreads();  // the counters are dead
#pragma unroll
        for (int k = 0; k < kRsItems; ++k) {
            if (base + k * 32 < n) {
                skeys[rank[k]] = key[k];
                svals[rank[k]] = val[k];
            }
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kRsItems; ++k) {
            const int i = base + k * 32;
            if (i < n) {
                key[k] = skeys[i];
                val[k] = svals[i];
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < kRsItems; ++k) {
        const int i = base + k * 32;
        if (i < n) {
            keys[i] = key[k];
            vals[i] = val[k];
        }
    }
}

constexpr int kRsSingleMax = 1024 * kRsItems;
// Tiles up to which a pass is two launches (FEW).  Sort phase with three and with
// two, Plummer sphere, 4 passes: 4 tiles 78 and 63 us, 12 78 and 64, 20 82 and 70,
// 28 81 and 74, 32 83 and 98; galaxy, 5 passes: 96 and 78, 99 and 80, 101 and 85,
// 101 and 91, 101 and 121.
constexpr int kRsFewTiles = 28;

constexpr int rs_single_smem(int threads) {
    return threads * kRsItems * (int)(sizeof(unsigned long long) + sizeof(unsigned));
}

template <int THREADS>
static void launch_single(SortBuffers& sb, int n, int passes, int shift0, cudaStream_t s) {
    rs_single_kernel<THREADS><<<1, THREADS, rs_single_smem(THREADS), s>>>(sb.keys, sb.vals, n, passes, shift0);
}

void sort_set_attributes() {
    const auto kind = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaFuncSetAttribute(rs_single_kernel<kRsThreads>, kind, rs_single_smem(kRsThreads));
    cudaFuncSetAttribute(rs_single_kernel<1024>, kind, rs_single_smem(1024));
    cudaFuncSetAttribute(rs_scatter_kernel<false>, kind, (int)kRsScatterSmem);
    cudaFuncSetAttribute(rs_scatter_kernel<true>, kind, (int)kRsScatterSmem);
}

long long radix_hist_size(long long n) { return ((n + kRsTile - 1) / kRsTile + 1) * kRsBins; }

bool sort_from_alt(long long n, int passes) { return n > kRsSingleMax && (passes & 1); }

int radix_sort_pairs(SortBuffers& sb, long long n, int passes, int shift0, cudaStream_t s) {
    if (n <= 1) return 0;
    if (n <= kRsTile) {
        launch_single<kRsThreads>(sb, (int)n, passes, shift0, s);
        return 1;
    }
    if (n <= kRsSingleMax) {
        launch_single<1024>(sb, (int)n, passes, shift0, s);
        return 1;
    }
    const int nb = (int)((n + kRsTile - 1) / kRsTile);
    const bool few = nb <= kRsFewTiles;
    unsigned* totals = sb.hist + (long long)nb * kRsBins;
    unsigned long long *kin = sb.keys, *kout = sb.keys_alt;
    unsigned *vin = sb.vals, *vout = sb.vals_alt;
    if (sort_from_alt(n, passes)) {
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    for (int p = 0; p < passes; ++p) {
        const int shift = shift0 + kRsDigitBits * p;
        rs_hist_kernel<<<nb, kRsThreads, 0, s>>>(kin, n, shift, sb.hist);
        if (few) {
            rs_scatter_kernel<true>
                <<<nb, kRsThreads, kRsScatterSmem, s>>>(kin, vin, kout, vout, n, shift, sb.hist, totals);
        } else {
            rs_scan_kernel<<<kRsBins, kRsThreads, 0, s>>>(sb.hist, nb, totals);
            rs_scatter_kernel<false>
                <<<nb, kRsThreads, kRsScatterSmem, s>>>(kin, vin, kout, vout, n, shift, sb.hist, totals);
        }
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    return (few ? 2 : 3) * passes;
}

// ---------------------------------------------------------------------------
// Gather the state into key order: new[k] = old[perm[k]] (into the *2 buffers)
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(256) permute_kernel(const unsigned* __restrict__ perm, long long n,
                                                      const float4* __restrict__ pos, const float4* __restrict__ plo,
                                                      const float4* __restrict__ vel, const float4* __restrict__ vlo,
                                                      const float4* __restrict__ acc,
                                                      const int* __restrict__ id, float4* __restrict__ pos2,
                                                      float4* __restrict__ plo2, float4* __restrict__ vel2,
                                                      float4* __restrict__ vlo2, float4* __restrict__ acc2,
                                                      int* __restrict__ id2) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const unsigned j = perm[k];
        pos2[k] = pos[j];
        if (plo) plo2[k] = plo[j];
        vel2[k] = vel[j];
        if (vlo) vlo2[k] = vlo[j];
        acc2[k] = acc[j];
        id2[k] = id[j];
    }
}

void launch_permute(const Particles& P, const unsigned* perm, long long n, bool split, cudaStream_t s) {
    long long blocks = (n + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (blocks < 1) blocks = 1;
    permute_kernel<<<(unsigned)blocks, 256, 0, s>>>(perm, n, P.pos, split ? P.plo : nullptr, P.vel,
                                                     split ? P.vlo : nullptr, P.acc, P.id, P.pos2,
                                                     split ? P.plo2 : nullptr, P.vel2, split ? P.vlo2 : nullptr,
                                                     P.acc2, P.id2);
}

}  // namespace ngrav
