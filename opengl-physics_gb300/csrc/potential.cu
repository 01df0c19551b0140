// potential.cu -- the exact pair potential of the conservation diagnostics,
// sum over i < j of -m_i m_j / sqrt(r^2 + eps^2) (Plummer) or m_i m_j phi(r/h)/h
// (spline), restating System::TotalEnergy (include/ngrav/System.hpp:119-150).
//
// The sum is needed to double-precision accuracy, and GB300's FP64 pipe runs at
// 1/64 of the FP32 rate: an FP64 pair costs about 21 FP64 operations, 1,344 FP32
// slots.  potential_df_kernel forms each term on the packed FP32 pipe as an
// unevaluated pair of floats instead, in about 54 FP32 operations, and leaves
// FP64 to the sums (one flush per 32 sources):
//
//  * Frame.  Targets and sources of a (128 targets, 32 sources) tile are taken
//    relative to the tile's middle target and scaled by a power of two so the
//    largest |coordinate| E lies in [1/2, 1).  Each coordinate is split into
//    x1 on the grid 2^-22 and the rest x2, so a difference of two x1 is exact
//    in one subtraction and the difference of two x2 is off by 2^-48 E only.
//    Masses are scaled by a power of two so the largest of the 32 lies in [1, 2).
//  * r^2 + eps^2.  B = the FP32 sum of squares seeds three fused steps h += s^2
//    that all round at B's exponent; h_k - h_(k-1) is then exact (Sterbenz) and
//    one more fma recovers what each step rounded off, so B plus the collected
//    remainder is r^2 + eps^2 (inv_dist).
//  * 1/r.  The hardware reciprocal square root y0 of B, with the residual
//    e = 1 - (r^2 + eps^2) y0^2 taken by fma: y = y0 (1 + e/2 + 3/8 e^2).
//  * Sum.  m y0 + m corr as a float pair, two-sum accumulated over 32 sources,
//    then added to the thread's FP64 total.
//
// What a term is good to falls with its distance, as the remainder and the
// differences of the x2 are single FP32 numbers: rms 2^-46 of it at r = E, 2^-42 at
// E/16, 2^-38.8 at worst.  So a sum is as good as its terms are many and their
// errors independent, and the rest goes other ways:
//  * a pair nearer than E/16 is formed again from the particles' own double-float
//    positions with error-free differences (refine_pair), and pairs inside the
//    spline's kernel or at r = 0 take the FP64 formula;
//  * where a target's 32 sources hold more than 2^-12 of the energy
//    (potential_large), or FP32 does not hold their numbers, they are summed in
//    FP64 (frame_f64);
//  * with masses of both signs, and below kPotDfMin, all pairs are FP64.
// Emulated on the CPU with exact rounding against 80-bit sums (Plummer spheres in
// double-float and in FP32 positions, eps 0 to 0.05), the sum's relative error, rms
// and worst, and that of FP64 terms: n = 1,000 6e-16, 1e-15 and 2e-16, 4e-16; 2,048
// 4e-16, 6e-16 and 2e-16, 4e-16; 4,096 1e-16, 2e-16 and 3e-16, 5e-16; 16,384 5e-17,
// 1e-16 and 4e-16, 7e-16; hence kPotDfMin.  On the GPU, 4,096 to 16,384 bodies
// (Plummer, galaxy; both softenings): rms 7e-17, worst 1.9e-16 in tree order, 2e-16
// and 3.6e-16 in another; FP64 terms 1.8e-16 and 5.7e-16.
//
// Measured (GB300, one diagnostics call on a Plummer sphere in tree order):
// 131,071 particles 300 ms with FP64 terms -> 17.4 to 18.0 ms (the kernel 17.0: 0.68 of
// the FP32 pipe's 54-operation time), 16,384 15.0 -> 0.37 ms, 2,048 (FP64 blocks of 32 sources
// instead of whole rows) 1.87 -> 0.17 ms; spline, 20,011: 53.6 -> 0.7 ms.
// Particles not yet in tree order have wide frames, so more pairs take
// refine_pair: 45 ms at 131,071.
#include "ctx_kernels.cuh"
#include "engine.cuh"
#include "softening.cuh"

#include <algorithm>
#include <cmath>

namespace ngrav {

constexpr int kPotThreads = 128;           // targets per block
constexpr int kPotSub = 32;                // sources per frame (one staging warp)
constexpr int kPotChunkMax = 8192;         // sources per block at most, but no more than
constexpr int kPotChunks = 16;             //   this many blocks per target tile
// Smallest n of the double-float kernel: from here on its error is below that of
// FP64 terms (above).  A call takes 0.30 ms at 4,095 and 0.12 at 4,096 particles.
constexpr long long kPotDfMin = 4096;
constexpr float kPotNear2 = 1.f / 512.f;   // (E/16)^2 at E = 1/sqrt(2); E is in [1/2, 1)

// Sources per block: whole frames, few enough that the triangle's blocks
// fill the GPU several times over (152 SMs x 4 CTAs x 6), up to kPotChunkMax
// or a kPotChunks-th of n.
static long long potential_chunk(long long n) {
    const long long unit = n < kPotDfMin ? kPotSub : kPotThreads;
    const long long want = n * n / (2LL * kPotThreads * 152 * 4 * 6);  // n < 2^31: no overflow
    const long long most = std::max<long long>(kPotChunkMax, (n + kPotChunks - 1) / kPotChunks);
    return (std::min(most, std::max(unit, want)) + unit - 1) / unit * unit;
}

static long long pot_tiles(long long n) { return (n + kPotThreads - 1) / kPotThreads; }
static long long pot_chunks(long long n) { return (n + potential_chunk(n) - 1) / potential_chunk(n); }

int potential_blocks(long long n) { return (int)std::max<long long>(1, pot_tiles(n) * pot_chunks(n)); }

// ---------------------------------------------------------------------------
// FP32 and packed FP32 steps under one name (no step may be contracted or
// reassociated: the error-free transformations depend on each rounding).
// ---------------------------------------------------------------------------

// A packed operand has no free negation, so differences are fused steps with
// -1 (the same rounding) and signs are carried where they are needed.
__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float vsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float vrsqrt(float a) { return rsqrtf(a); }
__device__ __forceinline__ float vneg(float a) { return -a; }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return add2(a, b); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return mul2(a, b); }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return fma2(a, b, c); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return fma2(b, dup2(-1.f), a); }
__device__ __forceinline__ float2 vrsqrt(float2 a) { return make_float2(rsqrtf(a.x), rsqrtf(a.y)); }
__device__ __forceinline__ float2 vneg(float2 a) { return make_float2(-a.x, -a.y); }
template <class V>
__device__ __forceinline__ V splat(float v);
template <>
__device__ __forceinline__ float splat<float>(float v) { return v; }
template <>
__device__ __forceinline__ float2 splat<float2>(float v) { return make_float2(v, v); }

// a + b = s + e exactly.
template <class V>
__device__ __forceinline__ void sum2(V a, V b, V& s, V& e) {
    s = vadd(a, b);
    const V bb = vsub(s, a);
    e = vadd(vsub(a, vsub(s, bb)), vsub(b, bb));
}

// One fused step h += s^2; returns what it rounded off.
template <class V>
__device__ __forceinline__ V square_step(V s, V& h) {
    const V h2 = vfma(s, s, h);
    const V rest = vfma(s, s, vsub(h, h2));
    h = h2;
    return rest;
}

// B: FP32 r^2 + eps^2 from the leading differences.
template <class V>
__device__ __forceinline__ V lead_r2(const V s[3], V e2h) {
    return vfma(s[0], s[0], vfma(s[1], s[1], vfma(s[2], s[2], e2h)));
}

// 1 / sqrt(|s + l|^2 + eps^2) as y0 + corr, from l2 = 2 l and B = lead_r2(s);
// ny0 = -y0.
//
// No rounding here may lean one way, or millions of terms add it up: 2^-50 of
// each would be more than the error of an FP64 sum.  So
//  * the cross terms are fused products s l2, exact before they are rounded, and
//    what the square steps rounded off and the error of adding e2h (all on the
//    grid 2^-44) are added exactly: a constant of finer bits would be rounded the
//    same way in every pair of a frame;
//  * what is always positive, |l|^2 and the rest of eps^2, comes in under a fused
//    product with y0, whose low bits differ from pair to pair;
//  * the second-order term of corr (3/8 e^2, about 2^-47) is added to e, and not
//    to 1/2, whose grid would swallow it.
template <class V>
__device__ __forceinline__ void inv_dist(const V s[3], const V l2[3], V e2h, V e2l, V B, V& y0, V& ny0, V& corr) {
    y0 = vrsqrt(B);
    ny0 = vneg(y0);
    V h = B;
    const V r0 = square_step(s[0], h), r1 = square_step(s[1], h), r2 = square_step(s[2], h);
    const V h4 = vadd(h, e2h);
    const V p = vadd(e2h, vsub(h, h4));
    const V rest = vadd(vadd(r0, r1), vadd(r2, vfma(splat<V>(-2.f), B, h4)));
    const V low = vadd(rest, vfma(s[2], l2[2], vfma(s[1], l2[1], vfma(s[0], l2[0], p))));
    const V ll = vfma(l2[0], l2[0], vfma(l2[1], l2[1], vmul(l2[2], l2[2])));
    const V least = vfma(splat<V>(0.25f), ll, e2l);  // B + low + least = r^2 + eps^2
    const V nz = vmul(B, ny0);
    const V v = vfma(low, y0, vfma(least, y0, vfma(B, y0, nz)));
    const V e = vfma(v, ny0, vfma(nz, y0, splat<V>(1.f)));
    corr = vmul(vmul(splat<V>(0.5f), y0), vfma(vmul(splat<V>(0.75f), e), e, e));
}

// ---------------------------------------------------------------------------
// Pairs the frame cannot resolve
// ---------------------------------------------------------------------------

__device__ __forceinline__ double pair_phi(double dx, double dy, double dz, double eps2, double spline_h) {
    // -potential of a unit-mass pair
    if (spline_h > 0.0) {
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        return -spline_phi_d(r / spline_h) / spline_h;
    }
    return rsqrt(dx * dx + dy * dy + dz * dz + eps2);
}

// The sources [jf, j_end) after target i, in FP64: of a frame whose numbers FP32
// does not hold, or whose sum is a large part of the energy.
__device__ __noinline__ double frame_f64(const float4* __restrict__ pos, const float4* __restrict__ plo, float4 th,
                                         float4 tl, long long i, long long jf, long long j_end, double eps2,
                                         double spline_h) {
    const double x = (double)th.x + (double)tl.x, y = (double)th.y + (double)tl.y, z = (double)th.z + (double)tl.z;
    double sum = 0.0;
    for (long long j = jf > i ? jf : i + 1; j < j_end; ++j) {
        const float4 q = pos[j];
        const float4 l = plo ? plo[j] : make_float4(0.f, 0.f, 0.f, 0.f);
        sum += (double)q.w * pair_phi(((double)q.x + (double)l.x) - x, ((double)q.y + (double)l.y) - y,
                                      ((double)q.z + (double)l.z) - z, eps2, spline_h);
    }
    return sum;
}

struct PotPair {
    float y, corr;  // double-float 1/r in the frame's unit (0, 0 when `wide` holds the term)
    double wide;    // 1/r or the spline's -phi/h in FP64, in the caller's unit
};

// One pair from the double-float positions themselves: difference of the
// high halves and of the low halves error-free, merged into a normalised
// float pair per axis.
__device__ __noinline__ PotPair refine_pair(float4 th, float4 tl, float4 qh, float4 ql, float sc, float e2h,
                                            float e2l, float kernel2, double eps2, double spline_h) {
    const float a[3] = {qh.x, qh.y, qh.z}, al[3] = {ql.x, ql.y, ql.z};
    const float b[3] = {th.x, th.y, th.z}, bl[3] = {tl.x, tl.y, tl.z};
    float s[3], l2[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float d, de, q, qe, u, ue;
        sum2(a[k], -b[k], d, de);
        sum2(al[k], -bl[k], q, qe);
        sum2(de, q, u, ue);
        float hi, lo;
        sum2(d, u, hi, lo);
        s[k] = hi * sc;
        l2[k] = 2.f * ((lo + (qe + ue)) * sc);
    }
    const float B = lead_r2(s, e2h);
    PotPair r = {0.f, 0.f, 0.0};
    // FP32 resolves the pair: neither inside the spline's kernel nor near the
    // ends of its range (a NaN fails both)
    if (B >= kernel2 && B >= 1e-20f && B <= 16.f) {
        float ny;
        inv_dist(s, l2, e2h, e2l, B, r.y, ny, r.corr);
        return r;
    }
    const double dx = ((double)qh.x + (double)ql.x) - ((double)th.x + (double)tl.x);
    const double dy = ((double)qh.y + (double)ql.y) - ((double)th.y + (double)tl.y);
    const double dz = ((double)qh.z + (double)ql.z) - ((double)th.z + (double)tl.z);
    r.wide = pair_phi(dx, dy, dz, eps2, spline_h);
    return r;
}

// ---------------------------------------------------------------------------
// Double-float kernel
// ---------------------------------------------------------------------------

struct __align__(16) PotStage {
    float x1[3][kPotThreads];  // source coordinates in the frame: grid part
    float x2[3][kPotThreads];  //   and twice the rest
    float m[kPotThreads];      // masses, the frame's largest in [1, 2)
    double unit[kPotThreads / kPotSub];        // what a sum in the frame's units is worth (0: summed in FP64)
    float sc[kPotThreads / kPotSub], e2h[kPotThreads / kPotSub], e2l[kPotThreads / kPotSub],
        near2[kPotThreads / kPotSub], kernel2[kPotThreads / kPotSub];
};

// x - c for a double-float x, as a normalised float pair.
__device__ __forceinline__ void rel_coord(float xh, float xl, float c, float& yh, float& yl) {
    float d, e;
    sum2(xh, -c, d, e);
    const float u = e + xl;
    yh = d + u;
    yl = u - (yh - d);
}

// y scaled by sc, split at the grid 2^-22 (|y sc| < 1); x2 is twice the rest.
__device__ __forceinline__ void grid_split(float yh, float yl, float sc, float& x1, float& x2) {
    x1 = __fadd_rn(__fmaf_rn(yh, sc, 3.f), -3.f);
    x2 = 2.f * __fmaf_rn(yl, sc, __fmaf_rn(yh, sc, -x1));
}

// Double total of a block (thread 0).
__device__ __forceinline__ double pot_block_sum(double v) {
    __shared__ double sh[kPotThreads / 32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int k = 0; k < kPotThreads / 32; ++k) t += sh[k];
    return t;
}

// Block (I, c): targets of tile I against sources [128 I + c chunk, + chunk),
// pairs i < j.  FP32-pipe bound: 54 operations per pair, two sources per
// packed instruction.  partial[c gridDim.x + I] (0 past the end).
template <bool SPLIT>
__global__ void __launch_bounds__(kPotThreads, 5) potential_df_kernel(long long n, const float4* __restrict__ pos,
                                                                      const float4* __restrict__ plo, double eps2,
                                                                      double spline_h, double large, long long chunk,
                                                                      double* __restrict__ partial) {
    __shared__ PotStage sm;
    __shared__ unsigned s_rho;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const long long i0 = blockIdx.x * (long long)kPotThreads;
    const long long j_begin = i0 + blockIdx.y * chunk;
    double* out = partial + (blockIdx.y * (long long)gridDim.x + blockIdx.x);
    if (j_begin >= n) {
        if (tid == 0) *out = 0.0;
        return;
    }
    const long long j_end = j_begin + chunk < n ? j_begin + chunk : n;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const long long i = i0 + tid;
    const bool have = i < n;
    const float4 th = have ? pos[i] : zero;
    const float4 tl = (SPLIT && have) ? plo[i] : zero;
    const float4 c = pos[i0 + kPotThreads / 2 < n ? i0 + kPotThreads / 2 : n - 1];
    float th_[3] = {0.f, 0.f, 0.f}, tl_[3] = {0.f, 0.f, 0.f};
    if (have) {
        rel_coord(th.x, tl.x, c.x, th_[0], tl_[0]);
        rel_coord(th.y, tl.y, c.y, th_[1], tl_[1]);
        rel_coord(th.z, tl.z, c.z, th_[2], tl_[2]);
    }
    if (tid == 0) s_rho = __float_as_uint(fmaxf(1e-30f, (float)sqrt(spline_h > 0.0 ? 0.0 : eps2)));
    __syncthreads();
    {  // largest target coordinate (float bits of |y| order like the value; a NaN sorts above)
        const unsigned a = max(max(__float_as_uint(fabsf(th_[0])), __float_as_uint(fabsf(th_[1]))),
                               __float_as_uint(fabsf(th_[2])));
        const unsigned r = __reduce_max_sync(0xffffffffu, a);
        if (lane == 0) atomicMax(&s_rho, r);
    }
    double acc = 0.0;
    for (long long t = j_begin; t < j_end; t += kPotThreads) {
        __syncthreads();
        {  // stage: warp w fills frame w
            const long long j = t + tid;
            const bool in = j < j_end;
            const float4 q = in ? pos[j] : zero;
            const float4 ql = (SPLIT && in) ? plo[j] : zero;
            float yh[3] = {0.f, 0.f, 0.f}, yl[3] = {0.f, 0.f, 0.f};
            if (in) {
                rel_coord(q.x, ql.x, c.x, yh[0], yl[0]);
                rel_coord(q.y, ql.y, c.y, yh[1], yl[1]);
                rel_coord(q.z, ql.z, c.z, yh[2], yl[2]);
            }
            unsigned a = max(max(__float_as_uint(fabsf(yh[0])), __float_as_uint(fabsf(yh[1]))),
                             __float_as_uint(fabsf(yh[2])));
            a = max(__reduce_max_sync(0xffffffffu, a), s_rho);
            // 2^-ex with E = 2^ex [1/2, 1).  A frame is summed in FP64 if E is
            // outside FP32's comfortable range (or a NaN), or if a source is
            // lighter than 2^-63 of the heaviest: its low parts (2^-46 of its
            // term) would not be normal numbers.
            const unsigned eb = a >> 23;
            const unsigned mb = __float_as_uint(fabsf(q.w));
            const unsigned heaviest = __reduce_max_sync(0xffffffffu, mb) >> 23;
            const unsigned lightest = __reduce_min_sync(0xffffffffu, mb ? mb : 0xffffffffu) >> 23;
            const bool fits = eb >= 8u && eb <= 245u && lightest > 0u && lightest + 63u >= heaviest && heaviest < 255u;
            const float sc = fits ? __uint_as_float((253u - eb) << 23) : 1.f;
            const double scd = (double)sc, e2 = spline_h > 0.0 ? 0.0 : eps2 * scd * scd;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                float x1, x2;
                grid_split(yh[k], yl[k], sc, x1, x2);
                sm.x1[k][tid] = x1;
                sm.x2[k][tid] = x2;
            }
            // in units of 2^(heaviest - 127)
            sm.m[tid] = (float)((double)q.w * __longlong_as_double((long long)(1150u - heaviest) << 52));
            if (lane == 0) {
                sm.unit[w] = fits ? __longlong_as_double((long long)(896u + heaviest) << 52) * scd : 0.0;
                // rounded up, so that every pair inside the kernel is caught
                const float k2 = spline_h > 0.0 ? (float)(4.00001 * (spline_h * scd) * (spline_h * scd)) : 0.f;
                sm.sc[w] = sc;
                const float e2h = (float)__dadd_rn(__dadd_rn(e2, 384.0), -384.0);  // on the grid 2^-44
                sm.e2h[w] = e2h;
                sm.e2l[w] = (float)(e2 - (double)e2h);
                sm.kernel2[w] = k2;
                sm.near2[w] = fmaxf(kPotNear2, k2);
            }
        }
        __syncthreads();
        const int frames = (int)((min((long long)kPotThreads, j_end - t) + kPotSub - 1) / kPotSub);
        for (int f = 0; f < frames; ++f) {
            const long long jf = t + f * kPotSub;
            const double unit = sm.unit[f];
            if (unit == 0.0) {
                if (have) acc += frame_f64(pos, SPLIT ? plo : nullptr, th, tl, i, jf, min(jf + kPotSub, j_end), eps2, spline_h);
                continue;
            }
            const float sc = sm.sc[f], near2 = sm.near2[f];
            const float2 e2h = splat<float2>(sm.e2h[f]), e2l = splat<float2>(sm.e2l[f]);
            float2 n1[3], n2[3];  // the target, negated
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                float x1, x2;
                grid_split(th_[k], tl_[k], sc, x1, x2);
                n1[k] = splat<float2>(-x1);
                n2[k] = splat<float2>(-x2);
            }
            const double before = acc;
            const bool diag = jf < i0 + kPotThreads;  // sources at or before some target
            float2 A = make_float2(0.f, 0.f), R = A;
            for (int k4 = 0; k4 < kPotSub; k4 += 4) {
                float4 q1[3], q2[3];
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    q1[x] = *reinterpret_cast<const float4*>(&sm.x1[x][f * kPotSub + k4]);
                    q2[x] = *reinterpret_cast<const float4*>(&sm.x2[x][f * kPotSub + k4]);
                }
                const float4 qm = *reinterpret_cast<const float4*>(&sm.m[f * kPotSub + k4]);
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const long long j0 = jf + k4 + 2 * half;
                    float2 s[3], l2[3], m = half ? make_float2(qm.z, qm.w) : make_float2(qm.x, qm.y);
#pragma unroll
                    for (int x = 0; x < 3; ++x) {
                        s[x] = vadd(half ? make_float2(q1[x].z, q1[x].w) : make_float2(q1[x].x, q1[x].y), n1[x]);
                        l2[x] = vadd(half ? make_float2(q2[x].z, q2[x].w) : make_float2(q2[x].x, q2[x].y), n2[x]);
                    }
                    if (diag) {
                        if (j0 <= i) m.x = 0.f;
                        if (j0 + 1 <= i) m.y = 0.f;
                    }
                    const float2 B = lead_r2(s, e2h);
                    float2 y0, ny0, corr;
                    inv_dist(s, l2, e2h, e2l, B, y0, ny0, corr);
                    if (!(fminf(B.x, B.y) >= near2)) {
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            if ((u ? B.y : B.x) >= near2) continue;
                            const long long j = j0 + u;
                            float y = 0.f, co = 0.f;
                            if (have && j > i && j < j_end) {
                                const float4 qh = pos[j];
                                const PotPair p = refine_pair(th, tl, qh, SPLIT ? plo[j] : zero, sc, e2h.x, e2l.x,
                                                              sm.kernel2[f], eps2, spline_h);
                                y = p.y;
                                co = p.corr;
                                acc += (double)qh.w * p.wide;
                            }
                            if (u) {
                                y0.y = y;
                                ny0.y = -y;
                                corr.y = co;
                            } else {
                                y0.x = y;
                                ny0.x = -y;
                                corr.x = co;
                            }
                        }
                    }
                    const float2 ph = vmul(m, y0);
                    const float2 npe = vfma(m, ny0, ph);  // what ph rounded off m y0, negated
                    float2 S, er;
                    sum2(A, ph, S, er);
                    A = S;
                    R = vadd(R, vsub(vfma(m, corr, er), npe));
                }
            }
            float S, er;
            sum2(A.x, A.y, S, er);
            const double high = (double)S * unit;
            if (high * (double)th.w > large)
                acc = before + frame_f64(pos, SPLIT ? plo : nullptr, th, tl, i, jf, min(jf + kPotSub, j_end), eps2, spline_h);
            else
                acc = fma((double)(er + (R.x + R.y)), unit, acc + high);
        }
    }
    const double t = pot_block_sum(have ? -(double)th.w * acc : 0.0);
    if (tid == 0) *out = t;
}

// ---------------------------------------------------------------------------
// FP64 kernel (small n): the same blocks, FP64-pipe bound, so the triangle is
// cut into blocks of 32 sources to spread over the SMs.
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(kPotThreads) potential_f64_kernel(long long n, const float4* __restrict__ pos,
                                                                    const float4* __restrict__ plo, double eps2,
                                                                    double spline_h, long long chunk,
                                                                    double* __restrict__ partial) {
    __shared__ double sx[kPotSub], sy[kPotSub], sz[kPotSub], smm[kPotSub];
    const int tid = threadIdx.x;
    const long long i0 = blockIdx.x * (long long)kPotThreads;
    const long long j_begin = i0 + blockIdx.y * chunk;
    double* out = partial + (blockIdx.y * (long long)gridDim.x + blockIdx.x);
    if (j_begin >= n) {
        if (tid == 0) *out = 0.0;
        return;
    }
    const long long j_end = j_begin + chunk < n ? j_begin + chunk : n;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const long long i = i0 + tid;
    const float4 p = i < n ? pos[i] : zero;
    const float4 l = (plo && i < n) ? plo[i] : zero;
    const double xi = (double)p.x + (double)l.x, yi = (double)p.y + (double)l.y, zi = (double)p.z + (double)l.z;
    double acc = 0.0;
    for (long long t = j_begin; t < j_end; t += kPotSub) {
        __syncthreads();
        if (tid < kPotSub && t + tid < j_end) {
            const float4 q = pos[t + tid];
            const float4 ql = plo ? plo[t + tid] : zero;
            sx[tid] = (double)q.x + (double)ql.x;
            sy[tid] = (double)q.y + (double)ql.y;
            sz[tid] = (double)q.z + (double)ql.z;
            smm[tid] = q.w;
        }
        __syncthreads();
        const int kmax = (int)min((long long)kPotSub, j_end - t);
#pragma unroll 4
        for (int k = 0; k < kmax; ++k)
            if (t + k > i) acc += smm[k] * pair_phi(sx[k] - xi, sy[k] - yi, sz[k] - zi, eps2, spline_h);
    }
    const double t = pot_block_sum(i < n ? -(double)p.w * acc : 0.0);
    if (tid == 0) *out = t;
}

// A target's sum over 32 sources above this is formed in FP64: 2^-12 of a lower
// bound of the energy, so that what is left are at least 2^12 sums of independent
// errors, the worst of 2^-42 each (rms), and their mean is good to 2^-48.  Sums that
// large are few: the bound is about half of the energy of a Plummer sphere or a
// galaxy, and 32 sources hold 2^-18 of it on average at n = 4,096.  The bound:
// 1/sqrt(r^2 + eps^2) is convex in r^2, so its mean over pairs is at least its
// value at their mean r^2, which `inertia`, the sum of m r^2 about the centre of
// mass, gives times the mass; the spline's potential is nowhere weaker than
// 1/sqrt(r^2 + h^2).  With masses of both signs (pairs < 0, diag_pass2_kernel) no
// bound holds: NaN, and every pair is FP64.
double potential_large(double mass, double pairs, double inertia, double eps2) {
    if (!(pairs >= 0.0)) return std::nan("");
    return pairs > 0.0 ? pairs / std::sqrt(mass * inertia / pairs + eps2) / 4096.0 : 0.0;
}

void launch_potential(long long n, const Particles& P, bool split, double eps2, double spline_h, double large,
                      double* partial, cudaStream_t s) {
    const dim3 grid((unsigned)pot_tiles(n), (unsigned)pot_chunks(n));
    const long long chunk = potential_chunk(n);
    if (n < kPotDfMin || !(large >= 0.0))
        potential_f64_kernel<<<grid, kPotThreads, 0, s>>>(n, P.pos, split ? P.plo : nullptr, eps2, spline_h, chunk,
                                                          partial);
    else if (split)
        potential_df_kernel<true><<<grid, kPotThreads, 0, s>>>(n, P.pos, P.plo, eps2, spline_h, large, chunk, partial);
    else
        potential_df_kernel<false><<<grid, kPotThreads, 0, s>>>(n, P.pos, nullptr, eps2, spline_h, large, chunk,
                                                                partial);
}

}  // namespace ngrav
