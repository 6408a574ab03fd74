#pragma once
// Persistent chain kernel: the ACHR sampling hot loop on sm_103a.
// (Template; instantiated for each block-size / elements-per-thread pair in
// achr_chain_cfg_*.cu, dispatched by achr_chain_launch.cu.)
//
// Replaces the reference's chain driver and step loop (ACHRcu/ACHRCuda.cu:
// stepPointProgress :361-385, createPoint :297-359, fillrandPoint :251-289,
// advNextStep :242-249, findMaxAbs :232-240, reprojectPoint(2) :208-230,
// correctBounds :193-206), which run one chain per GPU thread and launch child
// grids from the device for every step.
//
// Design (one CTA per chain, persistent over chains):
//   * The chain's point x and centre accumulator A = (W + t) c live in shared
//     memory for all T steps.  The warmup column w_r is read from HBM/L2
//     straight into the registers that hold the direction: each thread owns
//     pairs of neighbouring reactions (16-byte loads), and as soon as the step
//     has used a direction pair it requests the next step's column there.  A
//     chain needs two vectors of shared memory, not the three that a staged
//     column takes: an SM holds 4 chains of 3072 reactions, 2 of 6656.
//   * GB300's FP64 pipe takes one warp instruction per 19 clocks and SM (64
//     clocks for one warp alone), 72x less than FP32, and FP64 compares cost
//     as much as FMAs.  Per element and accepted step the kernel spends exactly
//     three FP64 pipe instructions (d = w - A/(W+t), x += s d, A += x).  The
//     norm is summed in FP32 (it only feeds tolerance tests, which carry
//     margins and fall back to FP64 when a margin is not enough); the ratio
//     test brackets every ratio in FP32 with rigorous error bounds and
//     evaluates in FP64 only the coordinates whose bracket can hold the
//     minimum; clipping and the min/max reductions compare FP64 values as
//     integers (order-preserving keys), and the quotients that decide the step
//     are divided with integer arithmetic (div_rn).
//   * The FP32 image of x that the clip test forms stays in registers for the
//     next step's brackets (where registers allow: chain_keeps_x32).
//   * The brackets are formed in the pass that forms d, before the block knows
//     ||d||, so they fill the FP64 latency and one block reduction serves the
//     norm and the bracket minima.  The few contenders meet in shared memory,
//     and one warp computes the step length (three barriers per accepted step).
//   * Per-step scalars (warmup index, step uniform, 1/(W+t)) come from a
//     shared-memory table that the CTA refills once every kTbl steps.
//   * The element loops are unrolled over compile-time BD x EPT with arrays
//     padded to that length, so no loop carries a bounds test.
//   * Reductions are warp shuffles plus one shared-memory exchange in a fixed
//     order, so a launch is bitwise repeatable; a one-warp CTA skips the
//     exchange.
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "achr_div.cuh"
#include "achr_float.cuh"
#include "achr_internal.h"
#include "achr_rng.cuh"

namespace achr {
namespace {

constexpr float kErrK = 2.384185791015625e-07f;        // 2^-22: bound on truncation + FP32 rounding
constexpr float kTiny = 2.350988701644575e-38f;        // 2^-125: absolute error of flushed tiny values
constexpr float kUp = 1.0f + 9.5367431640625e-07f;     // 1 + 2^-20
constexpr float kDn = 1.0f - 9.5367431640625e-07f;     // 1 - 2^-20
constexpr float kQUp = 1.0f + 1.9073486328125e-06f;    // 1 + 2^-19: relative error of a bracketed ratio
constexpr float kQDn = 1.0f - 1.9073486328125e-06f;
constexpr float kErrX = 2.4080276489257812e-07f;       // 2^-22 (1 + 2^-6.7): kErrK with room for kQUp and its rounding
constexpr float kAdUp = 1.0f + 4.76837158203125e-07f;  // 1 + 2^-21
constexpr float kNormUp = 1.0f + 1e-5f;                // FP32 norm relative error margin
constexpr float kNormDn = 1.0f - 1e-5f;
constexpr float kDMin = 7.888609052210118e-31f;        // 2^-100: smallest |d| the brackets tell apart
constexpr float kDCert = 1.5777218104420236e-30f;      // 2^-99: no smaller |d| is a certain candidate
constexpr unsigned long long kWaitNs = 2000000000ull;  // bounded mbarrier wait: 2 s
constexpr unsigned long long kInfBits = 0x7FF0000000000000ull;

// FP64 -> FP32 for the hot loops, in six integer operations: the magnitude is
// clamped to [2^LO_EXP, 2^128 (1 - 2^-20)) in its FP64 form (three spare low
// bits of a clamped value are below the error bound), then the exponent is
// re-biased with one addition.  |v - f| <= 2^-23 |f| inside the range; below
// it f is +-2^LO_EXP (1 + 2^-20) at most, above it the largest magnitude.
template <int LO_EXP>
__device__ __forceinline__ float f64_to_f32_clamped(double v) {
    const unsigned hi = (unsigned)__double2hiint(v);
    const unsigned lo = (unsigned)__double2loint(v);
    constexpr unsigned kLo = (unsigned)(1023 + LO_EXP) << 20, kHi = 0x47EFFFFFu;
    const unsigned h = min(max(hi & 0x7FFFFFFFu, kLo), kHi);
    const unsigned mag = __funnelshift_l(lo, h, 3) + 0x40000000u;  // - (896 << 23)
    return __uint_as_float((hi & 0x80000000u) | mag);
}
// x: clamped at 2^-126 (kTiny covers it); d: clamped at kDMin.
__device__ __forceinline__ float x_to_f32(double v) { return f64_to_f32_clamped<-126>(v); }
__device__ __forceinline__ float d_to_f32(double v) { return f64_to_f32_clamped<-100>(v); }

// |v| and its bit pattern through integer operations (fabs on a double can be
// issued to the FP64 pipe).
__device__ __forceinline__ unsigned long long abs_bits(double v) {
    return (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull;
}
__device__ __forceinline__ double abs_int(double v) { return __longlong_as_double((long long)abs_bits(v)); }
__device__ __forceinline__ bool positive_int(double v) {  // v > 0 for non-NaN v
    const long long b = __double_as_longlong(v);
    return b > 0;
}
// v > t for t >= 0 and non-NaN v (an FP64 compare would go to the FP64 pipe).
__device__ __forceinline__ bool above_int(double v, double t) {
    return __double_as_longlong(v) > __double_as_longlong(t);
}

// r[k] for a run-time k without indexing the register array dynamically: a
// tree of selects on the bits of k.
template <int N>
__device__ __forceinline__ double pick(const double (&r)[N], int k) {
    if constexpr (N == 1) {
        return r[0];
    } else {
        double h[(N + 1) / 2];
#pragma unroll
        for (int j = 0; j < N / 2; ++j) h[j] = (k & 1) ? r[2 * j + 1] : r[2 * j];
        if (N & 1) h[N / 2] = r[N - 1];
        return pick(h, k >> 1);
    }
}

// (lb, ub) of one reaction.  A volatile load, so that the compiler keeps it
// (and the FP64 work that depends on it) inside the rarely taken branches.
__device__ __forceinline__ double2 ld_lbub(const double2 *p) {
    double2 v;
    asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}

// (lb, ub) of one reaction in FP64: from the FP32 image when the host found
// every bound finite and exact there (the image is in L1; the FP64 bounds come
// from L2, several hundred clocks in the middle of a step).
__device__ __forceinline__ double2 exact_bounds(const ChainArgs &a, int i);

// A pair of a warmup column: 16 bytes, past L1 (a column is read once per
// step; L1 keeps the FP32 bounds, which every step reads twice).  Volatile, so
// that the request stays where it is issued, a whole phase ahead of its use.
__device__ __forceinline__ double2 ld_column(const double2 *p) {
    double2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}

// FP32 test that x (as its truncation x32) lies strictly inside (lb, ub):
// true only when the bracket arithmetic proves it; false means "test exactly".
__device__ __forceinline__ bool surely_inside(float x32, float lb, float ub, float berr) {
    const float ex = fmaf(fabsf(x32), kErrK, kTiny + berr);
    return fminf(x32 - lb, ub - x32) > ex;
}

__device__ __forceinline__ unsigned smem_addr(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wait for the phase with the given parity to complete, giving up after limit_ns.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, unsigned parity,
                                                  unsigned long long limit_ns = kWaitNs) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (;;) {
        if (mbar_try_wait(bar, parity)) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float sqrt_approx(float x) {  // within 2^-22; the norm's margin is 1e-5
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

template <class T>
__device__ __forceinline__ T umin(T a, T b) {
    return a < b ? a : b;
}
template <class T>
__device__ __forceinline__ T umax(T a, T b) {
    return a > b ? a : b;
}

// Warp minima with the single-instruction integer reductions (redux.sync)
// instead of five shuffle rounds: floats through an order-preserving key,
// 64-bit keys as (high word, then low word among the lanes holding the high
// minimum).
__device__ __forceinline__ unsigned f32_key(float f) {
    const unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_f32(unsigned k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
__device__ __forceinline__ float warp_min_f32(float v) {
    return key_f32(__reduce_min_sync(0xffffffffu, f32_key(v)));
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
    const unsigned hi = (unsigned)(v >> 32);
    const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? (unsigned)v : 0u);
    return ((unsigned long long)mhi << 32) | mlo;
}
__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v) {
    const unsigned hi = (unsigned)(v >> 32);
    const unsigned mhi = __reduce_min_sync(0xffffffffu, hi);
    const unsigned mlo = __reduce_min_sync(0xffffffffu, hi == mhi ? (unsigned)v : 0xffffffffu);
    return ((unsigned long long)mhi << 32) | mlo;
}

// CTA barriers; a one-warp CTA needs only its warp's.
template <int BD>
__device__ __forceinline__ void cta_sync() {
    if (BD == 32) __syncwarp();
    else __syncthreads();
}
template <int BD>
__device__ __forceinline__ bool cta_any(bool p) {
    if (BD != 32) return __syncthreads_or(p ? 1 : 0) != 0;
    const bool any = __any_sync(0xffffffffu, p) != 0;
    __syncwarp();
    return any;
}

// Shared-memory exchange slots, two sets selected by attempt parity so that
// consecutive attempts never overwrite slots another warp may still read.  The
// per-warp values are read back four at a time.
template <int NW>
struct alignas(16) RedSlots {
    static constexpr int NW4 = (NW + 3) / 4 * 4;
    float sum1[NW4], uh[NW4], ul[NW4];
    unsigned long long kh, kl;  // smallest exact ratios (bits) of the attempt's contenders
    double step;                // the step length over ||d||
    unsigned flags;             // 1: a valid contender, 2: one needs the FP64 norm
    unsigned pad;
    unsigned long long max4[NW];
    double sum5[NW];
    __device__ void clear() {
        kh = kl = kInfBits;
        flags = 0;
    }
};

// Sum of the warps' values in order / their minimum.
template <int NW>
__device__ __forceinline__ float slots_sum(const float *v) {
    float s = 0.0f;
#pragma unroll
    for (int w = 0; w < NW; w += 4) {
        const float4 x = *reinterpret_cast<const float4 *>(v + w);
        s += x.x;
        if (w + 1 < NW) s += x.y;
        if (w + 2 < NW) s += x.z;
        if (w + 3 < NW) s += x.w;
    }
    return s;
}
template <int NW>
__device__ __forceinline__ float slots_min(const float *v) {
    float m = INFINITY;
#pragma unroll
    for (int w = 0; w < NW; w += 4) {
        const float4 x = *reinterpret_cast<const float4 *>(v + w);
        m = fminf(m, x.x);
        if (w + 1 < NW) m = fminf(m, x.y);
        if (w + 2 < NW) m = fminf(m, x.z);
        if (w + 3 < NW) m = fminf(m, x.w);
    }
    return m;
}

struct StepEntry {
    double U;      // step uniform of attempt 0
    double inv;    // 1 / (W + t + centre_offset)
    unsigned idx;  // warmup index of attempt 0
    unsigned pad;
};

// ---- ratio-test brackets
// FP32 bracket of one coordinate's two ratios (reference fillrandPoint,
// ACHRCuda.cu:266-281: a coordinate is a candidate when distUb > dTol,
// distLb > dTol and |u_i| > uTol).  With r = 1 / d the ratios are
// (bh - x) r and (x - bl) r, bh the bound the step d moves towards and bl the
// other one, so the sign of d enters as one select per bound.
//   live: not certainly a non-candidate (its |d| may exceed the threshold)
//   lo_h, lo_l: lower ends; of a coordinate at a bound (within the FP32
//        error) they are not positive, so it is looked at exactly
//   ok: certainly a candidate; only then do the upper ends count
// e0 = (kTiny + bound error + d_tol) rounded up, so lo > 0 implies dist > d_tol.
struct Bracket {
    float lo_h, lo_l, up_h, up_l;
    bool live, ok;
};
__device__ __forceinline__ Bracket bracket(float x, float d, float lb, float ub, float e0, float uthr_hi,
                                           float uthr_lo) {
    Bracket B;
    const float ad = fabsf(d);
    const bool pos = d > 0.0f;
    const float bh = pos ? ub : lb, bl = pos ? lb : ub;
    const float r = rcp_approx(d);
    const float qh = (bh - x) * r, ql = (x - bl) * r;
    const float g = fmaf(fabsf(x), kErrX, e0) * fabsf(r);
    B.lo_h = fmaf(qh, kQDn, -g);
    B.lo_l = fmaf(ql, kQDn, -g);
    B.up_h = fmaf(qh, kQUp, g);
    B.up_l = fmaf(ql, kQUp, g);
    B.live = !(ad * kAdUp < uthr_lo);
    B.ok = B.lo_h > 0.0f && B.lo_l > 0.0f && ad > uthr_hi;
    return B;
}

// Calls f(row, (S x)_row) for the rows thread tid owns: with the sliced-ELL
// copy of S (32-row groups, slot-major, so each warp's loads of one nonzero
// slot are one coalesced segment) lane l of warp w has row l of groups w, w +
// BD/32, ...; without it (caller-owned models) rows tid, tid + BD, ... of the
// CSR are read directly.  Both visit a row's nonzeros in the same order, so
// the sums are bitwise equal (the ELL padding adds 0 * x_0).
//
// The structure comes from L2 and a row is a chain of dependent FP64
// instructions, so both latencies are shared by two groups at a time: their
// next kSlotLoads slots are requested before any is used, and the group offsets
// are loaded once for all of a warp's groups.
constexpr int kSlotLoads = 4;

template <int BD, class F>
__device__ __forceinline__ void residual_each(const ChainArgs &a, const double *xs, int tid, F &&f) {
    if (a.sell_off) {
        constexpr int NW = BD / 32;
        const int lane = tid & 31, warp = tid >> 5;
#pragma unroll 1
        for (int g0 = warp; g0 < a.sell_groups; g0 += 32 * NW) {
            const int mine = g0 + lane * NW;
            const int off0 = mine < a.sell_groups ? __ldg(a.sell_off + mine) : 0;
            const int off1 = mine < a.sell_groups ? __ldg(a.sell_off + mine + 1) : 0;
            const int cnt = min(32, (a.sell_groups - g0 + NW - 1) / NW);
#pragma unroll 1
            for (int j = 0; j < cnt; j += 2) {
                // the second group of an odd count is the first again, not used
                const bool two = j + 1 < cnt;
                int b0 = __shfl_sync(0xffffffffu, off0, j), b1 = __shfl_sync(0xffffffffu, off0, two ? j + 1 : j);
                const int n0 = (__shfl_sync(0xffffffffu, off1, j) - b0) >> 5;
                const int n1 = two ? (__shfl_sync(0xffffffffu, off1, j + 1) - b1) >> 5 : 0;
                if (n0 == 0) b0 = b1;  // an empty group may start at the array's end: read the other's entries
                if (n1 == 0) b1 = b0;
                double acc0 = 0.0, acc1 = 0.0;
#pragma unroll 1
                for (int t = 0; t < max(n0, n1); t += kSlotLoads) {
                    int c0[kSlotLoads], c1[kSlotLoads];
                    double v0[kSlotLoads], v1[kSlotLoads];
#pragma unroll
                    for (int u = 0; u < kSlotLoads; ++u) {  // past a row: its last slot again, not used
                        const int o0 = b0 + lane + (max(min(t + u, n0 - 1), 0) << 5);
                        const int o1 = b1 + lane + (max(min(t + u, n1 - 1), 0) << 5);
                        c0[u] = __ldg(a.sell_col + o0);
                        c1[u] = __ldg(a.sell_col + o1);
                        v0[u] = __ldg(a.sell_val + o0);
                        v1[u] = __ldg(a.sell_val + o1);
                    }
#pragma unroll
                    for (int u = 0; u < kSlotLoads; ++u) {  // (lengths are the warp's: uniform branches)
                        if (t + u < n0) acc0 = fma(v0[u], xs[c0[u]], acc0);
                        if (t + u < n1) acc1 = fma(v1[u], xs[c1[u]], acc1);
                    }
                }
                f(((g0 + j * NW) << 5) + lane, acc0);
                if (two) f(((g0 + (j + 1) * NW) << 5) + lane, acc1);
            }
        }
    } else {
        for (int row = tid; row < a.m; row += BD) {
            double acc = 0.0;
            const int q1 = __ldg(a.row_ptr + row + 1);
            for (int q = __ldg(a.row_ptr + row); q < q1; ++q) acc = fma(__ldg(a.val + q), xs[__ldg(a.col_idx + q)], acc);
            f(row, acc);
        }
    }
}

// Largest |(S x)_i| over this thread's rows, as the bits of a non-negative
// double (reference findMaxAbs, ACHRCuda.cu:232-240).
template <int BD>
__device__ __forceinline__ unsigned long long residual_max_bits(const ChainArgs &a, const double *xs, int tid) {
    unsigned long long mx = 0;
    residual_each<BD>(a, xs, tid, [&](int, double v) { mx = umax(mx, abs_bits(v)); });
    return mx;
}

// 0.0 from a volatile asm statement.  A computation that starts from it stays
// inside the branch that guards it: without it the compiler may compute the
// FP64 norm of d (one DFMA per element, which almost no step needs) ahead of
// its branch on every step, as it did in the segmented instantiation (a third
// more FP64 work per step on the pipe that bounds this kernel).
__device__ __forceinline__ double fp64_zero_here() {
    double z;
    asm volatile("mov.b64 %0, 0;" : "=d"(z));
    return z;
}

__device__ __forceinline__ double2 exact_bounds(const ChainArgs &a, int i) {
    if (!a.bound_exact) return ld_lbub(a.lbub + i);
    const float2 b = __ldg(a.bnd + i);
    return make_double2(f32_to_f64_exact(b.x), f32_to_f64_exact(b.y));
}

// The same row sums as residual_max_bits (same rows, same order of terms, so
// the same maximum), each written out for the batched reprojection of
// segmented sampling (chain p, device row order): FP64, and the BF16 split of
// its truncation to FP32 (no FP64 operation).
__device__ __forceinline__ void store_residual_row(const ChainArgs &a, int p, int row, double v) {
    unsigned short h, l;
    split_bf16_bits(f64_to_f32_rz(v), h, l);
    a.seg_Rh[(size_t)p * (size_t)a.kpad + (size_t)row] = h;
    a.seg_Rl[(size_t)p * (size_t)a.kpad + (size_t)row] = l;
    a.seg_rd[(size_t)p * (size_t)a.ld_r + (size_t)row] = v;
}
template <int BD>
__device__ __forceinline__ unsigned long long residual_rows(const ChainArgs &a, const double *xs, int p, int tid) {
    unsigned long long mx = 0;
    residual_each<BD>(a, xs, tid, [&](int row, double v) {
        mx = umax(mx, abs_bits(v));
        if (row < a.m) store_residual_row(a, p, row, v);
    });
    return mx;
}

// ys = N^T x (reference reprojectPoint, ACHRCuda.cu:208-218), eight columns of N
// per warp at a time: their loads are in flight together, and their sums over
// the lanes are formed together, each step halving the columns a lane carries
// (nine FP64 additions for eight columns; one column at a time they were 40,
// which at 95 reactions and 24 columns was 120 of a reprojection's 264 FP64
// instructions).
template <int BD>
__device__ __forceinline__ void null_coordinates(const ChainArgs &a, const double *xs, double *ys, int tid) {
    constexpr int NW = BD / 32;
    const int lane = tid & 31, warp = tid >> 5, n = a.n;
#pragma unroll 1
    for (int j0 = 8 * warp; j0 < a.d; j0 += 8 * NW) {
        const double *Nj = a.N + (size_t)j0 * (size_t)n;
        const int cols = min(8, a.d - j0);
        double acc[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[c] = 0.0;
        for (int i = lane; i < n; i += 32) {
            const double x = xs[i];
            double v[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) v[c] = __ldg(Nj + (size_t)min(c, cols - 1) * (size_t)n + i);
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (c < cols) acc[c] = fma(v[c], x, acc[c]);  // (uniform)
        }
#pragma unroll
        for (int half = 4, o = 16; half; half >>= 1, o >>= 1) {
            const bool upper = lane & o;  // carries the upper half of the columns on
#pragma unroll
            for (int c = 0; c < half; ++c) {
                const double keep = upper ? acc[c + half] : acc[c], send = upper ? acc[c] : acc[c + half];
                acc[c] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 2);
        acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
        const int c = ((lane & 16) ? 4 : 0) + ((lane & 8) ? 2 : 0) + ((lane & 4) ? 1 : 0);
        if (!(lane & 3) && c < cols) ys[j0 + c] = acc[0];
    }
}

// x <- x - S^T z, z = (S S^T)^+ S x: the reference's N (N^T x) written through
// the residual (equal in exact arithmetic).  S x is summed in FP64 over the
// same rows as the check and kept as FP32 hi + lo pairs in rr (m entries
// in the accumulator's place); z = (S S^T)^+ r runs in FP32 (a warp per row of the
// pseudo-inverse, coalesced), whose relative error (~1e-7 times the condition
// number) applies to the correction, not to x, which is at most of the size of
// the residual's preimage; the update x_j -= sum_i S_ij z_i is FP64 (CSC).
template <int BD>
__device__ __forceinline__ void residual_form_reproject(const ChainArgs &a, double *xs, float2 *rr, float *zs,
                                                        int zcap, int tid) {
    constexpr int NW = BD / 32;
    const int lane = tid & 31, warp = tid >> 5;
    const int m = a.m;
    residual_each<BD>(a, xs, tid, [&](int row, double v) {
        if (row < m) {
            const float hi = __double2float_rn(v);
            rr[row] = make_float2(hi, __double2float_rn(v - (double)hi));
        }
    });
    __syncthreads();
    for (int i0 = 0; i0 < m; i0 += zcap) {  // zcap rows of z at a time
        const int rows = min(zcap, m - i0);
        for (int i = i0 + warp; i < i0 + rows; i += NW) {
            const float *Bi = a.pinv32 + (size_t)i * (size_t)m;
            float acc = 0.0f;
            for (int k = lane; k < m; k += 32) {
                const float b = __ldg(Bi + k);
                const float2 r = rr[k];
                acc = fmaf(b, r.x, fmaf(b, r.y, acc));
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0) zs[i - i0] = acc;
        }
        __syncthreads();
        for (int j = tid; j < a.n; j += BD) {
            double dl = 0.0;
            const int q1 = __ldg(a.csc_ptr + j + 1);
            for (int q = __ldg(a.csc_ptr + j); q < q1; ++q) {
                const int i = __ldg(a.csc_row + q) - i0;
                if ((unsigned)i < (unsigned)rows) dl = fma(__ldg(a.csc_val + q), (double)zs[i], dl);
            }
            xs[j] -= dl;
        }
        if (i0 + zcap < m) __syncthreads();  // (read before the next rows take their place)
    }
}

// What a thread keeps of its brackets: the smallest lower and upper ends.
struct Minima {
    float uh = INFINITY, ul = INFINITY, lh = INFINITY, ll = INFINITY;
    __device__ __forceinline__ void add(const Bracket &B) {
        if (B.live) {
            lh = fminf(lh, B.lo_h);
            ll = fminf(ll, B.lo_l);
        }
        if (B.ok) {
            uh = fminf(uh, B.up_h);
            ul = fminf(ul, B.up_l);
        }
    }
};

// The ratio-test quantities phase B2 needs of an attempt.
struct RatioTest {
    float uh, ul, uthr_hi, uthr_lo, e0;
    bool have_norm64;
    double thr64;
    unsigned long long kh, kl;  // smallest exact ratios found (bits)
    int found;                  // 1: a valid contender, 2: one whose candidacy needs the FP64 norm
};

// FP64 evaluation of reaction i as a contender for the max step (side_h) or
// the min step: the candidacy test where the bracket left it open, then the
// quotient.
__device__ __forceinline__ void evaluate(const ChainArgs &a, RatioTest &t, double xi, double dk, int i, float2 b32,
                                         bool side_h) {
    const bool up = side_h == positive_int(dk);  // this ratio's distance: ub - x, else x - lb
    double2 lu;
    if (a.bound_exact) {
        lu.x = lu.y = f32_to_f64_exact(up ? b32.y : b32.x);
    } else {
        lu = ld_lbub(a.lbub + i);
    }
    const double num = (up ? lu.y : xi) - (up ? xi : lu.x);
    // a certain candidate, by the bracket's own bounds (with the norm known)
    const float x32 = x_to_f32(xi), ad = fabsf(d_to_f32(dk));
    bool valid = !a.exact_ratio && ad > fmaxf(t.uthr_hi, kDCert) &&
                 fminf(b32.y - x32, x32 - b32.x) * kQDn > fmaf(fabsf(x32), kErrX, t.e0);
    if (!valid) {  // undecided: full FP64 candidacy test
        if (a.bound_exact) lu = make_double2(f32_to_f64_exact(b32.x), f32_to_f64_exact(b32.y));
        const double oth = (up ? xi : lu.y) - (up ? lu.x : xi);
        bool u_pass;
        if (t.have_norm64) {
            u_pass = abs_bits(dk) > (unsigned long long)__double_as_longlong(t.thr64);
        } else {
            const float ad32 = fabsf(f64_to_f32_rz(dk));
            // inside the FP32 norm's margin: settled with the FP64 norm
            if (!(ad32 > t.uthr_hi) && !(ad32 * kAdUp < t.uthr_lo)) t.found |= 2;
            u_pass = ad32 > t.uthr_hi;
        }
        valid = above_int(num, a.d_tol) && above_int(oth, a.d_tol) && u_pass;
    }
    if (valid) {
        const unsigned long long q = (unsigned long long)__double_as_longlong(div_rn(num, abs_int(dk)));
        if (side_h) t.kh = umin(t.kh, q);
        else t.kl = umin(t.kl, q);
        t.found |= 1;
    }
}

}  // namespace

constexpr int kTbl = 64;  // steps per refill of the step table

// Shared memory of one CTA: xs, As (NP doubles each, see chain_kept_pairs; a reprojection parks the
// accumulator in registers and uses As as its scratch), the step table, two
// reduction slots, then eight statistics counters, the exact-evaluation count
// (two ints), the `never` barrier and the two worst-case words.
template <int BD>
__host__ __device__ constexpr size_t chain_tail_bytes() {
    return sizeof(StepEntry) * kTbl + 2 * sizeof(RedSlots<BD / 32>) + 128;
}
// Pairs of the accumulator a thread keeps in registers instead, the last ones:
// where two vectors in shared memory are just too long for two chains per SM
// (256 x 30), three pairs less make room for the second (7440 reactions, SM
// clocks per chain-step: 23090; one chain per SM, 384 x 20: 26500).
template <int BD, int EPT>
__host__ __device__ constexpr int chain_kept_pairs() {
    return BD == 256 && EPT == 30 ? 3 : 0;
}
// Doubles of the accumulator in shared memory: also the reprojection's scratch,
// which holds the d null-space coordinates or the m residuals.
template <int BD, int EPT>
__host__ __device__ constexpr int chain_acc_doubles() {
    return BD * (EPT - 2 * chain_kept_pairs<BD, EPT>());
}
template <int BD, int EPT>
__host__ __device__ constexpr size_t chain_smem_bytes_cfg() {
    return sizeof(double) * (size_t)(BD * EPT + chain_acc_doubles<BD, EPT>()) + chain_tail_bytes<BD>();
}

// Resident CTAs per SM a configuration is compiled for, with `regs` registers
// per thread: what shared memory and the registers allow.  An SM's registers
// lie in four files of 16384, one per scheduler, and the warps spread over
// them, so the fullest file counts (18 warps allow 96 registers each, 12 allow
// 168).
template <int BD, int EPT>
constexpr int chain_ctas_with(int regs) {
    const int by_smem = (int)(227 * 1024 / (chain_smem_bytes_cfg<BD, EPT>() + 1024));
    const int r = regs < 72 ? 72 : regs > 255 ? 255 : (regs + 7) / 8 * 8;
    const int by_regs = 4 * (16384 / (32 * r)) / (BD / 32);
    const int c = by_smem < by_regs ? by_smem : by_regs;
    return c < 1 ? 1 : c > 32 ? 32 : c;
}
// A thread keeps its direction (2 EPT registers) and, unless that costs a
// resident chain where there are few, the FP32 image of its point (EPT).
template <int BD, int EPT>
constexpr bool chain_keeps_x32() {
    const int kept = chain_ctas_with<BD, EPT>(3 * EPT + 58);
    return kept >= 4 || kept >= chain_ctas_with<BD, EPT>(2 * EPT + 48);
}
template <int BD, int EPT>
constexpr int chain_min_ctas() {
    return chain_ctas_with<BD, EPT>(chain_keeps_x32<BD, EPT>() ? 3 * EPT + 58 : 2 * EPT + 48);
}

template <int BD, int EPT>
__device__ __forceinline__ uint64_t *chain_never(unsigned char *smem_raw) {
    return reinterpret_cast<uint64_t *>(smem_raw + chain_smem_bytes_cfg<BD, EPT>() - 128 + 72);
}

// Entries e = tid, tid + BD, ... < kTbl of the step table for steps s + e below
// `end`: the step's Philox draw (uniform and warmup index) and 1 / (W + t).
template <int BD>
__device__ __forceinline__ void fill_step_table(const ChainArgs &a, StepEntry *tbl, unsigned long long chain, int s,
                                                int end, int tid) {
    for (int e = tid; e < kTbl; e += BD) {
        const int st = s + e;
        if (st < end) {
            const Philox4 pd = step_draw(a.seed, chain, (uint32_t)st, 0u);
            StepEntry en;
            en.U = step_uniform(pd);
            en.inv = 1.0 / (double)(a.W + st + a.centre_offset);
            en.idx = warmup_index(pd, (uint32_t)a.W);
            en.pad = 0;
            tbl[e] = en;
        }
    }
}

// One CTA's share of a launch: chains p_begin, p_begin + p_step, ... below
// p_end of the model `a` describes, then the CTA's statistics into
// a.counters.  Returns true when the launch failed (a bounded wait ran out, or
// a warmup index outside the matrix).
// SEG: segmented launches of the deferred reprojection (a separate
// instantiation, so the plain kernel carries none of its code or registers).
//
// What bounds it: the FP64 pipe (three instructions per reaction and step, one
// warp instruction per 19 clocks and SM), as long as other chains' FP64 work
// fills the latency of a chain's two reductions and its contenders.  So the
// split serves residency: as many chains per SM as two vectors of shared memory
// and the registers allow.  2766 x 3742, two chains per SM: 10.2 K clocks of an
// SM per chain-step (14.0 K with the column staged in shared memory, the
// brackets formed twice and the ratios divided on the FP64 pipe), 7.8 K of them
// the pipe's; a lone chain's step went from 16.4 K to 14.7 K.
template <int BD, int EPT, bool SEG>
__device__ __forceinline__ bool chain_run(const ChainArgs &a, int p_begin, int p_step, int p_end,
                                          unsigned char *smem_raw) {
    static_assert(EPT % 2 == 0, "threads own pairs of reactions");
    constexpr int NP = BD * EPT, KP = EPT / 2;
    constexpr int NW = BD / 32;
    constexpr int KA = KP - chain_kept_pairs<BD, EPT>();  // pairs of the accumulator in shared memory
    constexpr bool KX = chain_keeps_x32<BD, EPT>();
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    double *xs = reinterpret_cast<double *>(smem_raw);
    double *As = xs + NP;
    double2 *xs2 = reinterpret_cast<double2 *>(xs), *As2 = reinterpret_cast<double2 *>(As);
    double *ys = As;  // reprojection scratch (the accumulator waits in registers)
    StepEntry *tbl = reinterpret_cast<StepEntry *>(As + chain_acc_doubles<BD, EPT>());
    RedSlots<NW> *rsb = reinterpret_cast<RedSlots<NW> *>(tbl + kTbl);
    unsigned long long *cnt = reinterpret_cast<unsigned long long *>(rsb + 2);  // CTA statistics, CNT_* slots
    int *exact_count = reinterpret_cast<int *>(cnt + 8);
    uint64_t *never = chain_never<BD, EPT>(smem_raw);  // a barrier nothing arrives on
    // largest residual and bound violation of the CTA's emitted points (bits of non-negative doubles)
    unsigned long long *worst = reinterpret_cast<unsigned long long *>(never + 1);
    // (S S^T)^+ r of the residual-form reprojection (m floats), when enabled
    float *zs = a.z_rows ? reinterpret_cast<float *>(As) + 2 * a.m
                         : reinterpret_cast<float *>(smem_raw + chain_smem_bytes_cfg<BD, EPT>());

    if (tid == 0) {
        *exact_count = 0;
        for (int c = 0; c < 8; ++c) cnt[c] = 0;
        worst[0] = worst[1] = 0;
        rsb[0].clear();
        rsb[1].clear();
    }
    cta_sync<BD>();

    const bool hr = a.hit_and_run != 0;  // directions are the columns themselves (no centre)
    const bool merged = a.merged_ab != 0 && !a.exact_ratio;  // ratio-test brackets formed before ||d|| is known
    const int npair = (a.n + 1) >> 1;
    const int odd = (a.n & 1) ? npair - 1 : -1;  // the pair whose second reaction is padding
    // A warp whose pairs of the last slot (k = KP - 1) all lie in the padding
    // skips that slot: its coordinates stay 0 and its d is 0, so the FP64
    // operations on it would change nothing.
    const bool tail_live = warp * 32 + (KP - 1) * BD < npair;
#define ACHR_PAD_SLOT(k) ((k) == KP - 1 && !tail_live)
// Pair k of the accumulator (k a constant of an unrolled loop).
#define ACHR_ACC_GET(k) ((k) < KA ? As2[tid + (k) * BD] : make_double2(at[(k) < KA ? 0 : 2 * ((k) - KA)], at[(k) < KA ? 0 : 2 * ((k) - KA) + 1]))
#define ACHR_ACC_SET(k, v)                              \
    do {                                                \
        if ((k) < KA) {                                 \
            As2[tid + (k) * BD] = (v);                  \
        } else {                                        \
            at[(k) < KA ? 0 : 2 * ((k) - KA)] = (v).x;     \
            at[(k) < KA ? 0 : 2 * ((k) - KA) + 1] = (v).y; \
        }                                               \
    } while (0)
// Adds v to coordinate i, the thread's k-th of the accumulator (k not a constant).
#define ACHR_ACC_ADD(k, i, v)                                               \
    do {                                                                    \
        if (KA == KP || (k) < 2 * KA) {                                     \
            As[i] += (v);                                                   \
        } else {                                                            \
            _Pragma("unroll") for (int t_ = 0; t_ < 2 * (KP - KA); ++t_)    \
                if ((k) - 2 * KA == t_) at[t_] += (v);                      \
        }                                                                   \
    } while (0)
    const float e0 = (kTiny + a.bound_err + a.dtol_hi) * 1.01f;
    const float4 *bnd2 = reinterpret_cast<const float4 *>(a.bnd);  // (lb, ub, lb, ub) of a pair
    unsigned it = 0;
    bool failed = false;
    // The failure-detection test: a wait on a barrier nothing completes always runs out.
    if (a.wait_never && a.T > 0 && p_begin < p_end)
        failed = !mbar_wait_bounded(never, 0, a.wait_ns ? a.wait_ns : kWaitNs);
    failed = cta_any<BD>(failed);

    // (Scalars that stay constant over a launch are read from the kernel
    // parameters where they are used rather than held in registers.)
    for (int p = p_begin; p < p_end && !failed; p = (int)min((long long)p + p_step, (long long)p_end)) {
#define ACHR_CHAIN_ID (a.chain_offset + (unsigned long long)p)
        // Segmented sampling: the chain's state bits from the earlier launches.
        const unsigned sflags = SEG ? a.seg_flags[p] : 0u;
        double at[KA < KP ? 2 * (KP - KA) : 1];  // the accumulator's last pairs (KA < KP)
        // Point and accumulator: of an earlier launch, of the chain's state after
        // step0 steps (resume), or the centre and its sum.
        const double *x_src = a.c0, *A_src = a.A0;
        long long stride = 1;
        int stored = NP;
        if (sflags & SEG_STARTED) {
            x_src = a.seg_x + (size_t)p * (size_t)a.ld_seg;
            A_src = a.seg_A + (size_t)p * (size_t)a.ld_seg;
            stored = a.n;
        } else if (a.x_in) {
            x_src = a.x_in + p;
            A_src = a.A_in + p;
            stride = a.ld_state;
            stored = a.n;
        }
#pragma unroll
        for (int k = 0; k < KP; ++k) {
            const int i = 2 * (tid + k * BD);
            double2 x2 = make_double2(0.0, 0.0), A2 = x2;
            if (i < stored) {
                x2.x = x_src[(long long)i * stride];
                A2.x = A_src[(long long)i * stride];
            }
            if (i + 1 < stored) {
                x2.y = x_src[(long long)(i + 1) * stride];
                A2.y = A_src[(long long)(i + 1) * stride];
            }
            xs2[tid + k * BD] = x2;
            ACHR_ACC_SET(k, A2);
        }
        int buf_col = -1;  // the warmup column dreg holds (-1: none)
        bool any_accepted = a.x_in != nullptr || (sflags & SEG_ACCEPTED), stuck = false;
        bool seg_pending = false;  // this launch ended the chain after a check step's update
        const bool was_stuck = (sflags & SEG_STUCK) != 0;
        if (was_stuck) stuck = true;  // stopped in an earlier launch: no more steps
        if (sflags & SEG_CORR) {
            // The batched passes' correction of this chain, x <- x - S^T z summed over
            // the passes, held as a double-float pair: two FP64 subtractions per
            // reaction (the FP32 -> FP64 conversions are integer operations).
            cta_sync<BD>();  // this loop is per element, the others per pair
#pragma unroll
            for (int k = 0; k < EPT; ++k) {
                const int i = tid + k * BD;
                if (i < a.n) {
                    const size_t o = (size_t)p * (size_t)a.ld_seg + (size_t)i;
                    xs[i] = (xs[i] - f32_to_f64_exact(a.seg_dxh[o])) - f32_to_f64_exact(a.seg_dxl[o]);
                }
            }
        }
        cta_sync<BD>();
        double dreg[EPT];  // the next step's column, then the step's direction
        float xf[KX ? EPT : 2];  // FP32 image of the point (KX; else formed where it is used)
        if (sflags & SEG_PENDING) {
            // Finish the check step the previous launch ended on (the batched
            // pass has reprojected the point if its residual was above the
            // tolerance): clip, then add the point to the centre accumulator.
            unsigned edge = 0;
#pragma unroll
            for (int k = 0; k < EPT; ++k) {
                const int i = 2 * (tid + (k >> 1) * BD) + (k & 1);
                if (ACHR_PAD_SLOT(k >> 1)) continue;
                const double xv = xs[i];
                const float2 b = __ldg(a.bnd + i);
                if (surely_inside(x_to_f32(xv), b.x, b.y, a.bound_err)) {
                    if (!hr) {
                        if ((k >> 1) < KA) As[i] += xv;
                        else at[(k >> 1) < KA ? 0 : k - 2 * KA] += xv;
                    }
                } else {
                    edge |= 1u << k;
                }
            }
            for (; edge; edge &= edge - 1) {
                const int k = __ffs(edge) - 1, i = 2 * (tid + (k >> 1) * BD) + (k & 1);
                const double xc = clip_exact(xs[i], exact_bounds(a, i));
                xs[i] = xc;
                if (!hr) ACHR_ACC_ADD(k, i, xc);
            }
        }
// Pair k of the point's image.
#define ACHR_X32(k, f0, f1)                        \
    float f0, f1;                                  \
    if (KX) {                                      \
        f0 = xf[KX ? 2 * (k) : 0];                 \
        f1 = xf[KX ? 2 * (k) + 1 : 1];             \
    } else {                                       \
        const double2 xk_ = xs2[tid + (k) * BD];   \
        f0 = x_to_f32(xk_.x);                      \
        f1 = x_to_f32(xk_.y);                      \
    }
        if (KX) {
#pragma unroll
            for (int k = 0; k < KP; ++k) {
                const double2 x2 = xs2[tid + k * BD];
                xf[KX ? 2 * k : 0] = x_to_f32(x2.x);
                xf[KX ? 2 * k + 1 : 1] = x_to_f32(x2.y);
            }
        }
        // The reference checks when the step count is a multiple of the period
        // (ACHRCuda.cu:325); a period of INT_MAX stands for "never".
        int chk = a.check_period == 0x7fffffff ? 1 : a.step0 % a.check_period;
        int tbase = a.step0 - kTbl;
        float t_lo = 0.0f;  // lower end of the merged brackets' candidacy threshold

        for (int s = a.step0; s < (a.step0 + a.T) && !stuck && !failed && !seg_pending; ++s) {
            if (s - tbase >= kTbl) {
                // refill the step table: entry e holds step tbase + e
                tbase = s;
                cta_sync<BD>();
                fill_step_table<BD>(a, tbl, ACHR_CHAIN_ID, s, a.step0 + a.T, tid);
                cta_sync<BD>();
            }
            // this step's table entry (its fields are read where they are used)
            const StepEntry *te = tbl + (s - tbase);
            for (int att = 0;; ++att, ++it) {
                if (att >= a.max_attempts) {
                    stuck = true;
                    break;
                }
                RedSlots<NW> *rs = rsb + (it & 1u);
                const int r = att == 0
                                  ? (int)te->idx
                                  : (int)warmup_index(step_draw(a.seed, ACHR_CHAIN_ID, (uint32_t)s, (uint32_t)att),
                                                                  (uint32_t)a.W);
                if (r < 0 || r >= a.W) {  // never read outside the warmup matrix (uniform over the CTA)
                    failed = true;
                    break;
                }
                if (buf_col != r) {
                    const double2 *col = reinterpret_cast<const double2 *>(a.warmup + (size_t)r * (size_t)a.ldw);
#pragma unroll
                    for (int k = 0; k < KP; ++k) {
                        const int q = tid + k * BD;
                        double2 v = make_double2(0.0, 0.0);
                        if (q < npair) v = ld_column(col + q);
                        dreg[2 * k] = v.x;
                        dreg[2 * k + 1] = v.y;
                    }
                }
                buf_col = -1;  // from here on dreg is the direction

                // Phase A: d = w_r - A / (W + t)  (reference ACHRCuda.cu:260-264);
                // in hit-and-run mode the column is the direction itself.
                // Phase B1 (merged): the brackets need ||d|| only for the
                // candidacy test |d_i| > u_tol ||d||, so they are formed in the
                // same pass, where they fill the FP64 pipe's latency, with a
                // threshold interval checked once the block has the norm: above
                // by uthr_max, below by a hundredth of the last attempt's (0
                // before the first).  A coordinate certain under both is
                // classified; any other keeps its lower ends and is settled
                // exactly in phase B2.
                float ss = 0.0f;
                Minima mn;
                {
                    const double ninv = -te->inv;
                    const float t_hi = fmaxf(a.uthr_max, kDCert);
#pragma unroll
                    for (int k = 0; k < KP; ++k) {
                        const int q = tid + k * BD;
                        if (ACHR_PAD_SLOT(k)) continue;  // padding: d stays 0, never a candidate
                        // Long directions: one pair at a time.  Left to itself the compiler forms many
                        // pairs together and spills for it (SM clocks per chain-step without and
                        // with: n = 2500 6935, 6786; 5000 15320, 14672; 6500 19130, 17800; 7440
                        // 25010, 23090); short ones gain nothing.
                        if (EPT >= 16) __syncwarp();
                        if (q == odd) dreg[2 * k + 1] = 0.0;
                        if (!hr) {
                            const double2 A2 = ACHR_ACC_GET(k);
                            dreg[2 * k] = fma(A2.x, ninv, dreg[2 * k]);
                            dreg[2 * k + 1] = fma(A2.y, ninv, dreg[2 * k + 1]);
                        }
                        const float4 b = __ldg(bnd2 + q);
                        ACHR_X32(k, x0, x1)
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const float d32 = d_to_f32(dreg[2 * k + c]);
                            ss = fmaf(d32, d32, ss);
                            if (merged) mn.add(bracket(c ? x1 : x0, d32, c ? b.z : b.x, c ? b.w : b.y, e0, t_hi, t_lo));
                        }
                    }
                }
                float uh = warp_min_f32(mn.uh), ul = warp_min_f32(mn.ul);
#pragma unroll
                for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                if (NW > 1) {
                    if (lane == 0) {
                        rs->sum1[warp] = ss;
                        rs->uh[warp] = uh;
                        rs->ul[warp] = ul;
                    }
                    cta_sync<BD>();
                    if (tid == 0) rsb[(it + 1) & 1u].clear();  // read last before this barrier
                    ss = slots_sum<NW>(rs->sum1);
                    uh = slots_min<NW>(rs->uh);
                    ul = slots_min<NW>(rs->ul);
                }
                const float norm32 = sqrt_approx(ss);
                if (!(norm32 > 0.0f) || !(norm32 < INFINITY)) {
                    if (tid == 0) ++cnt[CNT_REJECTED];
                    continue;
                }

                // Phase B1: FP32 brackets (reference ratio test ACHRCuda.cu:266-281)
                const float uthr = a.utol32 * norm32;
                const float uthr_hi = uthr * kNormUp, uthr_lo = uthr * kNormDn;
                const bool stands = merged && uthr_hi <= a.uthr_max && t_lo <= uthr_lo;
                t_lo = 0.01f * uthr_lo;
                if (!stands) {
                    // separate pass (merged: ||d|| left the interval the merged brackets assumed)
                    if (merged) cta_sync<BD>();  // uh and ul of this attempt may still be read
                    mn = Minima();
                    if (!a.exact_ratio) {
                        const float t_hi = fmaxf(uthr_hi, kDCert);
#pragma unroll
                        for (int k = 0; k < KP; ++k) {
                            if (ACHR_PAD_SLOT(k)) continue;
                            const float4 b = __ldg(bnd2 + tid + k * BD);
                            ACHR_X32(k, x0, x1)
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                mn.add(bracket(c ? x1 : x0, d_to_f32(dreg[2 * k + c]), c ? b.z : b.x,
                                               c ? b.w : b.y, e0, t_hi, uthr_lo));
                            }
                        }
                    }
                    uh = warp_min_f32(mn.uh);
                    ul = warp_min_f32(mn.ul);
                    if (NW > 1) {
                        if (lane == 0) {
                            rs->uh[warp] = uh;
                            rs->ul[warp] = ul;
                        }
                        cta_sync<BD>();
                        uh = slots_min<NW>(rs->uh);
                        ul = slots_min<NW>(rs->ul);
                    }
                }

                // FP64 norm, only when some candidacy test sits inside the FP32
                // norm's margin (found in phase B2, which then runs once more)
                // or every candidate is evaluated in FP64.
                RatioTest t;
                t.uh = uh;
                t.ul = ul;
                t.uthr_hi = uthr_hi;
                t.uthr_lo = uthr_lo;
                t.e0 = e0;
                t.have_norm64 = false;
                t.thr64 = 0.0;
                bool want_norm64 = a.exact_ratio != 0;
                int anyv;
                for (;;) {
                    if (want_norm64) {
                        double s64 = fp64_zero_here();
#pragma unroll
                        for (int k = 0; k < EPT; ++k) s64 = fma(dreg[k], dreg[k], s64);
#pragma unroll
                        for (int o = 16; o; o >>= 1) s64 += __shfl_xor_sync(0xffffffffu, s64, o);
                        if (lane == 0) rs->sum5[warp] = s64;
                        cta_sync<BD>();
                        s64 = 0.0;
#pragma unroll
                        for (int w = 0; w < NW; ++w) s64 += rs->sum5[w];
                        t.have_norm64 = true;
                        t.thr64 = a.u_tol * sqrt(s64);
                    }

                    // Phase B2: FP64 evaluation of every coordinate whose bracket can
                    // hold a minimum.  Only a thread whose own smallest lower ends
                    // reach the block minima can hold one.
                    t.kh = t.kl = kInfBits;
                    t.found = 0;
                    const bool mine = mn.lh <= uh || mn.ll <= ul;
                    if (EPT <= 8 || a.exact_ratio) {
                        // Each thread its own: a few elements (or, exact_ratio, all of
                        // them), both sides of different lanes at once.
                        unsigned mh = 0, ml = 0;  // bit k: contender for max / min step
                        if (a.exact_ratio) {
                            mh = ml = (EPT >= 32) ? 0xFFFFFFFFu : ((1u << EPT) - 1u);
                        } else if (EPT <= 8 && mine) {
#pragma unroll
                            for (int k = 0; k < KP; ++k) {
                                if (ACHR_PAD_SLOT(k)) continue;
                                const float4 b = __ldg(bnd2 + tid + k * BD);
                                ACHR_X32(k, x0, x1)
#pragma unroll
                                for (int c = 0; c < 2; ++c) {
                                    const Bracket B = bracket(c ? x1 : x0, d_to_f32(dreg[2 * k + c]), c ? b.z : b.x,
                                                              c ? b.w : b.y, e0, 0.0f, uthr_lo);
                                    mh |= (B.live && B.lo_h <= uh ? 1u : 0u) << (2 * k + c);
                                    ml |= (B.live && B.lo_l <= ul ? 1u : 0u) << (2 * k + c);
                                }
                            }
                        }
                        if (mh | ml) atomicAdd(exact_count, __popc(mh | ml));
                        while (mh | ml) {
                            const int k = __ffs(mh | ml) - 1;
                            const unsigned bit = 1u << k;
                            const int i = 2 * (tid + (k >> 1) * BD) + (k & 1);
                            const bool side_h = (mh & bit) != 0;
                            if (side_h) mh &= ~bit;
                            else ml &= ~bit;
                            evaluate(a, t, xs[i], pick(dreg, k), i, __ldg(a.bnd + i), side_h);
                        }
                    } else {
                        // A thread's elements one per lane: the warp passes them their d
                        // (a thread forming its own EPT brackets again held up the chain
                        // for a thousand clocks a step).
                        for (unsigned m = __ballot_sync(0xffffffffu, mine); m; m &= m - 1) {
                            const int src = __ffs(m) - 1;
                            double dk = 0.0;
#pragma unroll
                            for (int k = 0; k < EPT; ++k) {
                                const double v = __shfl_sync(0xffffffffu, dreg[k], src);
                                dk = lane == k ? v : dk;
                            }
                            const int i = 2 * (warp * 32 + src + (lane >> 1) * BD) + (lane & 1);
                            bool h = false, l = false;
                            double xi = 0.0;
                            float2 b = make_float2(0.0f, 0.0f);
                            if (lane < EPT) {
                                xi = xs[i];
                                b = __ldg(a.bnd + i);
                                const Bracket B = bracket(x_to_f32(xi), d_to_f32(dk), b.x, b.y, e0, 0.0f, uthr_lo);
                                h = B.live && B.lo_h <= uh;
                                l = B.live && B.lo_l <= ul;
                            }
                            if (h || l) atomicAdd(exact_count, 1);
                            while (h || l) {  // one coordinate is rarely a contender for both
                                evaluate(a, t, xi, dk, i, b, h);
                                if (h) h = false;
                                else l = false;
                            }
                            __syncwarp();
                        }
                    }
                    if (NW > 1) {  // a contender or two per step: they meet in shared memory
                        if (t.found) {
                            atomicMin(&rs->kh, t.kh);
                            atomicMin(&rs->kl, t.kl);
                            atomicOr(&rs->flags, (unsigned)t.found);
                        }
                        cta_sync<BD>();
                        t.kh = rs->kh;
                        t.kl = rs->kl;
                        anyv = (int)rs->flags;
                    } else {
                        __syncwarp();
                        t.kh = warp_min_u64(t.kh);
                        t.kl = warp_min_u64(t.kl);
                        anyv = (int)__reduce_or_sync(0xffffffffu, (unsigned)t.found);
                    }
                    if (!(anyv & 2) || t.have_norm64) break;
                    // a contender's candidacy needs the FP64 norm: evaluate again with it
                    want_norm64 = true;
                    cta_sync<BD>();
                    if (tid == 0) rs->clear();  // (the norm's barrier follows)
                }
                anyv &= 1;
                if (!anyv) {  // no candidate: rejection (see ACHRCuda.cu:283-288)
                    if (tid == 0) ++cnt[CNT_REJECTED];
                    continue;
                }
                const double qh = __longlong_as_double((long long)t.kh);
                const double ql = __longlong_as_double((long long)t.kl);

                // Rejection test |min| < tol && |max| < tol (ACHRCuda.cu:316-319),
                // min = -ql ||d||, max = qh ||d||; FP32 unless inside the margin.
                bool reject;
                {
                    const float qh32 = f64_to_f32_rz(qh), ql32 = f64_to_f32_rz(ql);
                    const float th_lo = qh32 * norm32 * kNormDn, th_hi = qh32 * kAdUp * norm32 * kNormUp;
                    const float tl_lo = ql32 * norm32 * kNormDn, tl_hi = ql32 * kAdUp * norm32 * kNormUp;
                    const float tol_lo = a.mmt32 * kDn, tol_hi = a.mmt32 * kUp;
                    const bool big = th_lo >= tol_hi || tl_lo >= tol_hi;
                    const bool small = th_hi < tol_lo && tl_hi < tol_lo;
                    if (big) {
                        reject = false;
                    } else if (small) {
                        reject = true;
                    } else {
                        double s64 = fp64_zero_here();
#pragma unroll
                        for (int k = 0; k < EPT; ++k) s64 = fma(dreg[k], dreg[k], s64);
#pragma unroll
                        for (int o = 16; o; o >>= 1) s64 += __shfl_xor_sync(0xffffffffu, s64, o);
                        cta_sync<BD>();  // slot sum5 may hold this attempt's earlier norm
                        if (lane == 0) rs->sum5[warp] = s64;
                        cta_sync<BD>();
                        s64 = 0.0;
#pragma unroll
                        for (int w = 0; w < NW; ++w) s64 += rs->sum5[w];
                        const double nrm = sqrt(s64);
                        reject = fabs(ql * nrm) < a.max_min_tol && fabs(qh * nrm) < a.max_min_tol;
                    }
                }
                if (reject) {
                    if (tid == 0) ++cnt[CNT_REJECTED];
                    continue;
                }
                // t / ||d|| with t = U (max - min) + min (reference ACHRCuda.cu:314).
                // One warp computes it: its two FP64 instructions in each of 12 warps
                // would hold the pipe for 465 clocks, the extra barrier costs 60.
                double sstep;
                if (NW > 1) {
                    if (warp == 0) {
                        const double v = fma(te->U, qh + ql, -ql);
                        if (lane == 0) rs->step = v;
                    }
                    cta_sync<BD>();
                    sstep = rs->step;
                } else {
                    sstep = fma(te->U, qh + ql, -ql);
                }

                // Phase C: x = prev + t u (ACHRCuda.cu:242-249), residual check every
                // check_period steps (:325-344), clip + centre (:193-206, :347-350).
                const bool check = chk == 0;
                chk = (chk + 1 == a.check_period) ? 0 : chk + 1;
                // The next step's column, requested as dreg's pairs come free (the
                // table's last step leaves it to the next step's refill).
                const int nxt = (s + 1 < a.step0 + a.T && s + 1 - tbase < kTbl) ? (int)tbl[s + 1 - tbase].idx : -1;
                const bool pre = nxt >= 0 && nxt < a.W;
                const double2 *ncol =
                    reinterpret_cast<const double2 *>(a.warmup + (size_t)(pre ? nxt : 0) * (size_t)a.ldw);
                if (!check) {
                    unsigned edge = 0;  // bit k: not provably inside the box, clip exactly below
#pragma unroll
                    for (int k = 0; k < KP; ++k) {
                        const int q = tid + k * BD;
                        if (!ACHR_PAD_SLOT(k)) {
                            const float4 b = __ldg(bnd2 + q);
                            double2 x2 = xs2[q];
                            x2.x = fma(sstep, dreg[2 * k], x2.x);
                            x2.y = fma(sstep, dreg[2 * k + 1], x2.y);
                            xs2[q] = x2;
                            const float x0 = x_to_f32(x2.x), x1 = x_to_f32(x2.y);
                            if (KX) {
                                xf[KX ? 2 * k : 0] = x0;
                                xf[KX ? 2 * k + 1 : 1] = x1;
                            }
                            const bool in0 = surely_inside(x0, b.x, b.y, a.bound_err);
                            const bool in1 = surely_inside(x1, b.z, b.w, a.bound_err);
                            edge |= (in0 ? 0u : 1u << (2 * k)) | (in1 ? 0u : 2u << (2 * k));
                            if (!hr) {  // hit-and-run: no centre to update
                                double2 A2 = ACHR_ACC_GET(k);
                                if (in0) A2.x += x2.x;
                                if (in1) A2.y += x2.y;
                                ACHR_ACC_SET(k, A2);
                            }
                        }
                        if (pre && q < npair) {
                            const double2 v = ld_column(ncol + q);
                            dreg[2 * k] = v.x;
                            dreg[2 * k + 1] = v.y;
                        }
                    }
                    if (pre) buf_col = nxt;
                    if (edge) {
                        for (; edge; edge &= edge - 1) {
                            const int k = __ffs(edge) - 1, i = 2 * (tid + (k >> 1) * BD) + (k & 1);
                            const double xc = clip_exact(xs[i], exact_bounds(a, i));
                            xs[i] = xc;
                            if (!hr) ACHR_ACC_ADD(k, i, xc);
                        }
                        if (KX) {
#pragma unroll
                            for (int k = 0; k < KP; ++k) {
                                const double2 x2 = xs2[tid + k * BD];
                                xf[KX ? 2 * k : 0] = x_to_f32(x2.x);
                                xf[KX ? 2 * k + 1 : 1] = x_to_f32(x2.y);
                            }
                        }
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < KP; ++k) {
                        const int q = tid + k * BD;
                        if (ACHR_PAD_SLOT(k)) continue;
                        double2 x2 = xs2[q];
                        x2.x = fma(sstep, dreg[2 * k], x2.x);
                        x2.y = fma(sstep, dreg[2 * k + 1], x2.y);
                        xs2[q] = x2;
                    }
                    cta_sync<BD>();  // every x update visible
                    if (tid == 0) ++cnt[CNT_CHECKS];
                    if (SEG) {
                        // Segmented sampling: the check ends this launch for the chain.  S x goes
                        // out as it is summed (FP64 and BF16 split, device row order); the passes
                        // read it only for a chain flagged below.
                        unsigned long long mx = residual_rows<BD>(a, xs, p, tid);
                        mx = warp_max_u64(mx);
                        if (lane == 0) rs->max4[warp] = mx;
                        cta_sync<BD>();
                        mx = 0;
#pragma unroll
                        for (int w = 0; w < NW; ++w) mx = umax(mx, rs->max4[w]);
                        const bool reproject = mx > (unsigned long long)__double_as_longlong(a.residual_tol);
                        if (reproject && tid == 0) {
                            ++cnt[CNT_REPROJ];
                            if (*a.seg_any == 0ull) atomicOr(a.seg_any, 1ull);
                        }
#pragma unroll
                        for (int k = 0; k < KP; ++k) {
                            const int i = 2 * (tid + k * BD);
                            const size_t o = (size_t)p * (size_t)a.ld_seg + (size_t)i;
                            const double2 A2 = ACHR_ACC_GET(k), x2 = xs2[tid + k * BD];
                            if (i < a.n) {
                                a.seg_x[o] = x2.x;
                                a.seg_A[o] = A2.x;
                            }
                            if (i + 1 < a.n) {
                                a.seg_x[o + 1] = x2.y;
                                a.seg_A[o + 1] = A2.y;
                            }
                        }
                        if (tid == 0) {
                            a.seg_flags[p] =
                                SEG_STARTED | SEG_ACCEPTED | SEG_PENDING | (reproject ? SEG_REPROJ : 0u);
                            ++cnt[CNT_ACCEPTED];
                        }
                        any_accepted = true;
                        seg_pending = true;
                        ++it;
                        break;
                    }
                    unsigned long long mx = residual_max_bits<BD>(a, xs, tid);
                    mx = warp_max_u64(mx);
                    if (lane == 0) rs->max4[warp] = mx;
                    cta_sync<BD>();
                    mx = 0;
#pragma unroll
                    for (int w = 0; w < NW; ++w) mx = umax(mx, rs->max4[w]);
                    if (mx > (unsigned long long)__double_as_longlong(a.residual_tol)) {
                        // x <- N (N^T x) in FP64 (reference reprojectPoint(2), ACHRCuda.cu:208-230).
                        // The scratch is As: the accumulator waits in the direction's registers.
                        if (tid == 0) ++cnt[CNT_REPROJ];
#pragma unroll
                        for (int k = 0; k < KA; ++k) {
                            const double2 A2 = As2[tid + k * BD];
                            dreg[2 * k] = A2.x;
                            dreg[2 * k + 1] = A2.y;
                        }
                        cta_sync<BD>();
                        if (a.pinv32) {
                            residual_form_reproject<BD>(a, xs, reinterpret_cast<float2 *>(As), zs,
                                                        a.z_rows ? a.z_rows : a.m, tid);
                        } else {
                            const int n = a.n;
                            null_coordinates<BD>(a, xs, ys, tid);
                            cta_sync<BD>();
                            for (int i = tid; i < n; i += BD) {
                                double acc = 0.0;
                                for (int j = 0; j < a.d; ++j)
                                    acc = fma(__ldg(a.N + (size_t)j * (size_t)n + i), ys[j], acc);
                                xs[i] = acc;
                            }
                        }
                        cta_sync<BD>();
#pragma unroll
                        for (int k = 0; k < KA; ++k)
                            As2[tid + k * BD] = make_double2(dreg[2 * k], dreg[2 * k + 1]);
                    }
                    unsigned edge = 0;
#pragma unroll
                    for (int k = 0; k < KP; ++k) {
                        const int q = tid + k * BD;
                        if (!ACHR_PAD_SLOT(k)) {
                            const float4 b = __ldg(bnd2 + q);
                            const double2 x2 = xs2[q];
                            const float x0 = x_to_f32(x2.x), x1 = x_to_f32(x2.y);
                            if (KX) {
                                xf[KX ? 2 * k : 0] = x0;
                                xf[KX ? 2 * k + 1 : 1] = x1;
                            }
                            const bool in0 = surely_inside(x0, b.x, b.y, a.bound_err);
                            const bool in1 = surely_inside(x1, b.z, b.w, a.bound_err);
                            edge |= (in0 ? 0u : 1u << (2 * k)) | (in1 ? 0u : 2u << (2 * k));
                            if (!hr) {
                                double2 A2 = ACHR_ACC_GET(k);
                                if (in0) A2.x += x2.x;
                                if (in1) A2.y += x2.y;
                                ACHR_ACC_SET(k, A2);
                            }
                        }
                        if (pre && q < npair) {
                            const double2 v = ld_column(ncol + q);
                            dreg[2 * k] = v.x;
                            dreg[2 * k + 1] = v.y;
                        } else {
                            dreg[2 * k] = dreg[2 * k + 1] = 0.0;
                        }
                    }
                    if (pre) buf_col = nxt;
                    if (edge) {
                        for (; edge; edge &= edge - 1) {
                            const int k = __ffs(edge) - 1, i = 2 * (tid + (k >> 1) * BD) + (k & 1);
                            const double xc = clip_exact(xs[i], exact_bounds(a, i));
                            xs[i] = xc;
                            if (!hr) ACHR_ACC_ADD(k, i, xc);
                        }
                        if (KX) {
#pragma unroll
                            for (int k = 0; k < KP; ++k) {
                                const double2 x2 = xs2[tid + k * BD];
                                xf[KX ? 2 * k : 0] = x_to_f32(x2.x);
                                xf[KX ? 2 * k + 1 : 1] = x_to_f32(x2.y);
                            }
                        }
                    }
                }
                if (tid == 0) ++cnt[CNT_ACCEPTED];
                any_accepted = true;
                ++it;  // the next attempt takes the other slots
                break;
            }
        }
        if (stuck && !was_stuck && tid == 0) ++cnt[CNT_STUCK];
        if (cta_any<BD>(failed)) {
            failed = true;
            break;
        }
        if (SEG && !seg_pending && !a.seg_final) {
            // A segmented launch that is not the run's last: keep the state for the next one.
#pragma unroll
            for (int k = 0; k < KP; ++k) {
                const int i = 2 * (tid + k * BD);
                const size_t o = (size_t)p * (size_t)a.ld_seg + (size_t)i;
                const double2 A2 = ACHR_ACC_GET(k), x2 = xs2[tid + k * BD];
                if (i < a.n) {
                    a.seg_x[o] = x2.x;
                    a.seg_A[o] = A2.x;
                }
                if (i + 1 < a.n) {
                    a.seg_x[o + 1] = x2.y;
                    a.seg_A[o + 1] = A2.y;
                }
            }
            if (tid == 0)
                a.seg_flags[p] = SEG_STARTED | (any_accepted ? SEG_ACCEPTED : 0u) | (stuck ? SEG_STUCK : 0u);
        }
        if (SEG && (seg_pending || !a.seg_final)) {
            cta_sync<BD>();
            continue;  // the point is emitted by the run's last launch
        }

        // Emitted point: residual / bound diagnostics and, on request, the final
        // feasibility projection (project, clip, re-check).
        if (any_accepted) {
            RedSlots<NW> *rs = rsb;
            const int n = a.n;
            unsigned long long res = 0;
            for (int pass = 0; pass < 2; ++pass) {
                unsigned long long mx = residual_max_bits<BD>(a, xs, tid);
                mx = warp_max_u64(mx);
                cta_sync<BD>();
                if (lane == 0) rs->max4[warp] = mx;
                cta_sync<BD>();
                res = 0;
#pragma unroll
                for (int w = 0; w < NW; ++w) res = umax(res, rs->max4[w]);
                if (pass == 1 || !a.final_project || __longlong_as_double((long long)res) <= a.feasibility_tol) break;
                if (tid == 0) ++cnt[CNT_FINAL_PROJ];
#pragma unroll
                for (int k = 0; k < 2 * KA; ++k) dreg[k] = As[tid + k * BD];
                cta_sync<BD>();
                null_coordinates<BD>(a, xs, ys, tid);
                cta_sync<BD>();
                for (int i = tid; i < n; i += BD) {
                    double acc = 0.0;
                    for (int j = 0; j < a.d; ++j) acc = fma(__ldg(a.N + (size_t)j * (size_t)n + i), ys[j], acc);
                    xs[i] = clip_exact(acc, ld_lbub(a.lbub + i));
                }
                cta_sync<BD>();
#pragma unroll
                for (int k = 0; k < 2 * KA; ++k) As[tid + k * BD] = dreg[k];
            }
            double viol = 0.0;
            for (int i = tid; i < n; i += BD) {
                const double xi = xs[i];
                const double2 lu = ld_lbub(a.lbub + i);
                viol = fmax(viol, fmax(lu.x - xi, xi - lu.y));
            }
            unsigned long long vb = (unsigned long long)__double_as_longlong(viol);
            vb = warp_max_u64(vb);
            cta_sync<BD>();
            if (lane == 0) rs->max4[warp] = vb;
            cta_sync<BD>();
            vb = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) vb = umax(vb, rs->max4[w]);
            if (tid == 0) {
                worst[0] = umax(worst[0], res);
                worst[1] = umax(worst[1], vb);
            }
        }
        for (int i = tid; i < a.n; i += BD) a.out[(size_t)i * (size_t)a.ld_out + (size_t)p] = any_accepted ? xs[i] : 0.0;
        if (a.A_out) {
#pragma unroll
            for (int k = 0; k < KP; ++k) {
                const int i = 2 * (tid + k * BD);
                const double2 A2 = ACHR_ACC_GET(k);
                if (i < a.n) a.A_out[(size_t)i * (size_t)a.ld_state + (size_t)p] = A2.x;
                if (i + 1 < a.n) a.A_out[(size_t)(i + 1) * (size_t)a.ld_state + (size_t)p] = A2.y;
            }
        }
        cta_sync<BD>();
    }
#undef ACHR_CHAIN_ID
#undef ACHR_PAD_SLOT
#undef ACHR_ACC_GET
#undef ACHR_ACC_SET
#undef ACHR_ACC_ADD
#undef ACHR_X32

    cta_sync<BD>();
    if (tid == 0) {
        unsigned long long *c = a.counters;
        const int slots[6] = {CNT_ACCEPTED, CNT_REJECTED, CNT_CHECKS, CNT_REPROJ, CNT_STUCK, CNT_FINAL_PROJ};
        for (int q = 0; q < 6; ++q)
            if (cnt[slots[q]]) atomicAdd(c + slots[q], cnt[slots[q]]);
        if (*exact_count) atomicAdd(c + CNT_EXACT, (unsigned long long)*exact_count);
        if (worst[0]) atomicMax(c + CNT_MAXRES_BITS, worst[0]);
        if (worst[1]) atomicMax(c + CNT_MAXVIOL_BITS, worst[1]);
        if (failed) atomicOr(c + CNT_ERROR, ERR_WAIT_TIMEOUT);
    }
    return failed;
}

// The `never` barrier of a CTA (tail of the dynamic shared memory).
template <int BD, int EPT>
__device__ __forceinline__ void chain_init_barrier(unsigned char *smem_raw) {
    if (threadIdx.x == 0) mbar_init(chain_never<BD, EPT>(smem_raw), 1);
    __syncthreads();
}

// One model: CTA b takes chains b, b + grid, ...
template <int BD, int EPT, bool SEG>
__global__ void __launch_bounds__(BD, (chain_min_ctas<BD, EPT>())) achr_chain_kernel(const ChainArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    chain_init_barrier<BD, EPT>(smem_raw);
    chain_run<BD, EPT, SEG>(a, blockIdx.x, gridDim.x, a.P, smem_raw);
}

// Many models of one configuration in one persistent launch: each CTA takes
// the next (model, first chain, end chain) item of a device work queue until
// the queue is empty.  The host orders the items longest model first, with
// tiles that shrink towards the end of the queue, and gives each model's
// residual-form reprojection room for z beside the header (extra_smem) or in
// turns (z_rows), or sets the form off.  When a
// model's last chain is done, its finish time (globaltimer, ns) goes to
// done_ns[model].
template <int BD, int EPT>
__global__ void __launch_bounds__(BD, (chain_min_ctas<BD, EPT>())) achr_chain_queue_kernel(const ChainQueue q) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ ChainArgs sa;
    __shared__ int4 cur;
    static_assert(sizeof(ChainArgs) % sizeof(int) == 0, "ChainArgs is copied as 32-bit words");
    chain_init_barrier<BD, EPT>(smem_raw);
    int model = -1;
    for (;;) {
        if (threadIdx.x == 0) {
            const int k = atomicAdd(q.next, 1);
            cur = k < q.n_items ? q.items[k] : make_int4(-1, 0, 0, 0);
        }
        __syncthreads();
        const int4 item = cur;
        if (item.x < 0) break;
        if (item.x != model) {
            const int *src = reinterpret_cast<const int *>(q.args + item.x);
            int *dst = reinterpret_cast<int *>(&sa);
            for (int w = threadIdx.x; w < (int)(sizeof(ChainArgs) / sizeof(int)); w += BD) dst[w] = src[w];
            model = item.x;
        }
        __syncthreads();
        const bool failed = chain_run<BD, EPT, false>(sa, item.y, 1, item.z, smem_raw);
        if (threadIdx.x == 0) {
            const int n = item.z - item.y;
            if (atomicAdd(q.chains_done + item.x, n) + n == sa.P) q.done_ns[item.x] = global_ns();
        }
        if (failed) break;  // recorded in the model's counters; the CTA stops taking work
        __syncthreads();    // `cur` and `sa` are rewritten only after every thread is done with them
    }
    if (threadIdx.x == 0 && q.cta_ns) q.cta_ns[blockIdx.x] = global_ns();
}

// Lets a kernel be launched with `need` bytes of dynamic shared memory.  The limit belongs to the
// function, not to the launch: set to a launch's own need it fails another thread's launch that needs
// more, so it is always the same one (what a CTA may have, less 1 KB for static arrays).
inline cudaError_t allow_smem(const void *kernel, size_t need) {
    constexpr size_t kMost = 226 * 1024;
    if (need > kMost) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMost);
}

// Occupancy-sized persistent launch of one configuration.  max_ctas > 0 caps
// the grid.
template <int BD, int EPT, bool SEG>
cudaError_t launch_cfg_kernel(const ChainArgs &a_in, cudaStream_t stream, int max_ctas, ChainFit *fit) {
    auto *const KFN = achr_chain_kernel<BD, EPT, SEG>;
    ChainArgs a = a_in;
    const int turn = a.z_rows;  // > 0: the rows of z per turn that this launch has to take
    a.z_rows = 0;
    const size_t base = chain_smem_bytes_cfg<BD, EPT>();
    // The residual-form reprojection keeps z (m floats) in shared memory and
    // the residual in the accumulator's place.  Where z would cost a resident
    // CTA per SM, it takes turns in what the residual leaves of that place
    // (5063 x 7440, 256 x 30: three turns of 2162 rows), if those are at most
    // eight; else the form is not used.
    const size_t zbytes = ((size_t)a.m * sizeof(float) + 15) & ~(size_t)15;
    // (its residual takes the accumulator's place while that waits in registers: m <= ldw <= NP)
    if (a.pinv32 && a.m > a.ldw) a.pinv32 = nullptr;
    size_t smem = base + (a.pinv32 ? zbytes : 0);
    cudaError_t e = allow_smem(reinterpret_cast<const void *>(KFN), std::max(smem, base));
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KFN, BD, base);
    if (e != cudaSuccess) return e;
    if (a.pinv32) {
        int per_sm_z = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_z, KFN, BD, smem);
        if (e != cudaSuccess) return e;
        if (per_sm_z < per_sm || (turn > 0 && turn < a.m)) {
            a.z_rows = residual_z_rows(a.m, chain_acc_doubles<BD, EPT>());
            if (turn > 0) {
                if (a.z_rows >= turn) {
                    a.z_rows = turn;
                } else if (turn == a.m && per_sm_z > 0) {  // all of z at once, in memory of its own
                    a.z_rows = 0;
                    per_sm = per_sm_z;
                } else {
                    return cudaErrorInvalidConfiguration;  // (the caller's rule has ruled it out)
                }
            }
            if (a.z_rows) smem = base;
            else if (turn == 0) {
                a.pinv32 = nullptr;
                smem = base;
            }
        }
    }
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    if (fit) {
        fit->per_sm = per_sm;
        fit->turn = a.pinv32 ? (a.z_rows ? a.z_rows : a.m) : 0;
    }
    if (a.P <= 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    long long grid = (long long)sms * per_sm;
    if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
    if (grid > a.P) grid = a.P;
    if (grid < 1) return cudaSuccess;
    KFN<<<(unsigned)grid, BD, smem, stream>>>(a);
    return cudaGetLastError();
}

// Persistent work-queue launch of one configuration: `grid` CTAs (0: every
// resident slot of the GPU), with q.extra_smem bytes of shared memory beyond
// the header for the residual-form reprojection.  per_sm_out (if non-NULL)
// receives the CTAs that fit on one SM; with q.n_items = 0 nothing is launched.
template <int BD, int EPT>
cudaError_t launch_queue_cfg(const ChainQueue &q, cudaStream_t stream, int grid, int *per_sm_out) {
    auto *const KFN = achr_chain_queue_kernel<BD, EPT>;
    const size_t smem = chain_smem_bytes_cfg<BD, EPT>() + q.extra_smem;
    cudaError_t e = allow_smem(reinterpret_cast<const void *>(KFN), smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KFN, BD, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    if (per_sm_out) *per_sm_out = per_sm;
    if (q.n_items <= 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    long long g = grid > 0 ? grid : (long long)sms * per_sm;
    if (g > q.n_items) g = q.n_items;
    KFN<<<(unsigned)g, BD, smem, stream>>>(q);
    return cudaGetLastError();
}

// Occupancy-sized persistent launch of one configuration (segmented launches
// take the kernel's segmented instantiation).
template <int BD, int EPT>
cudaError_t launch_cfg(const ChainArgs &a, cudaStream_t stream, int max_ctas, ChainFit *fit) {
    return a.seg ? launch_cfg_kernel<BD, EPT, true>(a, stream, max_ctas, fit)
                 : launch_cfg_kernel<BD, EPT, false>(a, stream, max_ctas, fit);
}

}  // namespace achr
