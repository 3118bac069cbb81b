// Shared device helpers for the B200 PIV path.
//
// Where the reference computes in f64 (integral-image window statistics, preprocess.rs:76-125,
// 199-216) the fast path here uses no FP64: box sums are exact int64 fixed-point sums (integer
// addition is associative, so any parallel order gives the same bits), and the few divisions,
// squares and square roots that turn them into a mean and a standard deviation run in
// double-float arithmetic (an unevaluated sum hi + lo of two f32 values, ~48 significant bits).
// The final f32 values then agree with the reference's f64-then-round results except when the
// exact value lies within ~2^-48 (relative) of an f32 rounding boundary.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace pivb200 {

// field.rs:6-20
constexpr uint8_t F_NO_SIGNAL = 1u << 0;
constexpr uint8_t F_LOW_PPR = 1u << 1;
constexpr uint8_t F_MEDIAN_OUTLIER = 1u << 2;
constexpr uint8_t F_REPLACED = 1u << 3;
constexpr uint8_t F_OUT_OF_RANGE = 1u << 4;
constexpr uint8_t F_INVALID = F_NO_SIGNAL | F_LOW_PPR | F_MEDIAN_OUTLIER | F_OUT_OF_RANGE;

constexpr float MAX_PPR = 1000.0f;  // correlate.rs:24

// Grid of interrogation windows (grid.rs:8-16).
struct GridP {
    int32_t window, step, nx, ny, x0, y0;
};

// ---------------------------------------------------------------------------------------------
// Double-float arithmetic (error-free transformations; Dekker/Knuth two-sum and FMA two-product).
// The __f*_rn intrinsics are never contracted or reassociated by the compiler.
// ---------------------------------------------------------------------------------------------
struct dfloat {
    float hi, lo;
};

__device__ __forceinline__ dfloat dd_two_sum(float a, float b) {
    float s = __fadd_rn(a, b);
    float bb = __fsub_rn(s, a);
    float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return {s, e};
}

__device__ __forceinline__ dfloat dd_quick(float a, float b) {
    float s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}

__device__ __forceinline__ dfloat dd_two_prod(float a, float b) {
    float p = __fmul_rn(a, b);
    return {p, __fmaf_rn(a, b, -p)};
}

__device__ __forceinline__ dfloat dd_add(dfloat x, dfloat y) {
    dfloat s = dd_two_sum(x.hi, y.hi);
    dfloat t = dd_two_sum(x.lo, y.lo);
    float e = __fadd_rn(s.lo, t.hi);
    dfloat u = dd_quick(s.hi, e);
    return dd_quick(u.hi, __fadd_rn(u.lo, t.lo));
}

__device__ __forceinline__ dfloat dd_neg(dfloat x) { return {-x.hi, -x.lo}; }

__device__ __forceinline__ dfloat dd_mul(dfloat x, dfloat y) {
    dfloat p = dd_two_prod(x.hi, y.hi);
    float e = __fadd_rn(p.lo, __fadd_rn(__fmul_rn(x.hi, y.lo), __fmul_rn(x.lo, y.hi)));
    return dd_quick(p.hi, e);
}

// x / d for a plain float d.
__device__ __forceinline__ dfloat dd_div_f(dfloat x, float d) {
    float q1 = __fdiv_rn(x.hi, d);
    dfloat p = dd_two_prod(q1, d);
    float r = __fdiv_rn(__fadd_rn(__fsub_rn(__fsub_rn(x.hi, p.hi), p.lo), x.lo), d);
    return dd_quick(q1, r);
}

__device__ __forceinline__ dfloat dd_scale2(dfloat x, int k) {
    return {scalbnf(x.hi, k), scalbnf(x.lo, k)};
}

__device__ __forceinline__ dfloat dd_from_i64(long long v) {
    float hi = __ll2float_rn(v);
    long long rem = v - __float2ll_rn(hi);
    return dd_quick(hi, __ll2float_rn(rem));
}

__device__ __forceinline__ dfloat dd_sqrt(dfloat x) {
    if (!(x.hi > 0.0f)) return {0.0f, 0.0f};
    float s = __fsqrt_rn(x.hi);
    dfloat p = dd_two_prod(s, s);
    float r = __fdiv_rn(__fadd_rn(__fsub_rn(__fsub_rn(x.hi, p.hi), p.lo), x.lo), __fmul_rn(2.0f, s));
    return dd_quick(s, r);
}

__device__ __forceinline__ float dd_to_float(dfloat x) { return __fadd_rn(x.hi, x.lo); }

// ---------------------------------------------------------------------------------------------
// Exact fixed-point box statistics.
//
// A value v is quantised to q1 = round(v * 2^s1) and its exact square v*v (a two-product) to
// q2 = round(hi * 2^s2) + round(lo * 2^s2). The scales are chosen from the frame's largest |v|
// so that a sum over `count` values cannot overflow int64.
// ---------------------------------------------------------------------------------------------
struct FixScale {
    int s1, s2;
    // 2^s1 and 2^s2 as floats when 0 <= s <= 127: multiplying a finite float by 2^s with s >= 0
    // is exact up to overflow, where it rounds to +-inf as scalbnf does, so the product equals
    // scalbnf(v, s) bit for bit. Outside that range the quantisers fall back to scalbnf.
    float m1, m2;
    bool fast1, fast2;
};

__device__ __forceinline__ float pow2f(int s) { return __int_as_float((s + 127) << 23); }

// Largest exponent e with 2^e >= maxabs, then scales that keep count * 2^(e+s) <= 2^62.
__device__ __forceinline__ FixScale fix_scale(float maxabs, long long count) {
    FixScale fs{0, 0, 1.0f, 1.0f, true, true};
    if (!(maxabs > 0.0f) || !isfinite(maxabs)) return fs;
    int e;
    float m = frexpf(maxabs, &e);  // maxabs = m * 2^e, m in [0.5, 1)
    (void)m;
    int lc = 0;
    while ((1ll << lc) < count && lc < 62) ++lc;
    fs.s1 = 62 - lc - e;
    fs.s2 = 62 - lc - 2 * e;
    fs.fast1 = fs.s1 >= 0 && fs.s1 <= 127;
    fs.fast2 = fs.s2 >= 0 && fs.s2 <= 127;
    fs.m1 = fs.fast1 ? pow2f(fs.s1) : 1.0f;
    fs.m2 = fs.fast2 ? pow2f(fs.s2) : 1.0f;
    return fs;
}

__device__ __forceinline__ long long fix_q1(float v, const FixScale& fs) {
    return __float2ll_rn(fs.fast1 ? __fmul_rn(v, fs.m1) : scalbnf(v, fs.s1));
}

__device__ __forceinline__ long long fix_q2(float v, const FixScale& fs) {
    dfloat sq = dd_two_prod(v, v);
    if (fs.fast2) return __float2ll_rn(__fmul_rn(sq.hi, fs.m2)) + __float2ll_rn(__fmul_rn(sq.lo, fs.m2));
    return __float2ll_rn(scalbnf(sq.hi, fs.s2)) + __float2ll_rn(scalbnf(sq.lo, fs.s2));
}

// Entry (y, x) of an integral table stored in strips: rows that are multiples of kStripRows hold
// the full prefix, the others the prefix within their strip.
constexpr int kStripRows = 8;
__device__ __forceinline__ long long table_at(const long long* t, int stride, int y, int x) {
    const long long v = t[(size_t)y * stride + x];
    return y % kStripRows ? v + t[(size_t)(y / kStripRows * kStripRows) * stride + x] : v;
}

// IntegralImage::stats (preprocess.rs:114-125) from exact sums: mean and standard deviation as
// the reference's f64 arithmetic would round them to f32.
__device__ __forceinline__ void fix_stats(long long sum1, long long sum2, const FixScale& fs, float count,
                                          float* mean_out, float* std_out) {
    dfloat mean = dd_div_f(dd_scale2(dd_from_i64(sum1), -fs.s1), count);
    dfloat ex2 = dd_div_f(dd_scale2(dd_from_i64(sum2), -fs.s2), count);
    dfloat var = dd_add(ex2, dd_neg(dd_mul(mean, mean)));
    *mean_out = dd_to_float(mean);
    *std_out = dd_to_float(dd_sqrt(var));
}

// fix_stats without conversions, divisions or an IEEE square root, for scales that are plain powers of
// two (fix_stats_fast_ok) and many pixels: the local normalisation is bound by instructions, and 64-bit
// conversions and the reciprocals inside divisions run at an eighth of the FMA rate.
//   - an int64 (below 2^62) is split into 23-bit pieces that become floats by their bit patterns;
//   - a quotient by the small integer `count` is x * rc corrected by its exact remainder, which is the
//     rounded quotient for a correctly rounded rc (Markstein, "Computation of elementary functions on the
//     IBM RISC System/6000 processor", 1990). Both parts of mean and ex2 are therefore those of
//     fix_stats, and so is the variance, a difference of almost equal numbers in flat parts of an image.
//     (With one correction for both parts a frame of one value had a deviation in places, and the
//     largest error of a frame of 0.69 + 1e-6 noise grew by a tenth.) 0.3 % of a 1080p default pair.
//   - the root is x * rsqrt(x), refined once, corrected by its exact remainder (Karp and Markstein, "High
//     precision division and square root", 1997): accurate to about 2^-45, so the rounded root differs
//     from the one of fix_stats only within that distance of a rounding boundary.
// rc is 1 / count rounded to nearest; p1, p2 are 2^-s1, 2^-s2.
__device__ __forceinline__ bool fix_stats_fast_ok(const FixScale& fs) {
    return fs.s1 >= 0 && fs.s1 <= 100 && fs.s2 >= 0 && fs.s2 <= 100;
}

__device__ __forceinline__ dfloat dd_from_bits(long long v, float scale) {
    const float f2 = __fsub_rn(__int_as_float(0x4b400000 + (int)(v >> 46)), 12582912.0f);
    const float f1 = __fsub_rn(__int_as_float(0x4b000000 | ((int)(v >> 23) & 0x7fffff)), 8388608.0f);
    const float f0 = __fsub_rn(__int_as_float(0x4b000000 | ((int)v & 0x7fffff)), 8388608.0f);
    const dfloat a = dd_quick(__fmul_rn(f2, 70368744177664.0f), __fmul_rn(f1, 8388608.0f));  // exact
    const dfloat r = dd_quick(a.hi, __fadd_rn(a.lo, f0));
    return {__fmul_rn(r.hi, scale), __fmul_rn(r.lo, scale)};
}

// x / d rounded to nearest, for rc = 1 / d rounded to nearest.
__device__ __forceinline__ float div_rc(float x, float d, float rc) {
    const float q = __fmul_rn(x, rc);
    return __fmaf_rn(__fmaf_rn(-q, d, x), rc, q);
}

__device__ __forceinline__ dfloat dd_div_rc(dfloat x, float d, float rc) {
    const float q = div_rc(x.hi, d, rc);
    const dfloat p = dd_two_prod(q, d);
    return dd_quick(q, div_rc(__fadd_rn(__fsub_rn(__fsub_rn(x.hi, p.hi), p.lo), x.lo), d, rc));
}

__device__ __forceinline__ void fix_stats_fast(long long sum1, long long sum2, float p1, float p2, float count, float rc,
                                               float* mean_out, float* std_out) {
    const dfloat mean = dd_div_rc(dd_from_bits(sum1, p1), count, rc);
    const dfloat ex2 = dd_div_rc(dd_from_bits(sum2, p2), count, rc);
    const dfloat var = dd_add(ex2, dd_neg(dd_mul(mean, mean)));
    *mean_out = dd_to_float(mean);
    if (!(var.hi > 0.0f)) {
        *std_out = 0.0f;
        return;
    }
    const float y = rsqrtf(var.hi);
    float g = __fmul_rn(var.hi, y), h = __fmul_rn(0.5f, y);
    const float e = __fmaf_rn(-g, h, 0.5f);
    g = __fmaf_rn(g, e, g);
    h = __fmaf_rn(h, e, h);
    const dfloat p = dd_two_prod(g, g);
    *std_out = __fmaf_rn(__fadd_rn(__fsub_rn(__fsub_rn(var.hi, p.hi), p.lo), var.lo), h, g);
}

// ---------------------------------------------------------------------------------------------
// Programmatic dependent launch: a kernel launched through launch_dependent (kernels.h) may start
// while the kernel before it in the stream is finishing. Its threads call dependent_wait() before they
// read or write anything another kernel touches (it returns once that kernel has completed and its
// writes are visible; at once when the launch has no such predecessor), then let_dependents_start().
// The kernel before may still write while this one is resident, so nothing it touches counts as
// read-only here: such data is read through plain pointers, never through __ldg or a const
// __restrict__ argument (the compiler may move those loads above the wait, and their path need not be
// coherent). What was written by kernels further back is complete before this kernel starts, because
// the one in between has waited for it; the correlation kernels read the frames through __ldg on that
// ground (a placement or a copy always lies between them and the preparation).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void dependent_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_dependents_start() { asm volatile("griddepcontrol.launch_dependents;"); }

// Rust f32::clamp (NaN passes through).
__device__ __forceinline__ float rclamp(float x, float lo, float hi) {
    if (x < lo) return lo;
    if (x > hi) return hi;
    return x;
}

}  // namespace pivb200
