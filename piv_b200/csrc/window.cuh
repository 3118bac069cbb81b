// Window sampling and peak-fit helpers shared by the FP32 and tensor-core correlation kernels.
#pragma once

#include <cmath>

#include "common.cuh"
#include "packed.cuh"

namespace pivb200 {

// (value, row-major index): larger value wins, then the lower index (correlate.rs:233-238).
__device__ __forceinline__ void amax_combine(float& v, int& i, float ov, int oi) {
    if (ov > v || (ov == v && oi < i)) {
        v = ov;
        i = oi;
    }
}

// ---------------------------------------------------------------------------------------------
// Window sampling (correlate.rs:182-202): integer copy when both fractional parts are < 1e-4,
// otherwise bilinear with weights (1-tx)(1-ty), tx(1-ty), (1-tx)ty, tx*ty summed left to right, each
// product and sum rounded (no FMA), as the reference does it.
// Indices are clamped into the image so that no access can leave it whatever the origin.
//
// Both frames' windows of a pair are sampled together, A into the real and B into the imaginary
// part, in packed operations: a sample of both costs the 7 multiplications and additions of one.
// ---------------------------------------------------------------------------------------------
struct PairSource {
    const float* a;  // first pixel of the lane's column in frame A (B)
    const float* b;
    int last_a, last_b;  // rows below it that exist (row clamp)
    int right_a, right_b;  // right-hand tap: 1, or 0 at the right border of the image
    float2 tx, ty;
    bool copy_a, copy_b;
};

__device__ __forceinline__ PairSource pair_source(const float* __restrict__ img_a, const float* __restrict__ img_b, int H,
                                                  int W, float4 o, int x) {
    PairSource s;
    const float fax = floorf(o.x), fay = floorf(o.y), fbx = floorf(o.z), fby = floorf(o.w);
    const int xa = min(max((int)fax, 0), W - 1), ya = min(max((int)fay, 0), H - 1);
    const int xb = min(max((int)fbx, 0), W - 1), yb = min(max((int)fby, 0), H - 1);
    s.tx = make_float2(__fsub_rn(o.x, fax), __fsub_rn(o.z, fbx));
    s.ty = make_float2(__fsub_rn(o.y, fay), __fsub_rn(o.w, fby));
    s.copy_a = s.tx.x < 1e-4f && s.ty.x < 1e-4f;
    s.copy_b = s.tx.y < 1e-4f && s.ty.y < 1e-4f;
    const int ca = min(xa + x, W - 1), cb = min(xb + x, W - 1);
    s.a = img_a + (size_t)ya * W + ca;
    s.b = img_b + (size_t)yb * W + cb;
    s.last_a = H - 1 - ya;
    s.last_b = H - 1 - yb;
    s.right_a = min(xa + x + 1, W - 1) - ca;
    s.right_b = min(xb + x + 1, W - 1) - cb;
    return s;
}

// Copies rows first + step*p of whole-pixel windows. (With an address computed for every load, all of
// them ahead of the loads, the registers spill.)
template <int P>
__device__ __forceinline__ void copy_rows(const PairSource& s, int W, int first, int step, float2 (&z)[P]) {
    if (min(s.last_a, s.last_b) >= first + step * (P - 1)) {  // all rows exist: pointers step
        const float *qa = s.a + first * W, *qb = s.b + first * W;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            z[p] = make_float2(__ldg(qa), __ldg(qb));
            qa += step * W;
            qb += step * W;
        }
    } else {
#pragma unroll
        for (int p = 0; p < P; ++p)
            z[p] = make_float2(__ldg(s.a + min(first + step * p, s.last_a) * W), __ldg(s.b + min(first + step * p, s.last_b) * W));
    }
}

// Samples the P consecutive rows from row r0 of the lane's column: the lane streams down them
// carrying the row below, so each sample pair needs one new row (two loads and a pointer step per
// frame). Interleaved rows need all four taps of every sample from memory or from other lanes by
// shuffles; with the packed arithmetic and FFTs, the passes of a 2400 x 2400 pair at 75 % overlap went
// from 1.155 to 0.680 ms (96 px), 0.885 to 0.790 (48 px) and 0.770 to 0.667 (24 px), those of a 4096
// x 4096 pair from 1.83 to 1.63 (32 px) and 1.32 to 1.13 (16 px), and interpolated 128 px windows
// (2048 x 2048) from 0.773 to 0.627 (B200).
template <int N, int P>
__device__ __forceinline__ void stream_rows(PairSource s, int W, int r0, const SeparateProduct& mul, float2 (&z)[P]) {
    // When only one frame is copied, its fractions are zero and its taps stay inside the window, so
    // that no value outside of it (a NaN, say) enters; the weights 1, 0, 0, 0 then copy the pixel.
    if (s.copy_a) {
        s.tx.x = s.ty.x = 0.0f;
        s.right_a = 0;
        s.last_a = min(s.last_a, N - 1);
    }
    if (s.copy_b) {
        s.tx.y = s.ty.y = 0.0f;
        s.right_b = 0;
        s.last_b = min(s.last_b, N - 1);
    }
    const float2 one = make_float2(1.0f, 1.0f);
    const float2 ux = csub(one, s.tx), uy = csub(one, s.ty);
    const float2 w00 = cmul2(ux, uy), w01 = cmul2(s.tx, uy), w10 = cmul2(ux, s.ty), w11 = cmul2(s.tx, s.ty);
    auto blend = [&](float2 tl, float2 tr, float2 bl, float2 br) {
        float2 v = mul(w00, tl);
        v = cadd(v, mul(w01, tr));
        v = cadd(v, mul(w10, bl));
        return cadd(v, mul(w11, br));
    };
    const float* qa = s.a + min(r0, s.last_a) * W;
    const float* qb = s.b + min(r0, s.last_b) * W;
    float2 tl = make_float2(__ldg(qa), __ldg(qb)), tr = make_float2(__ldg(qa + s.right_a), __ldg(qb + s.right_b));
    if (min(s.last_a, s.last_b) >= r0 + P && (s.right_a & s.right_b)) {  // all taps exist: pointers step by the pitch
#pragma unroll
        for (int p = 0; p < P; ++p) {
            qa += W;
            qb += W;
            const float2 bl = make_float2(__ldg(qa), __ldg(qb)), br = make_float2(__ldg(qa + 1), __ldg(qb + 1));
            z[p] = blend(tl, tr, bl, br);
            tl = bl;
            tr = br;
        }
    } else {
#pragma unroll
        for (int p = 0; p < P; ++p) {
            qa += r0 + p < s.last_a ? W : 0;
            qb += r0 + p < s.last_b ? W : 0;
            const float2 bl = make_float2(__ldg(qa), __ldg(qb)),
                         br = make_float2(__ldg(qa + s.right_a), __ldg(qb + s.right_b));
            z[p] = blend(tl, tr, bl, br);
            tl = bl;
            tr = br;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Deformed windows (no counterpart in the reference, whose windows only shift): pixel (r, c) of
// the window at base position (x0, y0) (the grid origin under the placement clamp to W - n - 1,
// as a zero shift is placed by multipass.rs:207-231) is displaced by the bilinear blend D of the predictor at
// the window's four corner pixels, with u = c/(n-1), v = r/(n-1):
//   D = (1-u)(1-v) D00 + u(1-v) D10 + (1-u)v D01 + uv D11      (f32, summed left to right)
// frame A is sampled at (x0+c, y0+r) - D/2 and frame B at + D/2, bilinearly, coordinates
// clamped into the image and the tap clamped to the last full cell. Every operation rounds to
// nearest in that order (no FMA), so the samples are bit-identical to a sequential f32 evaluation.
//
// Both components of D and both frames' coordinates, weights and taps are pairs in packed
// operations. In windows whose displaced pixels all lie inside the image (the corner displacements
// bound them) nothing is clamped and nothing converted: adding 2^23 with rounding down leaves the
// whole part of a coordinate in the low bits. (A 2048 x 2048 pair's deformed passes: 32 px 197 -> 168
// us, 16 px 156 -> 150.)
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float corner_blend(float c00, float c10, float c01, float c11, float u, float v) {
    const float ou = __fsub_rn(1.0f, u), ov = __fsub_rn(1.0f, v);
    float d = __fmul_rn(__fmul_rn(ou, ov), c00);
    d = __fadd_rn(d, __fmul_rn(__fmul_rn(u, ov), c10));
    d = __fadd_rn(d, __fmul_rn(__fmul_rn(ou, v), c01));
    return __fadd_rn(d, __fmul_rn(__fmul_rn(u, v), c11));
}

__device__ __forceinline__ float2 splat(float v) { return make_float2(v, v); }

__device__ __forceinline__ float bilinear_clamped(const float* __restrict__ img, int H, int W, float px, float py) {
    px = px < 0.0f ? 0.0f : px;
    px = (float)(W - 1) < px ? (float)(W - 1) : px;
    py = py < 0.0f ? 0.0f : py;
    py = (float)(H - 1) < py ? (float)(H - 1) : py;
    const int ix = min((int)floorf(px), max(W - 2, 0)), iy = min((int)floorf(py), max(H - 2, 0));
    const float tx = __fsub_rn(px, (float)ix), ty = __fsub_rn(py, (float)iy);
    const int ix1 = min(ix + 1, W - 1), iy1 = min(iy + 1, H - 1);
    const float ux = __fsub_rn(1.0f, tx), uy = __fsub_rn(1.0f, ty);
    const float* top = img + (size_t)iy * W;
    const float* bot = img + (size_t)iy1 * W;
    float s = __fmul_rn(__fmul_rn(ux, uy), __ldg(top + ix));
    s = __fadd_rn(s, __fmul_rn(__fmul_rn(tx, uy), __ldg(top + ix1)));
    s = __fadd_rn(s, __fmul_rn(__fmul_rn(ux, ty), __ldg(bot + ix)));
    return __fadd_rn(s, __fmul_rn(__fmul_rn(tx, ty), __ldg(bot + ix1)));
}

// Samples of both frames at the points (px.x, py.x) of A and (px.y, py.y) of B, which lie in
// [0, W - 1) x [0, H - 1). Images have at most 65536 pixels a side, so unsigned 32-bit arithmetic
// gives the pixel index.
__device__ __forceinline__ float2 bilinear_inside(const float* __restrict__ img_a, const float* __restrict__ img_b, int W,
                                                  float2 px, float2 py, const SeparateProduct& mul) {
    const float2 two23 = splat(8388608.0f), one = splat(1.0f);
    const float2 mx = __fadd2_rd(px, two23), my = __fadd2_rd(py, two23);  // floor + 2^23
    const float2 tx = csub(px, csub(mx, two23)), ty = csub(py, csub(my, two23));
    const float2 ux = csub(one, tx), uy = csub(one, ty);
    const float* const a = img_a + ((__float_as_uint(my.x) - 0x4b000000u) * (unsigned)W + (__float_as_uint(mx.x) - 0x4b000000u));
    const float* const b = img_b + ((__float_as_uint(my.y) - 0x4b000000u) * (unsigned)W + (__float_as_uint(mx.y) - 0x4b000000u));
    float2 s = mul(cmul2(ux, uy), make_float2(__ldg(a), __ldg(b)));
    s = cadd(s, mul(cmul2(tx, uy), make_float2(__ldg(a + 1), __ldg(b + 1))));
    s = cadd(s, mul(cmul2(ux, ty), make_float2(__ldg(a + W), __ldg(b + W))));
    return cadd(s, mul(cmul2(tx, ty), make_float2(__ldg(a + W + 1), __ldg(b + W + 1))));
}

// The lane fills z[p] = (A, B) at column x, row r0 + p.
template <int N, int P>
__device__ __forceinline__ void sample_deformed(const float* __restrict__ img_a, const float* __restrict__ img_b, int H,
                                                int W, int x0, int y0, float4 k0, float4 k1, int x, int r0,
                                                const float* s_ramp, const SeparateProduct& mul, float2 (&z)[P]) {
    const float u = s_ramp[x], ou = __fsub_rn(1.0f, u);
    const float2 d00 = make_float2(k0.x, k0.y), d10 = make_float2(k0.z, k0.w);
    const float2 d01 = make_float2(k1.x, k1.y), d11 = make_float2(k1.z, k1.w);
    const float yf = (float)(y0 + r0);
    const float2 x2 = splat((float)(x0 + x)), sign = make_float2(-1.0f, 1.0f);
    // 0.5 |corner| bounds 0.5 |D| up to rounding; one pixel of margin covers that. (fmaxf drops a NaN,
    // so finite corners are asked for explicitly: every tap has to lie inside.)
    const float mx = 0.5f * fmaxf(fmaxf(fabsf(k0.x), fabsf(k0.z)), fmaxf(fabsf(k1.x), fabsf(k1.z))) + 1.0f;
    const float my = 0.5f * fmaxf(fmaxf(fabsf(k0.y), fabsf(k0.w)), fmaxf(fabsf(k1.y), fabsf(k1.w))) + 1.0f;
    const float sum = (k0.x + k0.y) + (k0.z + k0.w) + ((k1.x + k1.y) + (k1.z + k1.w));
    const bool inside = sum * 0.0f == 0.0f && (float)x0 >= mx && (float)(x0 + N) + mx <= (float)(W - 1) &&
                        (float)y0 >= my && (float)(y0 + N) + my <= (float)(H - 1);
    auto half = [&](float v) {  // D / 2 at the lane's column and ramp value v
        const float ov = __fsub_rn(1.0f, v);
        float2 d = mul(splat(__fmul_rn(ou, ov)), d00);
        d = cadd(d, mul(splat(__fmul_rn(u, ov)), d10));
        d = cadd(d, mul(splat(__fmul_rn(ou, v)), d01));
        d = cadd(d, mul(splat(__fmul_rn(u, v)), d11));
        return cmul2(splat(0.5f), d);
    };
    if (inside) {
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const float2 h = half(s_ramp[r0 + p]);
            z[p] = bilinear_inside(img_a, img_b, W, cfma2(splat(h.x), sign, x2),
                                   cfma2(splat(h.y), sign, splat(__fadd_rn(yf, (float)p))), mul);
        }
    } else {
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const float2 h = half(s_ramp[r0 + p]);
            const float2 px = cfma2(splat(h.x), sign, x2), py = cfma2(splat(h.y), sign, splat(__fadd_rn(yf, (float)p)));
            z[p] = make_float2(bilinear_clamped(img_a, H, W, px.x, py.x), bilinear_clamped(img_b, H, W, px.y, py.y));
        }
    }
}

// 3-point Gaussian sub-pixel offset, parabolic when a value is not positive (correlate.rs:269-281).
__device__ __forceinline__ float subpixel(float m, float c, float p) {
    float d;
    if (m > 0.0f && c > 0.0f && p > 0.0f) {
        const float lm = logf(m), lc = logf(c), lp = logf(p);
        d = __fdiv_rn(__fsub_rn(lm, lp), __fmul_rn(2.0f, __fadd_rn(__fsub_rn(lm, __fmul_rn(2.0f, lc)), lp)));
    } else {
        d = __fdiv_rn(__fsub_rn(m, p), __fmul_rn(2.0f, __fadd_rn(__fsub_rn(m, __fmul_rn(2.0f, c)), p)));
    }
    if (isfinite(d)) return fminf(fmaxf(d, -0.5f), 0.5f);
    return 0.0f;
}

}  // namespace pivb200
