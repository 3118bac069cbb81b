// Frame preparation: PreparedFrame::new (preprocess.rs:138-158) on the device.
//
//   raw u8/u16 -> f32 as v/255 or v/65535 (decode.rs:227-234); f32 frames pass through
//   optional percentile clip of the integer codes (not in the reference; see below)
//   base = max(raw - background, 0)                     preprocess.rs:140-142
//   integral tables of base for the signal mask          preprocess.rs:76-125 (exact int64 here)
//   separable Gaussian blur, radius ceil(3 sigma), clamped edges, f32 sums in kernel order
//                                                        preprocess.rs:161-195
//   local mean/std normalization over the clipped (2r+1)^2 box    preprocess.rs:199-216
//
// The blur repeats the reference's f32 operations in order (no FMA), so it is bit-exact given
// the same kernel weights. The normalization's box statistics are exact integer sums turned into
// f32 mean/std by the reference's steps (mean = s/n, var = sq/n - mean^2, sqrt) in double-float
// arithmetic (fix_stats in common.cuh; no FP64 instruction). These sums are exact where the
// reference's f64 integral image can round, and double-float carries ~48 of f64's 53 bits, so a
// result can differ from the reference's in a rounding-boundary case.
//
// Percentile clip (an addition, parity unpinned against the reference, pinned against the
// oracle): the clip code is the smallest code c with #(codes <= c) >= ceil(p/100 * H*W); codes
// above it are set to it before conversion. Found with two 256-bin histogram passes.
#include <cmath>

#include "common.cuh"
#include "kernels.h"

namespace pivb200 {

constexpr int kMaxBlurTaps = 65;  // radius <= 32
constexpr int kMaxNormRadius = 16;

struct BlurKernel {
    float w[kMaxBlurTaps];
    int radius;
};

// ------------------------------------------------------------------------------- percentile
// Two histogram passes find the clip code (u8: the second alone): level 0 counts the high bytes, level
// 1 the low bytes of the codes in the bin that holds the wanted rank. Each block counts in shared memory, and the block
// that finishes last picks the bin. Scratch: hist[256 * level ..], sel[0] = coarse bin, sel[1] = rank
// inside it, sel[2] = clip code, sel[3] = blocks finished; all zeroed before level 0.
//
// Bound by launches and by the latency of the selection, not by its bytes: as separate kernels, each
// selection walked its 256 bins in one thread (4 us). Codes come 16 bytes per load. Finer bins at level 0
// (code / 16, added up at the end) gain nothing, not even where all codes share one high byte, and cost a
// small frame 1 us (512 x 512 13.3 us against 14.3). Whole preparation with clip, per frame, B200: 1024 x
// 1024 u16 28.0 -> 16.4 us, u8 53.7 -> 12.8, 4096 x 4096 u16 65 -> 52.
constexpr int kHistThreads = 256;

template <typename CodeT, int LEVEL>
__global__ void __launch_bounds__(kHistThreads) hist_kernel(const CodeT* raw, long long n, unsigned int* hist,
                                                            unsigned int* sel, unsigned long long target) {
    constexpr int V = 16 / (int)sizeof(CodeT);
    __shared__ unsigned int h[kHistThreads];  // a bin per thread
    __shared__ bool last;
    h[threadIdx.x] = 0;
    __syncthreads();
    dependent_wait();
    let_dependents_start();
    constexpr bool kOneByte = sizeof(CodeT) == 1;  // level 1 alone, in the one coarse bin there is
    const unsigned int coarse = LEVEL && !kOneByte ? sel[0] : 0u;
    auto count = [&](unsigned int c) {
        if (LEVEL == 0)
            atomicAdd(&h[c >> 8], 1u);
        else if ((c >> 8) == coarse)
            atomicAdd(&h[c & 255u], 1u);
    };
    const long long tid = (long long)blockIdx.x * kHistThreads + threadIdx.x, stride = (long long)gridDim.x * kHistThreads;
    long long head = 0;
    if (reinterpret_cast<uintptr_t>(raw) % 16 == 0) {
        const long long nv = n / V;
        for (long long j = tid; j < nv; j += stride) {
            union {
                uint4 w;
                CodeT c[V];
            } u;
            u.w = reinterpret_cast<const uint4*>(raw)[j];
#pragma unroll
            for (int k = 0; k < V; ++k) count(u.c[k]);
        }
        head = nv * V;
    }
    for (long long i = head + tid; i < n; i += stride) count(raw[i]);
    __syncthreads();
    unsigned int* const out = hist + 256 * LEVEL;
    if (h[threadIdx.x]) atomicAdd(&out[threadIdx.x], h[threadIdx.x]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&sel[3], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // The bin that holds rank `want`: the first whose running sum reaches it.
    const unsigned long long want = LEVEL == 0 || kOneByte ? target : sel[1];
    __shared__ unsigned long long warp_sum[kHistThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long mine = *(volatile unsigned int*)&out[threadIdx.x];
    unsigned long long incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    for (int w = 0; w < warp; ++w) incl += warp_sum[w];
    const bool hit = incl >= want && (incl - mine < want || threadIdx.x == 0);
    if (hit) {
        if (LEVEL == 0) {
            sel[0] = threadIdx.x;
            sel[1] = (unsigned int)(want - (incl - mine));
        } else {
            sel[2] = (coarse << 8) | threadIdx.x;
        }
    }
    if (threadIdx.x == kHistThreads - 1) {
        sel[3] = 0;
        if (incl < want) {  // rank beyond the counts (not reached: the rank is at most n)
            if (LEVEL == 0) {
                sel[0] = 255;
                sel[1] = 0;
            } else {
                sel[2] = (coarse << 8) | 255u;
            }
        }
    }
}

// ------------------------------------------------------------------------------- conversion
// Integer codes to f32 as decode.rs:227-234 divides them: c / 255 (u8) or c / 65535 (u16),
// correctly rounded. The quotient is c * RN(1/d) corrected once by its exact residual
// (Markstein's method): q0 = RN(c r), e = fma(-q0, d, c), q = fma(e, r, q0); for these two
// divisors it equals the correctly rounded quotient for every code (checked exhaustively against
// exact rational arithmetic, and on the GPU against IEEE division).
template <typename CodeT>
struct CodeDivisor;
template <>
struct CodeDivisor<uint8_t> {
    static constexpr float d = 255.0f;
};
template <>
struct CodeDivisor<uint16_t> {
    static constexpr float d = 65535.0f;
};

__device__ __forceinline__ float div_code(float x, float d, float r) {
    const float q0 = __fmul_rn(x, r);
    return __fmaf_rn(__fmaf_rn(-q0, d, x), r, q0);
}

// The background-subtracted intensity of one sample (preprocess.rs:144-151): an integer code
// clipped to the percentile code, divided as above, then the background subtracted and clamped
// at zero. `begin()` reads the clip code on the device once per thread.
template <typename CodeT>
struct CodeSamples {
    const CodeT* raw;
    const float* bg;  // nullable
    const unsigned int* clip;  // nullable; clip[2] is the clip code
    unsigned int cl;
    float d, r;
    __device__ __forceinline__ void begin() {
        cl = clip ? clip[2] : 0xffffffffu;
        d = CodeDivisor<CodeT>::d;
        r = __frcp_rn(d);
    }
    __device__ __forceinline__ float value(unsigned int c, float b) const {
        if (c > cl) c = cl;
        float v = div_code((float)c, d, r);
        if (bg) v = fmaxf(__fsub_rn(v, b), 0.0f);
        return v;
    }
    __device__ __forceinline__ float operator()(size_t i) const { return value(raw[i], bg ? bg[i] : 0.0f); }
};

// f32 samples, background-subtracted and clamped at zero when a background is given.
struct FloatSamples {
    const float* raw;
    const float* bg;  // nullable
    __device__ __forceinline__ void begin() {}
    __device__ __forceinline__ float operator()(size_t i) const {
        float v = raw[i];
        if (bg) v = fmaxf(__fsub_rn(v, bg[i]), 0.0f);
        return v;
    }
};

// ------------------------------------------------------------------------------- max |v|
// Folds each thread's running max |v| into *out: one atomic per block of <= 256 threads. Every
// thread of the block calls it.
__device__ __forceinline__ void block_max_to(float m, unsigned int* out) {
    __shared__ float wmax[8];
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x >> 5) ? wmax[threadIdx.x] : 0.0f;
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) atomicMax(out, __float_as_uint(m));  // non-negative floats order as uints
    }
}

__global__ void maxabs_kernel(const float* __restrict__ v, long long n, unsigned int* out) {
    float m = 0.0f;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        m = fmaxf(m, fabsf(v[i]));
    block_max_to(m, out);
}

// ------------------------------------------------------------------------------- conversion kernels
// Streams codes 16 bytes per load (8 u16 or 16 u8) when the buffers are 16-byte aligned; the
// rest of the frame (or an unaligned one) one code at a time. With a non-null `maxout` the kernel
// also folds max |value| into it (the scale of the fixed-point sums), which saves a pass over the
// frame. Launched with 256 threads.
template <typename CodeT>
__device__ __forceinline__ float convert_codes(const CodeT* raw, long long n, const float* bg,
                                               const unsigned int* clip, float* out, long long tid,
                                               long long stride) {
    constexpr int V = 16 / (int)sizeof(CodeT);
    CodeSamples<CodeT> src{raw, bg, clip, 0u, 0.0f, 0.0f};
    src.begin();
    float m = 0.0f;
    auto value = [&](unsigned int c, float b) {
        const float v = src.value(c, b);
        m = fmaxf(m, fabsf(v));
        return v;
    };
    long long head = 0;
    const bool aligned = (reinterpret_cast<uintptr_t>(raw) | reinterpret_cast<uintptr_t>(out) |
                          reinterpret_cast<uintptr_t>(bg)) % 16 == 0;
    if (aligned) {
        const long long nv = n / V;
        for (long long j = tid; j < nv; j += stride) {
            union {
                uint4 w;
                CodeT c[V];
            } u;
            u.w = reinterpret_cast<const uint4*>(raw)[j];
#pragma unroll
            for (int k = 0; k < V; k += 4) {
                float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
                if (bg) b = *reinterpret_cast<const float4*>(bg + j * V + k);
                float4 o;
                o.x = value(u.c[k], b.x);
                o.y = value(u.c[k + 1], b.y);
                o.z = value(u.c[k + 2], b.z);
                o.w = value(u.c[k + 3], b.w);
                *reinterpret_cast<float4*>(out + j * V + k) = o;
            }
        }
        head = nv * V;
    }
    for (long long i = head + tid; i < n; i += stride) out[i] = value(raw[i], bg ? bg[i] : 0.0f);
    return m;
}

template <typename CodeT>
__global__ void convert_kernel(const CodeT* raw, long long n, const float* bg,
                               const unsigned int* clip, float* out, unsigned int* maxout) {
    dependent_wait();
    let_dependents_start();
    const float m = convert_codes(raw, n, bg, clip, out, (long long)blockIdx.x * blockDim.x + threadIdx.x,
                                  (long long)gridDim.x * blockDim.x);
    if (maxout) block_max_to(m, maxout);
}

// Several frames of one size and type in one launch: `per` blocks each. (Frame by frame, the 65 frames
// of a 64-pair batch of 1280 x 800 u16 took 4.8 us each, launch gaps included; together they are bound
// by their 6 bytes per pixel.)
struct ConvertBatch {
    long long n;
    int per;
    const void* raw[kMaxBatch];
    float* out[kMaxBatch];
    const float* bg;
};

template <typename CodeT>
__global__ void convert_frames_kernel(const __grid_constant__ ConvertBatch b) {
    dependent_wait();
    let_dependents_start();
    const int f = (int)blockIdx.x / b.per;
    const long long tid = (long long)(blockIdx.x - f * b.per) * blockDim.x + threadIdx.x;
    convert_codes(static_cast<const CodeT*>(b.raw[f]), b.n, b.bg, nullptr, b.out[f], tid, (long long)b.per * blockDim.x);
}

__global__ void convert_f32_kernel(const float* raw, long long n, const float* bg,
                                   float* out, unsigned int* maxout) {
    dependent_wait();
    let_dependents_start();
    const FloatSamples src{raw, bg};
    float m = 0.0f;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float v = src((size_t)i);
        m = fmaxf(m, fabsf(v));
        out[i] = v;
    }
    if (maxout) block_max_to(m, maxout);
}

// ------------------------------------------------------------------------------- integral tables
// T[y][x] = sum of q(v) over the rows above y and the columns left of x, for q = value and square,
// in strips of kStripRows rows: the strip kernel writes each strip's own 2-D prefix (one block per
// strip, every pixel read once), and the scan kernel turns every kStripRows-th row into the full
// prefix, in place. A reader adds the full row above an entry's strip (table_at in common.cuh), so
// no third pass over the tables is needed. Integer sums: any order gives the same bits.
//
// Writing 16 bytes per pixel bounds both tables. Two passes over all rows (a running sum down every
// column, W / 128 blocks) left most SMs without a block and took 236 us of a 1437 x 1003 frame's
// 310 us preparation; a masked pair of that size went from 667 to 394 us in all (B200).
constexpr int kStripThreads = 512;
constexpr int kStripWarps = kStripThreads / 32;

__device__ __forceinline__ long long warp_scan(long long v, int lane) {
    for (int o = 1; o < 32; o <<= 1) {
        const long long u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

__global__ void __launch_bounds__(kStripThreads) integral_strip_kernel(const float* v, int H, int W,
                                                                       long long* sum,
                                                                       long long* sumsq,
                                                                       const unsigned int* maxbits, int* scales) {
    constexpr int R = kStripRows;
    dependent_wait();
    let_dependents_start();
    static_assert(2 * R == kStripWarps, "one warp scans the warp totals of each row of each table");
    const FixScale fs = fix_scale(__uint_as_float(*maxbits), (long long)H * W);
    const int y0 = blockIdx.x * R, rows = min(R, H - y0);
    const int stride = W + 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ long long tot[kStripWarps][2 * R + 1];  // [warp][row of table 1, row of table 2]
    if (blockIdx.x == 0) {
        if (tid == 0) {
            scales[0] = fs.s1;
            scales[1] = fs.s2;
        }
        for (int x = tid; x <= W; x += kStripThreads) sum[x] = sumsq[x] = 0;
    }
    if (tid < 2 * rows) (tid < rows ? sum : sumsq)[(size_t)(y0 + 1 + tid % rows) * stride] = 0;
    long long carry = 0;  // warp j: total of value row j over the columns before `base`
    for (int base = 0; base < W; base += kStripThreads) {
        const int x = base + tid;
        long long a[R], b[R];  // running sums down the column, then 2-D prefixes within the warp
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float f = (x < W && r < rows) ? v[(size_t)(y0 + r) * W + x] : 0.0f;
            a[r] = fix_q1(f, fs) + (r ? a[r - 1] : 0);
            b[r] = fix_q2(f, fs) + (r ? b[r - 1] : 0);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            a[r] = warp_scan(a[r], lane);
            b[r] = warp_scan(b[r], lane);
            if (lane == 31) {
                tot[warp][r] = a[r];
                tot[warp][R + r] = b[r];
            }
        }
        __syncthreads();
        {
            const long long t = lane < kStripWarps ? tot[lane][warp] : 0;
            const long long incl = warp_scan(t, lane);
            if (lane < kStripWarps) tot[lane][warp] = carry + incl - t;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncthreads();
        if (x < W) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (r < rows) {
                    const size_t o = (size_t)(y0 + 1 + r) * stride + x + 1;
                    sum[o] = a[r] + tot[warp][r];
                    sumsq[o] = b[r] + tot[warp][R + r];
                }
        }
        __syncthreads();
    }
}

// Rows kStripRows, 2 kStripRows, ... of both tables become running sums down each column: 32
// columns and 32 groups of strips per block.
__global__ void __launch_bounds__(1024) integral_scan_kernel(int H, int W, long long* sum, long long* sumsq) {
    dependent_wait();
    let_dependents_start();
    const int strips = H / kStripRows;  // full strips; a last partial one has no row to update
    const int stride = W + 1;
    const int tx = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int x = blockIdx.x * 32 + tx;
    const int per = (strips + 31) / 32, s0 = min(g * per, strips), s1 = min(s0 + per, strips);
    __shared__ long long part[2][32][32];
    long long* const t[2] = {sum, sumsq};
    long long acc[2] = {0, 0};
    if (x <= W)
        for (int s = s0; s < s1; ++s)
            for (int k = 0; k < 2; ++k) acc[k] += t[k][(size_t)(s + 1) * kStripRows * stride + x];
    for (int k = 0; k < 2; ++k) part[k][g][tx] = acc[k];
    __syncthreads();
    for (int k = 0; k < 2; ++k) {
        acc[k] = 0;
        for (int j = 0; j < g; ++j) acc[k] += part[k][j][tx];
    }
    if (x <= W)
        for (int s = s0; s < s1; ++s)
            for (int k = 0; k < 2; ++k) {
                long long* e = t[k] + (size_t)(s + 1) * kStripRows * stride + x;
                acc[k] += *e;
                *e = acc[k];
            }
}

// ------------------------------------------------------------------------------- blur
constexpr int BT_X = 32, BT_Y = 32;
constexpr int kBlurThreads = 256;  // the blur's launch width; its loops stride by it

// The tile load reads samples through `Src`: the previous stage's f32 image, or (when nothing
// else needs the background-subtracted image) the raw frame decoded on the fly, which saves the
// conversion kernel and its H x W f32 round trip. With a non-null `maxout` the kernel also folds
// max |output| into *maxout for the local normalisation's fixed-point scale (launched with 256
// threads).
// RC > 0 fixes the radius at compile time (the taps unroll; the summation order is unchanged);
// RC = 0 takes it from k.
template <typename Src, int RC>
__global__ void blur_kernel(Src src, int H, int W, const BlurKernel k, float* out,
                            unsigned int* maxout) {
    extern __shared__ float sm[];
    dependent_wait();
    let_dependents_start();
    src.begin();
    const int R = RC > 0 ? RC : k.radius;
    const int TW = BT_X + 2 * R, TH = BT_Y + 2 * R;
    float* tin = sm;             // TH x TW
    float* trow = sm + TH * TW;  // TH x BT_X
    const int gx0 = blockIdx.x * BT_X, gy0 = blockIdx.y * BT_Y;
    // i / TW as a multiply-high by ceil(2^32 / TW), exact for i * TW < 2^32.
    const unsigned int tw_magic = 0xffffffffu / (unsigned int)TW + 1u;
#pragma unroll 2
    for (int i = threadIdx.x; i < TH * TW; i += kBlurThreads) {
        const int ty = (int)__umulhi((unsigned int)i, tw_magic), tx = i - ty * TW;
        const int gy = min(max(gy0 + ty - R, 0), H - 1);
        const int gx = min(max(gx0 + tx - R, 0), W - 1);
        tin[i] = src((size_t)gy * W + gx);
    }
    __syncthreads();
    // Row pass over every tile row (vertical halo included): sum in kernel order from -0.0.
#pragma unroll
    for (int i = threadIdx.x; i < TH * BT_X; i += kBlurThreads) {
        const int ty = i / BT_X, tx = i % BT_X;
        float s = -0.0f;
#pragma unroll
        for (int j = 0; j <= 2 * R; ++j) s = __fadd_rn(s, __fmul_rn(k.w[j], tin[ty * TW + tx + j]));
        trow[i] = s;
    }
    __syncthreads();
    // Column pass: out starts at 0.0 and accumulates kernel terms in order (preprocess.rs:186-193).
    float m = 0.0f;
#pragma unroll
    for (int i = threadIdx.x; i < BT_X * BT_Y; i += kBlurThreads) {
        const int ty = i / BT_X, tx = i % BT_X;
        const int gx = gx0 + tx, gy = gy0 + ty;
        if (gx >= W || gy >= H) continue;
        float o = 0.0f;
#pragma unroll
        for (int j = 0; j <= 2 * R; ++j) o = __fadd_rn(o, __fmul_rn(k.w[j], trow[(ty + j) * BT_X + tx]));
        out[(size_t)gy * W + gx] = o;
        m = fmaxf(m, fabsf(o));
    }
    if (maxout) block_max_to(m, maxout);
}

// ------------------------------------------------------------------------------- normalize
// Bound by instructions and shared-memory wavefronts (22 eight-byte accesses per output), not by its
// 8 bytes per pixel. Tiles of 32 x 24 with 8 outputs per thread in the row pass and 3 in the column
// pass keep both passes to one round of the 256 threads; 32 x 32 tiles with runs of 4 took two rounds
// in the row pass. With the statistics above (fix_stats_fast), blur and normalisation of a 1920 x 1080
// u8 frame went from 48.4 to 38.9 us (B200); 32 x 16 tiles 41.0, 32 x 32 with 320 threads 39.7.
constexpr int NT_X = 32, NT_Y = 24;
constexpr int NT_RUN = 3;  // output rows per thread in the column pass (256 threads = 32 columns x 8 runs)
constexpr int NT_XRUN = 8;  // outputs per thread in the row pass
constexpr int NT_HW = NT_X + 1;  // row stride of the row-pass sums (odd, in 8-byte words)
constexpr int kNormThreads = 256;  // the launch width; the loops stride by it

// RC > 0 fixes the radius at compile time; RC = 0 takes it from r_arg.
template <int RC>
__global__ void normalize_kernel(const float* src, int H, int W, int r_arg, float eps,
                                 const unsigned int* maxbits, float* out) {
    extern __shared__ long long smq[];
    dependent_wait();
    let_dependents_start();
    const int r = RC > 0 ? RC : r_arg;
    const int TW = NT_X + 2 * r, TH = NT_Y + 2 * r;
    // Row strides in 8-byte words are odd (QW, NT_HW), so 16 lanes on 16 consecutive rows of one
    // column hit 16 different bank pairs.
    const int QW = TW | 1;
    long long* q1 = smq;                 // TH x QW
    long long* q2 = q1 + TH * QW;        // TH x QW
    long long* h1 = q2 + TH * QW;        // TH x NT_HW
    long long* h2 = h1 + TH * NT_HW;     // TH x NT_HW
    const FixScale fs = fix_scale(__uint_as_float(*maxbits), (long long)(2 * r + 1) * (2 * r + 1));
    const int gx0 = blockIdx.x * NT_X, gy0 = blockIdx.y * NT_Y;
    // i / TW as a multiply-high by ceil(2^32 / TW): exact while i * TW < 2^32, which the tile's
    // shared-memory size guarantees by far.
    const unsigned int tw_magic = 0xffffffffu / (unsigned int)TW + 1u;
#pragma unroll 2
    for (int i = threadIdx.x; i < TH * TW; i += kNormThreads) {
        const int ty = (int)__umulhi((unsigned int)i, tw_magic), tx = i - ty * TW;
        const int gy = gy0 + ty - r, gx = gx0 + tx - r;
        long long a = 0, b = 0;
        if (gy >= 0 && gy < H && gx >= 0 && gx < W) {
            const float f = src[(size_t)gy * W + gx];
            a = fix_q1(f, fs);
            b = fix_q2(f, fs);
        }
        q1[ty * QW + tx] = a;
        q2[ty * QW + tx] = b;
    }
    __syncthreads();
    // Row pass: each thread slides a (2r+1)-tap window along NT_XRUN outputs of one tile row;
    // consecutive threads take consecutive rows. The sums are exact integers, so sliding gives
    // the same totals as summing afresh.
    const unsigned int th_magic = 0xffffffffu / (unsigned int)TH + 1u;
    for (int i = threadIdx.x; i < TH * (NT_X / NT_XRUN); i += kNormThreads) {
        const int run = (int)__umulhi((unsigned int)i, th_magic), row = i - run * TH;
        const long long* p1 = q1 + row * QW + run * NT_XRUN;
        const long long* p2 = q2 + row * QW + run * NT_XRUN;
        long long* o1 = h1 + row * NT_HW + run * NT_XRUN;
        long long* o2 = h2 + row * NT_HW + run * NT_XRUN;
        // Two accumulators per table shorten the first sum's add chains.
        long long a0 = p1[0], b0 = p2[0], a1 = 0, b1 = 0;
        int j = 1;
#pragma unroll
        for (; j + 1 <= 2 * r; j += 2) {
            a0 += p1[j];
            a1 += p1[j + 1];
            b0 += p2[j];
            b1 += p2[j + 1];
        }
        if (j <= 2 * r) {
            a0 += p1[j];
            b0 += p2[j];
        }
        long long a = a0 + a1, b = b0 + b1;
        o1[0] = a;
        o2[0] = b;
#pragma unroll
        for (int k = 1; k < NT_XRUN; ++k) {
            a += p1[k + 2 * r] - p1[k - 1];
            b += p2[k + 2 * r] - p2[k - 1];
            o1[k] = a;
            o2[k] = b;
        }
    }
    __syncthreads();
    // Column pass: each thread slides a (2r+1)-row window down NT_RUN output rows of one column
    // (the sums are exact integers, so sliding gives the same totals as summing afresh).
    const bool fast = fix_stats_fast_ok(fs);
    const float p1 = pow2f(fast ? -fs.s1 : 0), p2 = pow2f(fast ? -fs.s2 : 0);
    const float full = (float)((2 * r + 1) * (2 * r + 1)), full_rc = __frcp_rn(full);
    for (int i = threadIdx.x; i < NT_X * (NT_Y / NT_RUN); i += kNormThreads) {
        const int tx = i % NT_X, ty0 = (i / NT_X) * NT_RUN;
        const int gx = gx0 + tx;
        long long a = 0, b = 0;
#pragma unroll
        for (int j = 0; j <= 2 * r; ++j) {
            a += h1[(ty0 + j) * NT_HW + tx];
            b += h2[(ty0 + j) * NT_HW + tx];
        }
#pragma unroll
        for (int k = 0; k < NT_RUN; ++k) {
            const int ty = ty0 + k, gy = gy0 + ty;
            if (k > 0) {
                a += h1[(ty + 2 * r) * NT_HW + tx] - h1[(ty - 1) * NT_HW + tx];
                b += h2[(ty + 2 * r) * NT_HW + tx] - h2[(ty - 1) * NT_HW + tx];
            }
            if (gx >= W || gy >= H) continue;
            const int x0 = max(gx - r, 0), x1 = min(gx + r + 1, W);
            const int y0 = max(gy - r, 0), y1 = min(gy + r + 1, H);
            const int count = (x1 - x0) * (y1 - y0);
            float mean, sd;
            if (fast) {
                const bool whole = count == (2 * r + 1) * (2 * r + 1);
                fix_stats_fast(a, b, p1, p2, whole ? full : (float)count, whole ? full_rc : __frcp_rn((float)count), &mean, &sd);
            } else {
                fix_stats(a, b, fs, (float)count, &mean, &sd);
            }
            const float v = src[(size_t)gy * W + gx];
            out[(size_t)gy * W + gx] = __fdiv_rn(__fsub_rn(v, mean), __fadd_rn(sd, eps));
        }
    }
}

// ------------------------------------------------------------------------------- drivers
// Launches the blur through sample source `src`: the radius-3 instantiation (sigma 1, the
// default) or the general one, which is opted into more than 48 KB of dynamic shared memory when
// its tile needs it.
template <typename Src>
static cudaError_t run_blur(dim3 grid, size_t sm, cudaStream_t s, const Src& src, int H, int W, const BlurKernel& k,
                            float* dst, unsigned int* mx) {
    if (k.radius == 3) {
        return launch_dependent(blur_kernel<Src, 3>, grid, kBlurThreads, sm, s, src, H, W, k, dst, mx);
    }
    if (sm > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(blur_kernel<Src, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
    }
    return launch_dependent(blur_kernel<Src, 0>, grid, kBlurThreads, sm, s, src, H, W, k, dst, mx);
}

static int grid_for(long long n) {
    long long b = (n + 255) / 256;
    if (b > 148 * 16) b = 148 * 16;
    if (b < 1) b = 1;
    return (int)b;
}

// ------------------------------------------------------------------------------- reference tables
// IntegralImage's f64 summed-area tables (preprocess.rs:76-103), handed over by a caller that
// prepared its frames on the host, are turned into this library's int64 fixed-point tables in
// place (each f64 entry's 8 bytes become its int64 entry): q = round(T * 2^s), with s chosen per
// table from its largest |entry| so that every entry and every 4-term box difference fits in
// int64. Only integer operations on the f64 bit patterns are used (no FP64 instruction). Entries
// whose f64 spacing is below 2^-s are rounded to the nearest multiple of 2^-s (ties to even);
// box sums are then exact differences of these entries.
__global__ void table_maxbits_kernel(const unsigned long long* __restrict__ t, long long n, unsigned long long* out,
                                     unsigned int* nonfinite) {
    unsigned long long m = 0;
    bool bad = false;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long b = t[i] & 0x7fffffffffffffffull;
        if ((b >> 52) == 0x7ffull) bad = true;
        else m = b > m ? b : m;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long v = __shfl_xor_sync(0xffffffffu, m, o);
        m = v > m ? v : m;
    }
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(nonfinite, 1u);
}

// Scale exponent s with max|T| * 2^s < 2^61 (headroom for the box differences).
__device__ __forceinline__ int table_scale(unsigned long long maxbits) {
    if (!maxbits) return 0;
    const int e = (int)(maxbits >> 52) - 1022;  // max|T| < 2^e
    return 61 - e;
}

__device__ __forceinline__ long long f64_bits_to_fixed(unsigned long long bits, int s) {
    const bool neg = bits >> 63;
    const int be = (int)((bits >> 52) & 0x7ff);
    if (be == 0x7ff) return 0;  // non-finite: reported through the flag, never used
    unsigned long long m = bits & 0x000fffffffffffffull;
    int k;  // |value| = m * 2^k
    if (be) {
        m |= 1ull << 52;
        k = be - 1075;
    } else {
        k = -1074;
    }
    k += s;
    unsigned long long q;
    if (k >= 0) {
        q = m << k;  // the scale keeps |value| * 2^s below 2^61
    } else if (-k >= 64) {
        q = 0;  // below half a quantum
    } else {
        const int r = -k;
        q = m >> r;
        const unsigned long long rem = m & ((1ull << r) - 1), half = 1ull << (r - 1);
        if (rem > half || (rem == half && (q & 1))) ++q;
    }
    return neg ? -(long long)q : (long long)q;
}

__global__ void table_to_fixed_kernel(unsigned long long* t, long long n, const unsigned long long* maxbits,
                                      int* scale_out) {
    const int s = table_scale(*maxbits);
    if (blockIdx.x == 0 && threadIdx.x == 0) *scale_out = s;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        t[i] = (unsigned long long)f64_bits_to_fixed(t[i], s);
}

// The tables from `base` and its max |v| in *maxbits.
static cudaError_t run_tables(const float* base, int H, int W, long long* sum, long long* sumsq, int* scales,
                              const unsigned int* maxbits, cudaStream_t s, int* launches) {
    cudaError_t e = launch_dependent(integral_strip_kernel, (H + kStripRows - 1) / kStripRows, kStripThreads, 0, s, base, H, W,
                                     sum, sumsq, maxbits, scales);
    if (e == cudaSuccess) e = launch_dependent(integral_scan_kernel, (W + 1 + 31) / 32, 1024, 0, s, H, W, sum, sumsq);
    if (launches) *launches += 2;
    return e;
}

cudaError_t launch_stats(const float* base, int H, int W, long long* sum, long long* sumsq, int* scales,
                         unsigned int* maxbits, cudaStream_t s, int* launches) {
    const long long n = (long long)H * W;
    cudaError_t e = cudaMemsetAsync(maxbits, 0, sizeof(unsigned int), s);
    if (e != cudaSuccess) return e;
    maxabs_kernel<<<grid_for(n), 256, 0, s>>>(base, n, maxbits);
    if (launches) *launches += 1;
    return run_tables(base, H, W, sum, sumsq, scales, maxbits, s, launches);
}

// Blur weights exactly as preprocess.rs:162-168 computes them (f32 exp of an f32 argument,
// normalised by their f32 sum in order).
static BlurKernel make_blur(float sigma) {
    BlurKernel k{};
    const int radius = (int)std::max(std::ceil(3.0f * sigma), 1.0f);
    k.radius = radius;
    float total = 0.0f;
    for (int i = -radius; i <= radius; ++i) {
        const float v = std::exp(-(float)(i * i) / (2.0f * sigma * sigma));
        k.w[i + radius] = v;
    }
    for (int j = 0; j <= 2 * radius; ++j) total += k.w[j];
    for (int j = 0; j <= 2 * radius; ++j) k.w[j] /= total;
    return k;
}

cudaError_t launch_tables_to_fixed(long long* sum, long long* sumsq, int H, int W, int* scales,
                                   unsigned long long* maxbits2, unsigned int* nonfinite, cudaStream_t s, int* launches) {
    const long long n = (long long)(H + 1) * (W + 1);
    cudaError_t e = cudaMemsetAsync(maxbits2, 0, 2 * sizeof(unsigned long long), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(nonfinite, 0, sizeof(unsigned int), s);
    if (e != cudaSuccess) return e;
    unsigned long long* t1 = reinterpret_cast<unsigned long long*>(sum);
    unsigned long long* t2 = reinterpret_cast<unsigned long long*>(sumsq);
    table_maxbits_kernel<<<grid_for(n), 256, 0, s>>>(t1, n, maxbits2, nonfinite);
    table_maxbits_kernel<<<grid_for(n), 256, 0, s>>>(t2, n, maxbits2 + 1, nonfinite);
    table_to_fixed_kernel<<<grid_for(n), 256, 0, s>>>(t1, n, maxbits2, scales);
    table_to_fixed_kernel<<<grid_for(n), 256, 0, s>>>(t2, n, maxbits2 + 1, scales + 1);
    if (launches) *launches += 4;
    return cudaGetLastError();
}

cudaError_t launch_convert_frames(const void* const* raw, float* const* out, int count, int H, int W, int raw_type,
                                  const float* background, cudaStream_t s, int* launches) {
    for (int off = 0; off < count; off += kMaxBatch) {
        ConvertBatch b{};
        const int m = std::min(count - off, kMaxBatch);
        b.n = (long long)H * W;
        // 16 bytes of codes per thread and turn; few frames get more blocks each
        const long long want = (b.n * (raw_type == RAW_U8 ? 1 : 2) / 16 + 255) / 256;
        b.per = (int)std::max<long long>(1, std::min<long long>(want, std::max(148 * 16 / m, 64)));
        for (int i = 0; i < m; ++i) {
            b.raw[i] = raw[off + i];
            b.out[i] = out[off + i];
        }
        b.bg = background;
        cudaError_t e = cudaErrorInvalidValue;
        if (raw_type == RAW_U8)
            e = launch_dependent(convert_frames_kernel<uint8_t>, (unsigned)(m * b.per), 256, 0, s, b);
        else if (raw_type == RAW_U16)
            e = launch_dependent(convert_frames_kernel<uint16_t>, (unsigned)(m * b.per), 256, 0, s, b);
        if (e != cudaSuccess) return e;
        if (launches) ++*launches;
    }
    return cudaSuccess;
}

cudaError_t launch_prepare(const PrepParams& p, cudaStream_t s, int* launches) {
    const long long n = (long long)p.H * p.W;
    cudaError_t e = cudaSuccess;
    int nl = 0;
    const unsigned int* clip = nullptr;
    if (p.clip_percentile_on && (p.raw_type == RAW_U8 || p.raw_type == RAW_U16)) {
        e = cudaMemsetAsync(p.hist, 0, sizeof(unsigned int) * (512 + 4), s);
        if (e != cudaSuccess) return e;
        double pc = std::min(std::max(p.clip_percentile, 0.0), 100.0);
        unsigned long long target = (unsigned long long)std::ceil(pc / 100.0 * (double)n);
        if (target < 1) target = 1;
        unsigned int* sel = p.hist + 512;
        const int blocks = (int)std::min<long long>(grid_for(n), 148 * 2);
        if (p.raw_type == RAW_U16) {
            const uint16_t* raw = (const uint16_t*)p.raw;
            e = launch_dependent(hist_kernel<uint16_t, 0>, blocks, kHistThreads, 0, s, raw, n, p.hist, sel, target);
            if (e == cudaSuccess)
                e = launch_dependent(hist_kernel<uint16_t, 1>, blocks, kHistThreads, 0, s, raw, n, p.hist, sel, target);
        } else {
            e = launch_dependent(hist_kernel<uint8_t, 1>, blocks, kHistThreads, 0, s, (const uint8_t*)p.raw, n, p.hist, sel, target);
        }
        if (e != cudaSuccess) return e;
        nl += p.raw_type == RAW_U16 ? 2 : 1;
        clip = sel;
    }
    const bool blur = p.smooth_sigma > 0.0f;
    const bool norm = p.normalize_radius > 0;
    // base goes straight to `image` when no further stage follows. When the blur follows and no
    // integral tables are wanted, the blur decodes the raw samples itself and base is not written.
    float* base = p.base;
    const bool fused = blur && !p.build_stats;
    // max |base| for the tables' scale, and for the normalisation's when it reads base itself: both
    // find it in words the conversion fills.
    const bool base_max = p.build_stats || (norm && !blur);
    if (base_max || norm) {
        e = cudaMemsetAsync(p.maxbits, 0, 2 * sizeof(unsigned int), s);
        if (e != cudaSuccess) return e;
    }
    unsigned int* bmax = base_max ? p.maxbits : nullptr;
    if (!fused) switch (p.raw_type) {
        case RAW_U8:
            e = launch_dependent(convert_kernel<uint8_t>, grid_for(n), 256, 0, s, (const uint8_t*)p.raw, n, p.background, clip, base, bmax);
            break;
        case RAW_U16:
            e = launch_dependent(convert_kernel<uint16_t>, grid_for(n), 256, 0, s, (const uint16_t*)p.raw, n, p.background, clip, base, bmax);
            break;
        default:
            e = launch_dependent(convert_f32_kernel, grid_for(n), 256, 0, s, (const float*)p.raw, n, p.background, base, bmax);
            break;
    }
    if (e != cudaSuccess) return e;
    if (!fused) nl += 1;
    if (p.build_stats) {
        e = run_tables(base, p.H, p.W, p.sum, p.sumsq, p.scales, p.maxbits, s, &nl);
        if (e != cudaSuccess) return e;
    }
    const float* cur = base;
    if (blur) {
        const BlurKernel k = make_blur(p.smooth_sigma);
        if (k.radius > (kMaxBlurTaps - 1) / 2) return cudaErrorInvalidValue;
        const int R = k.radius;
        const size_t sm = sizeof(float) * ((size_t)(BT_Y + 2 * R) * (BT_X + 2 * R) + (size_t)(BT_Y + 2 * R) * BT_X);
        float* dst = norm ? p.tmp : p.image;
        unsigned int* mx = norm ? p.maxbits + 1 : nullptr;
        dim3 grid((p.W + BT_X - 1) / BT_X, (p.H + BT_Y - 1) / BT_Y);
        if (!fused) {
            e = run_blur(grid, sm, s, FloatSamples{cur, nullptr}, p.H, p.W, k, dst, mx);
        } else if (p.raw_type == RAW_U8) {
            e = run_blur(grid, sm, s, CodeSamples<uint8_t>{(const uint8_t*)p.raw, p.background, clip, 0u, 0.0f, 0.0f},
                         p.H, p.W, k, dst, mx);
        } else if (p.raw_type == RAW_U16) {
            e = run_blur(grid, sm, s, CodeSamples<uint16_t>{(const uint16_t*)p.raw, p.background, clip, 0u, 0.0f, 0.0f},
                         p.H, p.W, k, dst, mx);
        } else {
            e = run_blur(grid, sm, s, FloatSamples{(const float*)p.raw, p.background}, p.H, p.W, k, dst, mx);
        }
        if (e != cudaSuccess) return e;
        nl += 1;
        cur = dst;
    }
    if (norm) {
        const int r = p.normalize_radius;
        if (r > kMaxNormRadius) return cudaErrorInvalidValue;
        const unsigned int* const mx = blur ? p.maxbits + 1 : p.maxbits;  // max |cur|
        const size_t sm = sizeof(long long) * (2 * (size_t)(NT_Y + 2 * r) * ((NT_X + 2 * r) | 1) + 2 * (size_t)(NT_Y + 2 * r) * NT_HW);
        dim3 grid((p.W + NT_X - 1) / NT_X, (p.H + NT_Y - 1) / NT_Y);
        if (r == 4) {  // the default radius: 37.9 KB of tile, under the 48 KB default
            e = launch_dependent(normalize_kernel<4>, grid, kNormThreads, sm, s, cur, p.H, p.W, r, p.normalize_eps, mx, p.image);
        } else {
            if (sm > 48 * 1024) {
                e = cudaFuncSetAttribute(normalize_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
                if (e != cudaSuccess) return e;
            }
            e = launch_dependent(normalize_kernel<0>, grid, kNormThreads, sm, s, cur, p.H, p.W, r, p.normalize_eps, mx, p.image);
        }
        if (e != cudaSuccess) return e;
        nl += 1;
        cur = p.image;
    }
    if (cur != p.image) {
        e = cudaMemcpyAsync(p.image, cur, sizeof(float) * n, cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) return e;
    }
    if (launches) *launches += nl;
    return cudaGetLastError();
}

}  // namespace pivb200
