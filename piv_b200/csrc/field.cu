// Window placement, signal mask, validation and summary kernels.
//
// These stages are bit-exact against the reference: every f32 operation is written with the
// round-to-nearest intrinsics in the reference's order (Rust never contracts into FMA), and the
// translation unit is additionally compiled with --fmad=false.
//   placement:  PivAnalyzer::pass (multipass.rs:204-231) with VectorField::sample (field.rs:56-81)
//   mask:       has_signal (multipass.rs:233-241) over IntegralImage::stats (preprocess.rs:114-125)
//   validation: validate (validate.rs:51-130), collect_neighbours / residual / median (:133-170)
#include <cmath>

#include "common.cuh"
#include "kernels.h"

namespace pivb200 {

__device__ __forceinline__ float grid_center(int origin0, int i, int step, int window) {
    // grid.rs:60-66: (origin0 + i*step) as f32 + (window as f32 - 1) / 2
    return __fadd_rn((float)(origin0 + i * step), __fdiv_rn(__fsub_rn((float)window, 1.0f), 2.0f));
}

// VectorField::sample (field.rs:56-81).
__device__ float2 sample_predictor(const float* dx, const float* dy, const GridP& g, float x,
                                   float y) {
    const float fx = rclamp(__fdiv_rn(__fsub_rn(x, grid_center(g.x0, 0, g.step, g.window)), (float)g.step), 0.0f,
                            (float)(g.nx - 1));
    const float fy = rclamp(__fdiv_rn(__fsub_rn(y, grid_center(g.y0, 0, g.step, g.window)), (float)g.step), 0.0f,
                            (float)(g.ny - 1));
    const int ix = (int)floorf(fx), iy = (int)floorf(fy);
    const float tx = __fsub_rn(fx, (float)ix), ty = __fsub_rn(fy, (float)iy);
    const int ix1 = min(ix + 1, g.nx - 1), iy1 = min(iy + 1, g.ny - 1);
    const int rr[4] = {iy, iy, iy1, iy1};
    const int cc[4] = {ix, ix1, ix, ix1};
    const float ux = __fsub_rn(1.0f, tx), uy = __fsub_rn(1.0f, ty);
    const float ww[4] = {__fmul_rn(ux, uy), __fmul_rn(tx, uy), __fmul_rn(ux, ty), __fmul_rn(tx, ty)};
    float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float u = dx[rr[j] * g.nx + cc[j]], v = dy[rr[j] * g.nx + cc[j]];
        if (ww[j] > 0.0f && isfinite(u) && isfinite(v)) {
            a0 = __fadd_rn(a0, __fmul_rn(ww[j], u));
            a1 = __fadd_rn(a1, __fmul_rn(ww[j], v));
            a2 = __fadd_rn(a2, ww[j]);
        }
    }
    if (a2 > 0.0f) return make_float2(__fdiv_rn(a0, a2), __fdiv_rn(a1, a2));
    return make_float2(0.0f, 0.0f);
}

// The `place` closure (multipass.rs:224-231): returns (a0, a0 + shift).
__device__ __forceinline__ float2 place1(int origin, float shift, float mx) {
    const float s = rclamp(shift, -mx, mx);
    const float a0 = rclamp(__fsub_rn((float)origin, __fdiv_rn(s, 2.0f)), fmaxf(-s, 0.0f), fminf(__fsub_rn(mx, s), mx));
    return make_float2(a0, __fadd_rn(a0, s));
}

__device__ __forceinline__ long long rect(const StatsView& s, const long long* t, int x0, int y0, int x1, int y1) {
    const int stride = s.W + 1;
    if (s.strips)
        return table_at(t, stride, y1, x1) - table_at(t, stride, y0, x1) - table_at(t, stride, y1, x0) +
               table_at(t, stride, y0, x0);
    return t[(size_t)y1 * stride + x1] - t[(size_t)y0 * stride + x1] - t[(size_t)y1 * stride + x0] + t[(size_t)y0 * stride + x0];
}

// has_signal (multipass.rs:233-241): stats of the n x n box at the rounded origin.
__device__ bool has_signal(const StatsView& s, float x, float y, int n, float min_mean, float min_std) {
    int bx = (int)roundf(x), by = (int)roundf(y);  // f32::round: half away from zero
    bx = min(max(bx, 0), s.W - n);
    by = min(max(by, 0), s.H - n);
    const FixScale fs{s.scales[0], s.scales[1]};
    float mean, sd;
    fix_stats(rect(s, s.sum, bx, by, bx + n, by + n), rect(s, s.sumsq, bx, by, bx + n, by + n), fs, (float)(n * n), &mean,
              &sd);
    return mean >= min_mean && sd >= min_std;
}

// Batches of items of any grid size: item i owns cells [cell_start[i], cell_start[i+1]).
struct PlaceBatch {
    int n;
    int cell_start[kMaxBatch + 1];
    PlaceParams item[kMaxBatch];
};

struct ValidateBatch {
    int n;
    int tile_start[kMaxBatch + 1];
    ValidateParams item[kMaxBatch];
};

__global__ void place_kernel(const __grid_constant__ PlaceBatch b) {
    dependent_wait();
    let_dependents_start();
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= b.cell_start[b.n]) return;
    const int it = batch_item(b.cell_start, b.n, u);
    const PlaceParams& p = b.item[it];
    const int k = u - b.cell_start[it];
    const int ix = k % p.grid.nx, iy = k / p.grid.nx;
    const int n = p.grid.window;
    if (k == 0 && p.zero_counts)
        for (int j = 0; j < 5; ++j) p.zero_counts[j] = 0;
    // max = (w - n).saturating_sub(1) (multipass.rs:207-208)
    const float max_x = (float)max(p.W - n - 1, 0), max_y = (float)max(p.H - n - 1, 0);
    float2 shift = make_float2(0.0f, 0.0f);
    if (p.has_pred)
        shift = sample_predictor(p.pdx, p.pdy, p.pgrid, grid_center(p.grid.x0, ix, p.grid.step, n),
                                 grid_center(p.grid.y0, iy, p.grid.step, n));
    const float2 xs = place1(p.grid.x0 + ix * p.grid.step, shift.x, max_x);
    const float2 ys = place1(p.grid.y0 + iy * p.grid.step, shift.y, max_y);
    const float4 o = make_float4(xs.x, ys.x, xs.y, ys.y);
    p.origins[k] = o;
    if (p.corners) {
        // Predictor at the corner pixels (x0, y0), (x0+n-1, y0), (x0, y0+n-1), (x0+n-1, y0+n-1) of
        // the deformed window's base position: the zero-shift origin under the placement clamp.
        const float xa = (float)min(p.grid.x0 + ix * p.grid.step, max(p.W - n - 1, 0));
        const float ya = (float)min(p.grid.y0 + iy * p.grid.step, max(p.H - n - 1, 0));
        const float xb = __fadd_rn(xa, (float)(n - 1)), yb = __fadd_rn(ya, (float)(n - 1));
        float2 c00 = make_float2(0.0f, 0.0f), c10 = c00, c01 = c00, c11 = c00;
        if (p.has_pred) {
            c00 = sample_predictor(p.pdx, p.pdy, p.pgrid, xa, ya);
            c10 = sample_predictor(p.pdx, p.pdy, p.pgrid, xb, ya);
            c01 = sample_predictor(p.pdx, p.pdy, p.pgrid, xa, yb);
            c11 = sample_predictor(p.pdx, p.pdy, p.pgrid, xb, yb);
        }
        p.corners[2 * (size_t)k] = make_float4(c00.x, c00.y, c10.x, c10.y);
        p.corners[2 * (size_t)k + 1] = make_float4(c01.x, c01.y, c11.x, c11.y);
    }
    uint8_t st = 1;
    if (p.use_stats)
        st = has_signal(p.sa, o.x, o.y, n, p.min_mean, p.min_std) && has_signal(p.sb, o.z, o.w, n, p.min_mean, p.min_std);
    p.status[k] = st;
}

__global__ void mask_kernel(const PlaceParams p, const float4* origins, int ncells) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ncells) return;
    const float4 o = origins[k];
    const int n = p.grid.window;
    uint8_t st = 1;
    if (p.use_stats)
        st = has_signal(p.sa, o.x, o.y, n, p.min_mean, p.min_std) && has_signal(p.sb, o.z, o.w, n, p.min_mean, p.min_std);
    p.status[k] = st;
}

cudaError_t launch_place_items(const PlaceParams* items, int count, cudaStream_t s, int* launches) {
    for (int off = 0; off < count; off += kMaxBatch) {
        PlaceBatch b;
        b.n = min(count - off, kMaxBatch);
        long long total = 0;
        for (int i = 0; i < b.n; ++i) {
            b.item[i] = items[off + i];
            b.cell_start[i] = (int)total;
            total += (long long)b.item[i].grid.nx * b.item[i].grid.ny;
        }
        b.cell_start[b.n] = (int)total;
        if (total <= 0) continue;
        if (total > 0x7fffffffll) return cudaErrorInvalidValue;
        const cudaError_t e = launch_dependent(place_kernel, (unsigned)((total + 255) / 256), 256, 0, s, b);
        if (e != cudaSuccess) return e;
        if (launches) ++*launches;
    }
    return cudaSuccess;
}

cudaError_t launch_place(const PlaceParams& p, cudaStream_t s) { return launch_place_items(&p, 1, s, nullptr); }

cudaError_t launch_mask(const PlaceParams& p, const float4* origins, int ncells, cudaStream_t s) {
    if (ncells <= 0) return cudaSuccess;
    mask_kernel<<<(ncells + 255) / 256, 256, 0, s>>>(p, origins, ncells);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Validation
// ---------------------------------------------------------------------------------------------
// Total-order key of a non-NaN float: signed integer order of the keys is f32::total_cmp order
// (-0.0 before +0.0), which validate.rs:164 sorts by. The map is its own inverse.
__device__ __forceinline__ int tkey(float f) {
    const int b = __float_as_int(f);
    return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float tval(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

// Sorts v[0..n) ascending by total order (insertion sort) and returns the median, the mean of
// the middle two when n is even (validate.rs:163-170).
__device__ float median_sorted(float* v, int n) {
    for (int i = 1; i < n; ++i) {
        const float x = v[i];
        const int kx = tkey(x);
        int j = i;
        while (j > 0 && tkey(v[j - 1]) > kx) {
            v[j] = v[j - 1];
            --j;
        }
        v[j] = x;
    }
    if (n % 2 == 1) return v[n / 2];
    return __fmul_rn(0.5f, __fadd_rn(v[n / 2 - 1], v[n / 2]));
}

// Radius-1 neighbourhoods in registers: eight key slots, absent or unusable neighbours padded with
// INT_MAX (above every finite key), sorted by Batcher's odd-even merge network (19 exchanges), so
// the c usable keys come first in order.
__device__ __forceinline__ void kx_swap(int& a, int& b) {
    const int lo = min(a, b), hi = max(a, b);
    a = lo;
    b = hi;
}
__device__ __forceinline__ void sort8(int (&k)[8]) {
    kx_swap(k[0], k[1]); kx_swap(k[2], k[3]); kx_swap(k[4], k[5]); kx_swap(k[6], k[7]);
    kx_swap(k[0], k[2]); kx_swap(k[1], k[3]); kx_swap(k[4], k[6]); kx_swap(k[5], k[7]);
    kx_swap(k[1], k[2]); kx_swap(k[5], k[6]);
    kx_swap(k[0], k[4]); kx_swap(k[1], k[5]); kx_swap(k[2], k[6]); kx_swap(k[3], k[7]);
    kx_swap(k[2], k[4]); kx_swap(k[3], k[5]);
    kx_swap(k[1], k[2]); kx_swap(k[3], k[4]); kx_swap(k[5], k[6]);
}
// Median of the first c (1..8) of eight sorted keys, as median_sorted computes it.
__device__ __forceinline__ float median8(const int (&k)[8], int c) {
    int lo = k[0], hi = k[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        if (i == (c - 1) / 2) lo = k[i];
        if (i == c / 2) hi = k[i];
    }
    if (c % 2 == 1) return tval(hi);
    return __fmul_rn(0.5f, __fadd_rn(tval(lo), tval(hi)));
}
// Normalised residual |value - med| / (median |nb - med| + eps) over the first c sorted keys
// (validate.rs:157-161).
__device__ __forceinline__ float residual8(float value, const int (&k)[8], int c, float eps) {
    const float med = median8(k, c);
    int dev[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) dev[i] = i < c ? tkey(fabsf(__fsub_rn(tval(k[i]), med))) : 0x7fffffff;
    sort8(dev);
    return __fdiv_rn(fabsf(__fsub_rn(value, med)), __fadd_rn(median8(dev, c), eps));
}

// Usable neighbours within `radius` of (x, y) of a tile stored with row stride `stride`: flags in f
// (cells outside the field are not usable there), values in u, v; appended to nu, nv.
template <int RU, int RF>
__device__ int collect_neighbours(const float (*u)[RU], const float (*v)[RU], const uint8_t (*f)[RF], int vy, int vx,
                                  int fy, int fx, int radius, float* nu, float* nv) {
    int c = 0;
    for (int j = -radius; j <= radius; ++j)
        for (int i = -radius; i <= radius; ++i)
            if ((i || j) && (f[fy + j][fx + i] & F_INVALID) == 0) {
                nu[c] = u[vy + j][vx + i];
                nv[c] = v[vy + j][vx + i];
                ++c;
            }
    return c;
}

// Validation of one TX x TY tile of a field in one launch: the per-vector tests (validate.rs:59-78)
// on the tile and a halo of 3 cells, the normalized median test (:80-100) on the tile and a halo of
// 2, the replacement by the median of usable neighbours at radius 1, then 2 (:102-128) on the tile,
// and on the last pass the summary counts (:40-46). The flag snapshots between the stages stay in
// shared memory; the halo cells are computed again by each tile that needs them (32 x 32: 1.27 times
// the median tests of separate launches; 32 x 8: 1.69 times).
//
// The stages are short and their launches were not: as three kernels with flag planes in memory and
// two more for the summary, each pass of a small field spent 13 us in them and the last one 6 us
// more (31 x 31 cells, B200); a 512 x 512 pair of one pass went from 48.6 to 39.1 us and a
// batch of 64 pairs of 1280 x 800 from 4.17 to 3.76 ms with this and the export below.
//
// The median and replacement loops walk only the cells that lie in the field, so that a tile of few
// columns keeps its warps full: a warp that replaces one cell takes as long as one that replaces 32.
constexpr int kValidateThreads = 256;

template <int TX, int TY>
__global__ void __launch_bounds__(kValidateThreads) validate_kernel(const __grid_constant__ ValidateBatch b) {
    constexpr int LX = TX + 6, LY = TY + 6;  // values and first flags
    constexpr int MX = TX + 4, MY = TY + 4;  // flags after the median test
    __shared__ float su[LY][LX], sv[LY][LX];
    __shared__ uint8_t s1[LY][LX], s2[MY][MX];
    __shared__ unsigned int s_count[5];
    dependent_wait();
    let_dependents_start();
    const int it = batch_item(b.tile_start, b.n, (int)blockIdx.x);
    const ValidateParams& p = b.item[it];
    const int tile = (int)blockIdx.x - b.tile_start[it], tiles_x = (p.nx + TX - 1) / TX;
    const int x0 = (tile % tiles_x) * TX, y0 = (tile / tiles_x) * TY;
    if (threadIdx.x < 5) s_count[threadIdx.x] = 0;
    for (int i = threadIdx.x; i < LX * LY; i += kValidateThreads) {
        const int ly = i / LX, lx = i - ly * LX, x = x0 + lx - 3, y = y0 + ly - 3;
        uint8_t f = F_NO_SIGNAL;  // outside the field: not usable
        float u = 0.0f, v = 0.0f;
        if (x >= 0 && x < p.nx && y >= 0 && y < p.ny) {
            const int k = y * p.nx + x;
            f = p.flags0[k];
            u = p.dx[k];
            v = p.dy[k];
            if (!(f & F_NO_SIGNAL)) {
                if (hypotf(u, v) > p.max_displacement) f |= F_OUT_OF_RANGE;
                if (p.ppr[k] < p.ppr_threshold) f |= F_LOW_PPR;
            }
        }
        su[ly][lx] = u;
        sv[ly][lx] = v;
        s1[ly][lx] = f;
    }
    for (int i = threadIdx.x; i < MX * MY; i += kValidateThreads) s2[i / MX][i % MX] = F_NO_SIGNAL;
    __syncthreads();
    const int mx0 = max(2 - x0, 0), my0 = max(2 - y0, 0);  // first of s2's columns and rows in the field
    const unsigned mw = min(p.nx - x0 + 2, MX) - mx0, mh = min(p.ny - y0 + 2, MY) - my0;
    for (unsigned i = threadIdx.x; i < mw * mh; i += kValidateThreads) {
        const unsigned row = mw == MX ? i / MX : i / mw;  // whole tiles divide by a constant
        const int my = my0 + row, mx = mx0 + i - row * mw, ly = my + 1, lx = mx + 1;
        uint8_t f = s1[ly][lx];
        if ((f & F_INVALID) == 0) {
            // usable 3x3 neighbours (validate.rs:133-155), padded slots for the others
            int ku[8], kv[8];
            int c = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int dxo = (j < 3) ? j - 1 : (j < 5 ? (j == 3 ? -1 : 1) : j - 6);
                const int dyo = (j < 3) ? -1 : (j < 5 ? 0 : 1);
                const bool use = (s1[ly + dyo][lx + dxo] & F_INVALID) == 0;
                ku[j] = use ? tkey(su[ly + dyo][lx + dxo]) : 0x7fffffff;
                kv[j] = use ? tkey(sv[ly + dyo][lx + dxo]) : 0x7fffffff;
                c += use;
            }
            if (c >= 2) {
                sort8(ku);
                sort8(kv);
                const float ru = residual8(su[ly][lx], ku, c, p.median_eps);
                const float rv = residual8(sv[ly][lx], kv, c, p.median_eps);
                if (__fsqrt_rn(__fadd_rn(__fmul_rn(ru, ru), __fmul_rn(rv, rv))) > p.median_threshold) f |= F_MEDIAN_OUTLIER;
            }
        }
        s2[my][mx] = f;
    }
    __syncthreads();
    const unsigned w = min(p.nx - x0, TX), h = min(p.ny - y0, TY);
    for (unsigned i0 = 0; i0 < w * h; i0 += kValidateThreads) {
        const unsigned i = i0 + threadIdx.x;
        const int ty = w == TX ? i / TX : i / w, tx = i - ty * w, x = x0 + tx, y = y0 + ty;
        const bool in = i < w * h;
        uint8_t f = 0;
        if (in) {
            f = s2[ty + 2][tx + 2];
            float u = su[ty + 3][tx + 3], v = sv[ty + 3][tx + 3];
            if (p.replace && (f & F_NO_SIGNAL) == 0 && (f & F_INVALID) != 0) {
                float nu[24], nv[24];
                bool done = false;
                for (int radius = 1; radius <= 2 && !done; ++radius) {
                    const int c = collect_neighbours<LX, MX>(su, sv, s2, ty + 3, tx + 3, ty + 2, tx + 2, radius, nu, nv);
                    if (c > 0) {
                        u = median_sorted(nu, c);
                        v = median_sorted(nv, c);
                        f |= F_REPLACED;
                        done = true;
                    }
                }
                if (!done) {
                    u = NAN;
                    v = NAN;
                }
            }
            const int k = y * p.nx + x;
            p.out_dx[k] = u;
            p.out_dy[k] = v;
            p.out_flags[k] = f;
        }
        if (p.counts) {  // the same branch for the whole block; every lane takes part in the ballots
            const bool none = f & F_NO_SIGNAL;
            const bool bit[5] = {none, !none && (f & F_LOW_PPR), !none && (f & F_MEDIAN_OUTLIER),
                                 !none && (f & F_OUT_OF_RANGE), !none && (f & F_REPLACED)};
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                const unsigned m = __ballot_sync(0xffffffffu, in && bit[j]);
                if (m && (threadIdx.x & 31) == 0) atomicAdd(&s_count[j], (unsigned)__popc(m));
            }
        }
    }
    if (!p.counts) return;
    __syncthreads();
    if (threadIdx.x < 5 && s_count[threadIdx.x])
        atomicAdd(&p.counts[threadIdx.x], (unsigned long long)s_count[threadIdx.x]);
}

struct ValidateTile {
    int x, y;
    void (*kernel)(ValidateBatch);
};

// The tile by the cells of the batch and its largest extents (us per call on fields of noise, B200, beside
// the three separate launches that this kernel replaced):
//   - few cells want many tiles, many cells little halo. 511 x 511: 32 x 8 35, 32 x 16 43, 32 x 32 44,
//     separate 41; 660 x 660: 49, 47, 52, 50; 1021 x 1021: 100, 93, 100, 89; 1440 x 1440: 190, 167, 164, 162;
//   - a field of few columns or rows fills only part of those tiles. 262,144 x 8 cells: 248, 205, 189, and
//     158 in 16 x 64 (separate 158); 262,144 x 1: 146, 92, 66, and 25 in 4 x 128 (separate 25); 1 x 262,144:
//     42 in 32 x 8 and 22 in 128 x 4 (separate 23); 16 x 131,072: 175 in 32 x 8, 149 in 64 x 16 (157). Below 32,768 cells no shape takes more than 22 us.
ValidateTile validate_tile(const ValidateParams* items, int n) {
    long long cells = 0;
    int nx = 0, ny = 0;
    for (int i = 0; i < n; ++i) {
        cells += (long long)items[i].nx * items[i].ny;
        nx = max(nx, items[i].nx);
        ny = max(ny, items[i].ny);
    }
    if (cells >= 32768) {
        if (nx <= 2) return {4, 128, validate_kernel<4, 128>};
        if (ny <= 2) return {128, 4, validate_kernel<128, 4>};
        if (nx <= (cells >= 400000 ? 16 : 4)) return {16, 64, validate_kernel<16, 64>};
    }
    if (cells < 400000) return {32, 8, validate_kernel<32, 8>};
    if (ny <= 16) return {64, 16, validate_kernel<64, 16>};
    if (cells < 1400000) return {32, 16, validate_kernel<32, 16>};
    return {32, 32, validate_kernel<32, 32>};
}

cudaError_t launch_validate_items(const ValidateParams* items, int count, cudaStream_t s, int* launches) {
    for (int off = 0; off < count; off += kMaxBatch) {
        ValidateBatch b;
        b.n = min(count - off, kMaxBatch);
        const ValidateTile t = validate_tile(items + off, b.n);
        long long total = 0;
        for (int i = 0; i < b.n; ++i) {
            b.item[i] = items[off + i];
            b.tile_start[i] = (int)total;
            total += (long long)((b.item[i].nx + t.x - 1) / t.x) * ((b.item[i].ny + t.y - 1) / t.y);
        }
        b.tile_start[b.n] = (int)total;
        if (total <= 0) continue;
        if (total > 0x7fffffffll) return cudaErrorInvalidValue;
        const cudaError_t e = launch_dependent(t.kernel, (unsigned)total, kValidateThreads, 0, s, b);
        if (e != cudaSuccess) return e;
        if (launches) ++*launches;
    }
    return cudaSuccess;
}

cudaError_t launch_validate(const ValidateParams& p, cudaStream_t s) { return launch_validate_items(&p, 1, s, nullptr); }

// ---------------------------------------------------------------------------------------------
// Final fields to the caller's device buffers: one launch for all arrays of all items (a copy
// command each had cost a batch of 64 pairs 256 of them, about 1.5 us apiece).
// ---------------------------------------------------------------------------------------------
struct ExportBatch {
    int n;
    int block_start[kMaxBatch + 1];
    ExportItem item[kMaxBatch];
};
constexpr int kExportThreads = 256, kExportCells = 4 * kExportThreads;

__global__ void __launch_bounds__(kExportThreads) export_kernel(const __grid_constant__ ExportBatch b) {
    dependent_wait();
    let_dependents_start();
    const int it = batch_item(b.block_start, b.n, (int)blockIdx.x);
    const ExportItem& q = b.item[it];
    const int base = ((int)blockIdx.x - b.block_start[it]) * kExportCells;
    if (base == 0 && threadIdx.x < 5 && q.out_counts) q.out_counts[threadIdx.x] = q.counts[threadIdx.x];
    const float* const src[3] = {q.dx, q.dy, q.ppr};
    float* const dst[3] = {q.out_dx, q.out_dy, q.out_ppr};
    const uintptr_t at = (uintptr_t)q.dx | (uintptr_t)q.dy | (uintptr_t)q.ppr | (uintptr_t)q.out_dx | (uintptr_t)q.out_dy |
                         (uintptr_t)q.out_ppr;
    const uintptr_t at1 = (uintptr_t)q.flags | (uintptr_t)q.out_flags;
    if (at % 16 == 0 && at1 % 4 == 0 && base + kExportCells <= q.n) {
        const int k = base + 4 * threadIdx.x;
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (dst[j]) *reinterpret_cast<float4*>(dst[j] + k) = *reinterpret_cast<const float4*>(src[j] + k);
        if (q.out_flags) *reinterpret_cast<uchar4*>(q.out_flags + k) = *reinterpret_cast<const uchar4*>(q.flags + k);
        return;
    }
    for (int k = base + threadIdx.x; k < min(base + kExportCells, q.n); k += kExportThreads) {
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (dst[j]) dst[j][k] = src[j][k];
        if (q.out_flags) q.out_flags[k] = q.flags[k];
    }
}

cudaError_t launch_export_items(const ExportItem* items, int count, cudaStream_t s, int* launches) {
    for (int off = 0; off < count; off += kMaxBatch) {
        ExportBatch b;
        b.n = min(count - off, kMaxBatch);
        long long total = 0;
        for (int i = 0; i < b.n; ++i) {
            b.item[i] = items[off + i];
            b.block_start[i] = (int)total;
            total += ((long long)b.item[i].n + kExportCells - 1) / kExportCells;
        }
        b.block_start[b.n] = (int)total;
        if (total <= 0) continue;
        if (total > 0x7fffffffll) return cudaErrorInvalidValue;
        const cudaError_t e = launch_dependent(export_kernel, (unsigned)total, kExportThreads, 0, s, b);
        if (e != cudaSuccess) return e;
        if (launches) ++*launches;
    }
    return cudaSuccess;
}

}  // namespace pivb200
