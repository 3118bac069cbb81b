// Field validation without any device allocation.
//
// Who needs this: callers that cannot call cudaMalloc once they are running. Two kinds are
// common. An acquisition or control loop that must hand back each field on a deadline cannot
// afford an allocation call: cudaFree waits for the whole device, and a first cudaMalloc of a
// size can take milliseconds. A process whose device memory is already handed out by another
// allocator (a framework's caching pool that reserved most of the GPU) can see a plain
// cudaMalloc fail even though the pool has room. Such callers own every buffer they pass in and
// need the library to allocate nothing.
//
// The validation kernel keeps its flag snapshots (validate.rs:81 and :103 take them) in shared
// memory, tile by tile, so it needs no scratch in device memory. The entry point is defined for
// fields of at most kNoAllocMaxCells cells; larger ones are rejected.
//
// Outputs must not overlap inputs: a tile reads its neighbours' dx/dy while other blocks write
// theirs, so in-place validation would race. Overlapping buffers are rejected.
#include <cstdint>
#include <cstdio>
#include <string>

#include "../../include/piv_b200.h"
#include "kernels.h"

using namespace pivb200;

namespace {

constexpr long long kNoAllocMaxCells = 1ll << 21;

int reject(int code, const std::string& msg) {
    set_last_error(msg.c_str());
    return code;
}

// Whether the byte ranges [a, a + na) and [b, b + nb) share a byte.
bool overlap(const void* a, size_t na, const void* b, size_t nb) {
    const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b);
    return x < y + nb && y < x + na;
}

}  // namespace

extern "C" {

int32_t piv_validate_field_noalloc(int64_t ny, int64_t nx, const float* dx, const float* dy, const float* peak_ratio,
                                   const uint8_t* flags, float max_displacement, float ppr_threshold,
                                   float median_threshold, float median_eps, int32_t replace, float* out_dx,
                                   float* out_dy, uint8_t* out_flags, void* stream) {
    if (!dx || !dy || !peak_ratio || !flags || !out_dx || !out_dy || !out_flags)
        return reject(PIV_ERR_ARGUMENT, "piv_validate_field_noalloc: null pointer");
    if (ny <= 0 || nx <= 0) return reject(PIV_ERR_ARGUMENT, "piv_validate_field_noalloc: empty field");
    // nx > max / ny rather than ny * nx > max: the product of two huge sizes would overflow.
    if (nx > kNoAllocMaxCells / ny) {
        char buf[200];
        snprintf(buf, sizeof(buf),
                 "piv_validate_field_noalloc: a %lld x %lld field exceeds the limit of %lld cells",
                 (long long)ny, (long long)nx, kNoAllocMaxCells);
        return reject(PIV_ERR_UNSUPPORTED, buf);
    }
    const size_t n = (size_t)(ny * nx), nf = n * sizeof(float);
    const void* ins[4] = {dx, dy, peak_ratio, flags};
    const size_t in_bytes[4] = {nf, nf, nf, n};
    const void* outs[3] = {out_dx, out_dy, out_flags};
    const size_t out_bytes[3] = {nf, nf, n};
    for (int o = 0; o < 3; ++o) {
        for (int i = 0; i < 4; ++i)
            if (overlap(outs[o], out_bytes[o], ins[i], in_bytes[i]))
                return reject(PIV_ERR_ARGUMENT, "piv_validate_field_noalloc: an output buffer overlaps an input "
                                                "(in-place validation would race)");
        for (int q = o + 1; q < 3; ++q)
            if (overlap(outs[o], out_bytes[o], outs[q], out_bytes[q]))
                return reject(PIV_ERR_ARGUMENT, "piv_validate_field_noalloc: output buffers overlap");
    }
    ValidateParams vp{(int)nx, (int)ny, dx, dy, peak_ratio, flags, out_dx, out_dy, out_flags,
                      max_displacement, ppr_threshold, median_threshold, median_eps, replace, nullptr};
    const cudaError_t e = launch_validate(vp, static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return reject(PIV_ERR_CUDA, std::string("piv_validate_field_noalloc: ") + cudaGetErrorString(e));
    return PIV_OK;
}

}  // extern "C"
