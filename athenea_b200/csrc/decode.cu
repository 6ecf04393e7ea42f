// The upload's decode: 3DGS-encoded float records to the packed layout the
// rasteriser reads (common/packing.slang:5-27). Follows
// scene/splat_validate.slang:16-31 (which records are kept) and
// scene/splat_decode.slang:45-173 (how each is packed), with the 3DGS field
// modes of scene/splat_encoding.slang:71-113 (logit opacity, log scale, SH DC,
// rest coefficients colour-outer). The reference validates, prefix-sums and
// decodes in three dispatches; here one kernel does all three, the compaction
// by a decoupled look-back over a ticketed block order.
//
// Bound by memory traffic. A warp brings its 32 records into shared memory as one
// contiguous run (16-byte loads where the run allows them) and writes its splats' SH
// rows, which follow each other in the output, as one run too: a lane reading its own
// record, or writing its own row, touches a sector a value. 1.5M records of
// degree 3: 257 -> 193 us.
//
// Built with --fmad=false: see splat_math.cuh.
#include <cuda_runtime.h>
#include <cuda_fp16.h>

#include "kernels.h"
#include "raster_types.cuh"
#include "splat_math.cuh"

namespace ath {
namespace {

constexpr uint32_t kDecodeThreads = 128, kDecodeWarps = kDecodeThreads / 32;
constexpr float kSH0 = 0.28209479177387814f;

__device__ __forceinline__ float halfSafe(float v) { return fminf(fmaxf(v, -65000.0f), 65000.0f); }
__device__ __forceinline__ uint32_t packHalves(float a, float b) {
    const __half2 two = __floats2half2_rn(a, b);   // a in the low half
    return *reinterpret_cast<const uint32_t*>(&two);
}

// common/packing.slang:33-57; `round` as Slang's CUDA target emits it (roundf).
__device__ uint32_t encodeQuaternion(float q0, float q1, float q2, float q3) {
    const float kSqrtHalf = 0.70710678f;
    const float len = sqrtf(((q0 * q0 + q1 * q1) + q2 * q2) + q3 * q3);
    float q[4] = {q0 / len, q1 / len, q2 / len, q3 / len};
    uint32_t largest = 0;
    float best = fabsf(q[0]);
#pragma unroll
    for (uint32_t k = 1; k < 4; ++k) {
        if (fabsf(q[k]) > best) {
            best = fabsf(q[k]);
            largest = k;
        }
    }
    const bool flip = (largest == 0 ? q[0] : largest == 1 ? q[1] : largest == 2 ? q[2] : q[3]) < 0.0f;
    uint32_t word = largest;
    uint32_t shift = 22;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        if (k == largest) continue;
        const float v = flip ? -q[k] : q[k];
        const float unit = clampf((v / kSqrtHalf) * 0.5f + 0.5f, 0.0f, 1.0f);
        word |= (uint32_t)roundf(unit * 1023.0f) << shift;
        shift -= 10;
    }
    return word;
}

// kStaged: the records pass through shared memory (kDecodeThreads of them fit); else each
// lane reads its own where it lies, and rows go out the same way.
template <bool kStaged>
__global__ void __launch_bounds__(kDecodeThreads)
    decodeKernel(const float* __restrict__ records, uint32_t count, const ath_encoding E, float4* __restrict__ positions,
                 uint4* __restrict__ shape, uint32_t* __restrict__ sh, uint64_t* __restrict__ flags,
                 uint32_t* __restrict__ words) {
    extern __shared__ __align__(16) float sRecords[];
    __shared__ uint32_t sTicket;
    __shared__ uint32_t sWarp[kDecodeWarps];
    __shared__ uint64_t sPrefix;
    __shared__ uint8_t sLane[kDecodeWarps][32];   // the lane of each of a warp's valid records
    __shared__ uint32_t sField[48];               // where coefficient k of a packed row lies in a record
    for (uint32_t k = threadIdx.x; k < 48; k += kDecodeThreads) sField[k] = E.rest_base + (k % 3u) * E.file_per_colour + k / 3u;
    if (threadIdx.x == 0) sTicket = atomicAdd(&words[0], 1u);
    __syncthreads();
    const uint32_t b = sTicket;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t i = b * kDecodeThreads + threadIdx.x;
    float* staged = sRecords + (size_t)warp * 32 * E.stride;
    const float* r = records + (size_t)i * E.stride;
    if constexpr (kStaged) {
        const uint32_t first = b * kDecodeThreads + warp * 32;
        const uint32_t here = first < count ? min(32u, count - first) : 0u;
        const float* run = records + (size_t)first * E.stride;
        const uint32_t floats = here * E.stride;
        if ((reinterpret_cast<uintptr_t>(run) & 15u) == 0) {
            // every 16-byte piece in flight at once, straight into shared memory
            const uint32_t quads = floats / 4;
            const uint32_t to = (uint32_t)__cvta_generic_to_shared(staged);   // 32 E.stride floats a warp: 128-byte aligned
            for (uint32_t k = lane; k < quads; k += 32)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 16 * k), "l"(run + 4 * k) : "memory");
            for (uint32_t f = quads * 4 + lane; f < floats; f += 32) staged[f] = run[f];
            asm volatile("cp.async.wait_all;" ::: "memory");
        } else {
            for (uint32_t f = lane; f < floats; f += 32) staged[f] = run[f];
        }
        __syncwarp();
        r = staged + (size_t)lane * E.stride;
    }
    bool valid = false;
    float p[3] = {0, 0, 0}, a = 0.0f, ls[3] = {0, 0, 0};
    if (i < count) {
        p[0] = r[E.x];
        p[1] = r[E.y];
        p[2] = r[E.z];
        a = 1.0f / (1.0f + exp_f(-r[E.opacity]));
        ls[0] = r[E.scale0];
        ls[1] = r[E.scale1];
        ls[2] = r[E.scale2];
        uint32_t flats = 0;
        bool ok = true;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (ls[k] < -30.0f) ls[k] = __int_as_float(0xFF800000);   // a surfel's flat axis
            if (ls[k] <= -1024.0f) {
                flats += 1;
            } else if (!isfinite(ls[k]) || !(fabsf(ls[k]) < 60.0f)) {
                ok = false;
            }
        }
        valid = isfinite(p[0]) && isfinite(p[1]) && isfinite(p[2]) && flats <= 1u && ok && a >= kFaint;
    }
    // compaction: exclusive scan of `valid` over the records, in record order
    const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, valid);
    const uint32_t rank = __popc(ballot & ((1u << lane) - 1u));
    if (lane == 0) sWarp[warp] = __popc(ballot);
    if (valid) sLane[warp][rank] = (uint8_t)lane;
    __syncthreads();
    uint32_t warpBase = 0, blockTotal = 0;
#pragma unroll
    for (uint32_t w = 0; w < kDecodeWarps; ++w) {
        warpBase += w < warp ? sWarp[w] : 0u;
        blockTotal += sWarp[w];
    }
    if (warp == 0) {
        const uint64_t prefix = lookbackExclusive(flags, b, blockTotal, &words[1]);
        if (lane == 0) {
            sPrefix = prefix;
            if (b == gridDim.x - 1) words[2] = (uint32_t)(prefix + blockTotal);
        }
    }
    __syncthreads();
    const uint32_t first = (uint32_t)sPrefix + warpBase;   // where the warp's splats start
    const uint32_t j = first + rank;
    if (first + __popc(ballot) > count) {   // never, for a look-back that completed
        if (lane == 0) atomicOr(&words[1], kStatusIndexRange);
        return;
    }
    const uint32_t keep = E.keep_per_colour;
    const uint32_t shWords = keep == 0 ? 1 : (keep * 3 + 1) / 2;
    if (valid) {
        positions[j] = make_float4(p[0], p[1], p[2], clampf(a, 0.0f, 5.0f));
        const float q0 = r[E.rot_x], q1 = r[E.rot_y], q2 = r[E.rot_z], q3 = r[E.rot_w];
        const float qLength = sqrtf(((q0 * q0 + q1 * q1) + q2 * q2) + q3 * q3);
        const uint32_t rotation = qLength > 1e-8f ? encodeQuaternion(q0, q1, q2, q3) : encodeQuaternion(0, 0, 0, 1);
        const float base0 = 0.5f + kSH0 * r[E.dc0], base1 = 0.5f + kSH0 * r[E.dc1], base2 = 0.5f + kSH0 * r[E.dc2];
        shape[j] = make_uint4(rotation, packHalves(halfSafe(ls[0]), halfSafe(ls[1])),
                              packHalves(halfSafe(ls[2]), halfSafe(base0)), packHalves(halfSafe(base1), halfSafe(base2)));
    }
    // coefficient k of the packed row (basis * 3 + colour) of a record; past the last, zero
    auto rest = [&](const float* rec, uint32_t k) {
        return k < keep * 3 ? halfSafe(rec[sField[k]]) : 0.0f;
    };
    if constexpr (kStaged) {
        // the warp's rows, one contiguous run of the output
        const uint32_t run = __popc(ballot) * shWords;
        uint32_t* out = sh + (size_t)first * shWords;
        uint32_t row = lane / shWords, col = lane % shWords;
        const uint32_t rowStep = 32u / shWords, colStep = 32u % shWords;
        for (uint32_t k = lane; k < run; k += 32) {
            const float* rec = staged + (size_t)sLane[warp][row] * E.stride;
            out[k] = packHalves(rest(rec, 2 * col), rest(rec, 2 * col + 1));
            row += rowStep;
            col += colStep;
            if (col >= shWords) {
                col -= shWords;
                ++row;
            }
        }
    } else if (valid) {
        for (uint32_t k = 0; k < shWords; ++k) sh[(size_t)j * shWords + k] = packHalves(rest(r, 2 * k), rest(r, 2 * k + 1));
    }
}

}   // namespace

uint32_t decodeBlocks(uint32_t count) { return (count + kDecodeThreads - 1) / kDecodeThreads; }

// words: [0] ticket, [1] status, [2] kept; flags: decodeBlocks(count) words. Both zeroed by the caller.
cudaError_t launchDecode(const float* records, uint32_t count, const ath_encoding& E, float4* positions, uint4* shape,
                         uint32_t* sh, uint64_t* flags, uint32_t* words, cudaStream_t stream) {
    if (count == 0) return cudaSuccess;
    const size_t bytes = (size_t)kDecodeThreads * E.stride * sizeof(float);
    constexpr size_t kMostBytes = 200 * 1024;
    if (bytes <= kMostBytes) {
        const cudaError_t err = cudaFuncSetAttribute(decodeKernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     (int)kMostBytes);
        if (err != cudaSuccess) return err;
        decodeKernel<true><<<decodeBlocks(count), kDecodeThreads, bytes, stream>>>(records, count, E, positions, shape,
                                                                                  sh, flags, words);
    } else {
        decodeKernel<false><<<decodeBlocks(count), kDecodeThreads, 0, stream>>>(records, count, E, positions, shape, sh,
                                                                               flags, words);
    }
    return cudaGetLastError();
}

}   // namespace ath
