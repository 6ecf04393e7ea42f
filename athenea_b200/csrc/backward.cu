// The adjoint of the raster path, for FP32 training parameters.
//
// The reference differentiates only colour (splat_blend.slang:381-398,
// contributionMode 4: each Gaussian's colour gradient is the sum over its
// pixels of weight * dL/dpixel). This pass differentiates everything the
// forward computes from the parameters: the blend in reverse order, then the
// projection (EWA covariance, the Mip-Splatting opacity payback, SH colour,
// sRGB decode, the Jacobian with its frustum clamp).
//
// Nothing is checkpointed: the forward keeps, per pixel, only its final
// transmittance and one past the last record it blended, and, per box of pixels
// and 32 records, which of them some pixel blended. The reverse walk recomputes
// those records' power and alpha exactly as the forward did (this file is built
// with --fmad=false), so it skips the same records, and divides the
// transmittance back out record by record.
#include <algorithm>
#include <utility>

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "adjoint.cuh"
#include "gauss.cuh"
#include "kernels.h"
#include "raster_types.cuh"
#include "splat_math.cuh"
#include "walk.cuh"

namespace ath {
namespace {

// 1 / x for x = 1 - alpha, in [0.01, 1]: the hardware's approximation and one Newton step.
// Rounded as __frcp_rn for every such x (all 66.9M of the 32-bit alphas from 1/255 to 0.99
// compared, none differed), without its test for exponents that do not occur here: 20k
// Gaussians at 333x251 295 us by this, 310 by the call.
__device__ __forceinline__ float reciprocal(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return __fmaf_rn(y, __fmaf_rn(-x, y, 1.0f), y);
}

// dL/d(record) of every slot: centre x y, conic a b c, alpha, colour r g b, view z.
//
// One block a tile, its warps independent, a box of pixels each, as the forward
// (walk.cuh). A warp gathers the records its box blended (the forward's live bits), last
// first, 32 at a time into slots of its own, and walks them down from its pixels' last
// contributor. A lane sums its pixels' terms, the warp its lanes' through columns in
// shared memory, kRecords records at a time: lane k then sums column k and adds what it
// gives into that record's words in global memory. The moments in dy come from the
// columns' row sums (walk.cuh's rowSums).
//
// Bound by instruction issue. Against one thread a pixel over every record of the tile
// up to its last contributor, ten values summed by shuffles a record and warp, then
// through shared memory by atomics: 0.28 ms for 500k Gaussians at 1280x720 (0.71), 75 us
// for 20k at 333x251 (201).
template <int kPx, bool kDepth>
__global__ void __launch_bounds__(Box<kPx>::kThreads)   // what shared memory and no spill allow
    blendBackwardKernel(const FrameConst F, uint32_t pairs, uint32_t slots, const uint2* __restrict__ ranges,
                        const uint64_t* __restrict__ sorted, const float4* __restrict__ recs,
                        const TrainingState training, const float4* __restrict__ dLdColour,
                        const float* __restrict__ dLdDepth, const float* __restrict__ depthOut,
                        float* __restrict__ grads, uint32_t* __restrict__ status) {
    // of alpha dL/dalpha: its sum, its moments dx and dx dx; dL/dcolour r g b; dL/dz
    constexpr uint32_t kValues = kDepth ? 7 : 6;
    constexpr uint32_t kRecords = kPx == 2 ? 4 : 3;       // kRecords * kValues lanes sum a column each
    static_assert(kRecords * kValues <= 32, "a column a lane");
    struct Shared {
        WalkRecord<kPx> records[32];
        float sums[kRecords * kValues * kColumnStride];
    };
    __shared__ Shared sShared[Box<kPx>::kCount];
    const uint32_t tile = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    Shared& sh = sShared[warp];
    uint2 range = ranges[tile];
    if (range.y > pairs || range.x > range.y) {
        if (threadIdx.x == 0) atomicOr(status, kStatusIndexRange);
        return;
    }
    const uint32_t boxX = (tile % F.tilesX) * kTile + Box<kPx>::x0(warp);
    const uint32_t boxY = (tile / F.tilesX) * kTile + Box<kPx>::y0(warp);
    const uint32_t py = boxY + Box<kPx>::laneY(lane);
    const Px<kPx> yc = both<kPx>((float)py + 0.5f);
    Px<kPx> xc, T, dR, dG, dB, sd, rest, dDepth;
    uint32_t last[kPx], most = 0;
    bool wild = false;   // a gradient that is not finite, or whose products may not be
#pragma unroll
    for (int p = 0; p < kPx; ++p) {
        const uint32_t px = boxX + Box<kPx>::laneX(lane) + 4u * (uint32_t)p;
        const bool inside = px < F.width && py < F.height;
        const uint32_t at = inside ? py * F.width + px : 0u;
        xc.v[p] = (float)px + 0.5f;
        const float left = inside ? training.finalT[at] : 1.0f;
        last[p] = inside ? min(training.lastContrib[at], range.y - range.x) : 0u;
        // a pixel that blended nothing gives nothing, whatever its gradient holds
        const float4 dC = last[p] ? dLdColour[at] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        T.v[p] = left;
        dR.v[p] = dC.x;
        dG.v[p] = dC.y;
        dB.v[p] = dC.z;
        // the colour behind a record enters through its product with dL/dcolour alone (and,
        // with the depth's gradient, the depth behind times its)
        sd.v[p] = (F.bg[0] * dC.x + F.bg[1] * dC.y) + F.bg[2] * dC.z;
        // what a record's alpha takes through the final transmittance, over 1 - alpha: the alpha
        // channel's 1 - T + T bg_a, and the depth's division by the coverage
        rest.v[p] = dC.w * left * (1.0f - F.bg[3]);
        dDepth.v[p] = 0.0f;
        if (kDepth && last[p]) {
            const float cov = 1.0f - left, dD = dLdDepth[at];
            if (cov > 1e-6f && dD != 0.0f) {
                dDepth.v[p] = dD / cov;
                rest.v[p] -= dDepth.v[p] * depthOut[at] * left;
            }
        }
        const float size = ((fabsf(dC.x) + fabsf(dC.y)) + fabsf(dC.z)) + ((fabsf(sd.v[p]) + fabsf(rest.v[p])) + fabsf(dDepth.v[p]));
        wild = wild || !(size < kWalkLimit);
        most = max(most, last[p]);
    }
    const uint32_t sumRecord = lane / kValues, sumValue = lane % kValues;   // the column this lane sums
    wild = __any_sync(0xFFFFFFFFu, wild);
    const int32_t chunks = (int32_t)((__reduce_max_sync(0xFFFFFFFFu, most) + 31u) >> 5);
    const uint32_t* liveOf = training.live + ((size_t)(range.x >> 5) + tile) * Box<kPx>::kCount + warp;
    for (int32_t hi = chunks - 1; hi >= 0; hi -= 32) {
        // lane l: the live bits of chunk hi - l
        const int32_t ch = hi - (int32_t)lane;
        const uint32_t word = ch >= 0 ? liveOf[(size_t)ch * Box<kPx>::kCount] : 0u;
        const uint32_t n = __popc(word);
        uint32_t incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= (uint32_t)o) incl += u;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        for (uint32_t r0 = 0; r0 < total; r0 += 32) {
            uint32_t chunk, bit;
            liveRecord(word, incl - n, r0 + lane, chunk, bit);
            const uint32_t count = min(32u, total - r0);
            if (lane < count) {
                const uint32_t rel = (uint32_t)(hi - (int32_t)chunk) * 32u + bit;
                uint32_t s = (uint32_t)sorted[range.x + rel];
                if (s >= slots) {
                    atomicOr(status, kStatusIndexRange);
                    s = 0;
                }
                sh.records[lane].set(recs[(size_t)s * 3 + 0], recs[(size_t)s * 3 + 1], recs[(size_t)s * 3 + 2], s, rel + 1u);
            }
            __syncwarp();
            const bool odd = wild || __any_sync(0xFFFFFFFFu, lane < count && sh.records[lane].odd != 0u);
            auto walk = [&](auto oddHere) {
            constexpr bool kOdd = decltype(oddHere)::value;
            for (uint32_t q0 = 0; q0 < count; q0 += kRecords) {
                const uint32_t batch = min(kRecords, count - q0);
                float* column = sh.sums + lane;
                for (uint32_t q = q0; q < q0 + batch; ++q, column += kValues * kColumnStride) {
                    using Rec = WalkRecord<kPx>;
                    const Rec& R = sh.records[q];
                    const WalkPoint<kPx, kOdd> at(R, xc, yc);
                    Px<kPx> alpha, inv;
                    bool on[kPx];
#pragma unroll
                    for (int p = 0; p < kPx; ++p) {
                        const float a = fminf(0.99f, at.raw.v[p]);
                        on[p] = R.place <= last[p] && !(at.power.v[p] > R.cutoff) && !(a < kFaint);
                        alpha.v[p] = on[p] ? a : 0.0f;
                    }
                    const Px<kPx> minus = alpha + both<kPx>(-1.0f);   // -(1 - alpha), rounded alike
#pragma unroll
                    for (int p = 0; p < kPx; ++p) inv.v[p] = reciprocal(-minus.v[p]);
                    // the transmittance before the record: T / (1 - alpha), its quotient corrected by its
                    // remainder (P. Markstein, "Computation of elementary functions on the IBM RISC
                    // System/6000 processor", IBM J. Res. Dev. 34, 1990): with a rounded reciprocal
                    // the rounded quotient
                    Px<kPx> Tb = T * inv;
                    Tb = fused(fused(minus, Tb, T), inv, Tb);
                    const Px<kPx> w = Tb * alpha;
                    // where a colour or a gradient may not be finite, alpha 0 does not keep the pixels
                    // that did not blend the record out of its sums: their terms are left out
                    Px<kPx> vR = dR, vG = dG, vB = dB, vDepth = dDepth, vRest = rest;
                    if (kOdd) {
#pragma unroll
                        for (int p = 0; p < kPx; ++p)
                            if (!on[p]) vR.v[p] = vG.v[p] = vB.v[p] = vDepth.v[p] = vRest.v[p] = 0.0f;
                    }
                    Px<kPx> cd = fused(Rec::px(R.bl), vB, fused(Rec::px(R.g), vG, Rec::px(R.r) * vR));
                    if (kDepth) cd = fused(Rec::px(R.z), vDepth, cd);
                    Px<kPx> u = fused(sd, both<kPx>(-1.0f), cd);
                    if (kOdd) {
#pragma unroll
                        for (int p = 0; p < kPx; ++p)
                            if (!on[p]) u.v[p] = 0.0f;
                    }
                    // alpha dL/dalpha: the opacity times dL/dopacity, and -2 dL/dpower, where alpha is
                    // neither clamped nor of an opacity over 1
                    Px<kPx> aDA = fused(alpha * inv, vRest, w * u);
                    sd = fused(alpha, u, sd);
                    T = Tb;
#pragma unroll
                    for (int p = 0; p < kPx; ++p)
                        if (!(at.raw.v[p] < 0.99f && R.alpha[0] <= 1.0f)) aDA.v[p] = 0.0f;
                    const Px<kPx> x1 = aDA * at.dx, x2 = x1 * at.dx;
                    auto sum = [](const Px<kPx>& v) { return kPx == 2 ? v.v[0] + v.v[kPx - 1] : v.v[0]; };
                    column[0 * kColumnStride] = sum(aDA);
                    column[1 * kColumnStride] = sum(x1);
                    column[2 * kColumnStride] = sum(x2);
                    column[3 * kColumnStride] = sum(w * vR);
                    column[4 * kColumnStride] = sum(w * vG);
                    column[5 * kColumnStride] = sum(w * vB);
                    if (kDepth) column[6 * kColumnStride] = sum(w * vDepth);
                }
                __syncwarp();
                // dL/dpower is -1/2 alpha dL/dalpha; its moments over (dx, dy) give the centre's and
                // the conic's gradients, the centre's x and y both in the lane of the moment dx
                const bool mine = lane < batch * kValues;
                RowSums v{0.0f, 0.0f, 0.0f};
                const WalkRecord<kPx>& R = sh.records[q0 + min(sumRecord, batch - 1u)];
                if (mine)
                    v = rowSums<(int)Box<kPx>::kHeight>(sh.sums + lane * kColumnStride, (float)boxY + 0.5f, R.ny[0]);
                const float my = __shfl_up_sync(0xFFFFFFFFu, v.first, 1);   // of the moment dx: sum dy
                if (mine) {
                    float* words = grads + (size_t)R.slot * kGradWords;
                    auto add = [&](uint32_t word, float value) {
                        if (value != 0.0f) atomicAdd(words + word, value);
                    };
                    if (sumValue == 0) {
                        add(kGradAlpha, v.sum / R.alpha[0]);
                        add(kGradC, -0.5f * v.second);
                    } else if (sumValue == 1) {
                        add(kGradCx, __fmaf_rn(R.a[0], v.sum, 0.5f * R.b2[0] * my));
                        add(kGradCy, __fmaf_rn(0.5f * R.b2[0], v.sum, R.c[0] * my));
                        add(kGradB2, -v.first);
                    } else {
                        add(sumValue == 2 ? (uint32_t)kGradA : (uint32_t)kGradR + sumValue - 3u,
                            sumValue == 2 ? -0.5f * v.sum : v.sum);
                    }
                }
                __syncwarp();   // the next records overwrite the columns
            }
            };
            if (odd) {
                walk(std::true_type());
                // a pixel that blended a colour past the limit has it behind the records in front
                bool past = false;
#pragma unroll
                for (int p = 0; p < kPx; ++p) past = past || !(fabsf(sd.v[p]) < kWalkLimit);
                wild = wild || __any_sync(0xFFFFFFFFu, past);
            } else {
                walk(std::false_type());
            }
        }
    }
}

// The slots whose records took a gradient, in `list` (their number in *listed, which starts
// at zero): most records of a frame lie behind their pixels' early stop, or in no pixel's
// footprint, and take none.
__global__ void __launch_bounds__(256)
    listGradientsKernel(uint32_t slots, const uint32_t* __restrict__ keys, const float* __restrict__ grads,
                        uint32_t* __restrict__ list, uint32_t* __restrict__ listed) {
    const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    bool some = false;
    if (slot < slots && keys[slot] < kCulledKey) {
        const float2* g = reinterpret_cast<const float2*>(grads + (size_t)slot * kGradWords);
#pragma unroll
        for (uint32_t k = 0; k < kGradWords / 2; ++k) {
            const float2 v = g[k];
            some = some || v.x != 0.0f || v.y != 0.0f;
        }
    }
    // a block's places by one addition: one a warp, all to one word, was most of the
    // kernel (500k Gaussians: 14 us, now 7)
    __shared__ uint32_t sCount[8], sFirst;
    const uint32_t warp = threadIdx.x >> 5, ballot = __ballot_sync(0xFFFFFFFFu, some);
    if (lane == 0) sCount[warp] = __popc(ballot);
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (uint32_t w = 0; w < 8; ++w) {
        before += w < warp ? sCount[w] : 0u;
        all += sCount[w];
    }
    if (threadIdx.x == 0 && all) sFirst = atomicAdd(listed, all);
    __syncthreads();
    if (some) list[sFirst + before + __popc(ballot & ((1u << lane) - 1u))] = slot;
}

// The projection's adjoint, one thread a listed Gaussian: dL/d(record) -> dL/d(parameters),
// added in. A warp brings its 32 SH rows into shared memory a row at a time (stride 49:
// lane l's value k at bank (17 l + k) mod 32), each thread puts its gradient in its row's
// place, and the warp adds the rows to the gradients a row at a time: every access covers
// whole sectors, where a lane at its own row touched a line a load.
// Over every slot in order, each thread its own rows: 500k Gaussians at 1280x720, degree 3,
// 308 us; the list 7 and this 49.
constexpr uint32_t kRowsAtOnce = 8;   // of rows that are not whole pieces

__global__ void __launch_bounds__(128)
    projectBackwardKernel(const FrameConst F, const InstanceConst I, const uint32_t* __restrict__ list,
                          const uint32_t* __restrict__ listed, const float* __restrict__ grads,
                          float4* __restrict__ gMeans, float4* __restrict__ gScales, float4* __restrict__ gQuats,
                          float* __restrict__ gSh) {
    __shared__ float sSh[4][32 * 49];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t count = min(*listed, I.count);
    const uint32_t degree = min(degreeOf(I.restPerColour), F.shLimit);
    const uint32_t bases = degree >= 3 ? 15u : degree == 2 ? 8u : degree == 1 ? 3u : 0u;
    const uint32_t cols = 3u + 3u * bases;   // past the degree's the gradient is zero
    const bool aligned = cols % 4 == 0 && I.shStride % 4 == 0 &&
                         ((reinterpret_cast<uintptr_t>(I.shf) | reinterpret_cast<uintptr_t>(gSh)) & 15u) == 0;
    const uint32_t quads = aligned ? cols / 4 : 0u;   // 12 at degree 3, 3 at degree 1; 27 and 3 values are not whole pieces
    for (uint32_t k0 = (blockIdx.x * 4 + warp) * 32; k0 < count; k0 += gridDim.x * 128) {
        const bool active = k0 + lane < count;
        const uint32_t rows = min(32u, count - k0);
        const uint32_t slot = active ? list[k0 + lane] : I.base, i = slot - I.base;
        // the warp's rows `quads` 16-byte pieces each where they are aligned so, a lane a piece,
        // several in flight; else some rows at a time, a lane a value
        const uint32_t pieces = rows * quads;
        if (quads) {
#pragma unroll 6
            for (uint32_t k = 0; k < 12; ++k) {
                const uint32_t at = min(k * 32 + lane, pieces - 1u), r = at / quads, q = at % quads;
                const uint32_t ri = __shfl_sync(0xFFFFFFFFu, i, r);
                if (k * 32 < pieces) {
                    const float4 v = __ldg(reinterpret_cast<const float4*>(I.shf + (size_t)ri * I.shStride) + q);
                    float* to = sSh[warp] + r * 49 + 4 * q;
                    to[0] = v.x; to[1] = v.y; to[2] = v.z; to[3] = v.w;
                }
            }
        } else {
            for (uint32_t r0 = 0; r0 < rows; r0 += kRowsAtOnce)
                for (uint32_t c = lane; c < cols; c += 32) {
                    float v[kRowsAtOnce];
#pragma unroll
                    for (uint32_t k = 0; k < kRowsAtOnce; ++k)
                        if (r0 + k < rows) v[k] = __ldg(I.shf + (size_t)(list[k0 + r0 + k] - I.base) * I.shStride + c);
#pragma unroll
                    for (uint32_t k = 0; k < kRowsAtOnce; ++k)
                        if (r0 + k < rows) sSh[warp][(r0 + k) * 49 + c] = v[k];
                }
        }
        __syncwarp();
        if (active) {
            const float* gr = grads + (size_t)slot * kGradWords;
            float gw[kGradWords];
#pragma unroll
            for (int k = 0; k < (int)kGradWords; ++k) gw[k] = gr[k];
            ParamGrad acc;
            acc.clear();
            projectAdjoint(F, I, i, degree, bases, gw, sSh[warp] + lane * 49, acc);
            acc.addGeometryTo(i, gMeans, gScales, gQuats);
        }
        __syncwarp();
        if (quads) {
#pragma unroll 6
            for (uint32_t k = 0; k < 12; ++k) {
                const uint32_t at = min(k * 32 + lane, pieces - 1u), r = at / quads, q = at % quads;
                const uint32_t ri = __shfl_sync(0xFFFFFFFFu, i, r);
                if (k * 32 + lane < pieces) {
                    float4* to = reinterpret_cast<float4*>(gSh + (size_t)ri * I.shStride) + q;
                    const float* add = sSh[warp] + r * 49 + 4 * q;
                    float4 v = *to;
                    v.x += add[0]; v.y += add[1]; v.z += add[2]; v.w += add[3];
                    *to = v;
                }
            }
        } else {
            for (uint32_t r0 = 0; r0 < rows; r0 += kRowsAtOnce)
                for (uint32_t c = lane; c < cols; c += 32) {
                    float v[kRowsAtOnce];
#pragma unroll
                    for (uint32_t k = 0; k < kRowsAtOnce; ++k)
                        if (r0 + k < rows) v[k] = gSh[(size_t)(list[k0 + r0 + k] - I.base) * I.shStride + c];
#pragma unroll
                    for (uint32_t k = 0; k < kRowsAtOnce; ++k)
                        if (r0 + k < rows)
                            gSh[(size_t)(list[k0 + r0 + k] - I.base) * I.shStride + c] = v[k] + sSh[warp][(r0 + k) * 49 + c];
                }
        }
        __syncwarp();
    }
}

// L = mean over pixels and r g b of (colour - target)^2: its value (added into
// *loss) and dL/dcolour (float4 a pixel, alpha 0). The threads' shares are summed in 64
// bits over a cluster of blocks, one 32-bit addition into *loss a cluster, 148 at most: one
// a block of 256 pixels, thousands an image, each rounded *loss, 3e-6 of it in all at
// 1920x1080 (3e-7 now), though without clusters the blocks drift apart less where the target
// comes from memory. The grid fills every SM once, which takes 32 registers a thread, and
// a block writes its sum into the first block's shared memory, a barrier's first half at the
// start standing for that block's being there. 333x251: 2.6 us a block at a time, 3.3 so
// (4.0 by 40 registers and two barriers at the end); 1280x720 8.5, 9.8 (11.3), 7.9, 7.0 (9.1)
// where the target is in the L2; 1920x1080 16.0, 17.1 (18.7); 3840x2160 58, 72 (70).
constexpr uint32_t kLossThreads = 256, kLossCluster = 8, kLossBlocks = 148 * kLossCluster;

__global__ void __cluster_dims__(kLossCluster, 1, 1) __launch_bounds__(kLossThreads, 2048 / kLossThreads)
    l2LossKernel(const float4* __restrict__ colour, const float* __restrict__ target, uint32_t pixels, float scale,
                 float4* __restrict__ dLdColour, float* __restrict__ loss) {
    __shared__ double sPart[kLossThreads / 32], sBlocks[kLossCluster];
    const auto cluster = cooperative_groups::this_cluster();
    auto started = cluster.barrier_arrive();
    float share = 0.0f;
#pragma unroll 1
    for (uint64_t p = blockIdx.x * kLossThreads + threadIdx.x; p < pixels; p += (uint64_t)gridDim.x * kLossThreads) {
        const float4 c = colour[p];
        const float er = c.x - target[p * 3 + 0], eg = c.y - target[p * 3 + 1], eb = c.z - target[p * 3 + 2];
        share += (er * er + eg * eg + eb * eb) * scale;
        dLdColour[p] = make_float4(2.0f * scale * er, 2.0f * scale * eg, 2.0f * scale * eb, 0.0f);
    }
    double sum = (double)share;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if ((threadIdx.x & 31u) == 0) sPart[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        sum = 0.0;
#pragma unroll
        for (uint32_t w = 0; w < kLossThreads / 32; ++w) sum += sPart[w];
    }
    cluster.barrier_wait(std::move(started));   // every block runs: its shared memory is there
    if (threadIdx.x == 0) *cluster.map_shared_rank(sBlocks + cluster.block_rank(), 0) = sum;
    cluster.sync();
    if (threadIdx.x == 0 && cluster.block_rank() == 0) {
        sum = 0.0;
#pragma unroll
        for (uint32_t b = 0; b < kLossCluster; ++b) sum += sBlocks[b];
        if (sum != 0.0) atomicAdd(loss, (float)sum);
    }
}

}   // namespace

cudaError_t launchBlendBackward(const FrameConst& F, uint32_t pairs, uint32_t slots, const uint2* ranges,
                                const uint64_t* sorted, const float4* recs, const TrainingState& training,
                                const float4* dLdColour, const float* dLdDepth, const float* depthOut, float* grads,
                                uint32_t* status, cudaStream_t stream) {
    const uint32_t tiles = F.tilesX * F.tilesY;
    if (tiles == 0) return cudaSuccess;
    const bool d = dLdDepth != nullptr && F.depthMode == 0;
#define ATH_BACKWARD(P_, D_)                                                                                   \
    blendBackwardKernel<P_, D_><<<tiles, Box<P_>::kThreads, 0, stream>>>(F, pairs, slots, ranges, sorted, recs, \
                                                                        training, dLdColour, dLdDepth, depthOut, grads, \
                                                                        status)
    if (training.onePixel) {
        if (d) ATH_BACKWARD(1, true);
        else ATH_BACKWARD(1, false);
    } else {
        if (d) ATH_BACKWARD(2, true);
        else ATH_BACKWARD(2, false);
    }
#undef ATH_BACKWARD
    return cudaGetLastError();
}

cudaError_t launchProjectBackward(const FrameConst& F, const InstanceConst& I, const uint32_t* keys,
                                  const float* grads, uint32_t* list, uint32_t* listed, float4* gMeans, float4* gScales,
                                  float4* gQuats, float* gSh, int sms, cudaStream_t stream) {
    if (I.count == 0) return cudaSuccess;
    listGradientsKernel<<<(I.count + 255) / 256, 256, 0, stream>>>(I.base + I.count, keys, grads, list, listed);
    const uint32_t blocks = std::min((I.count + 127) / 128, (uint32_t)sms * 4);   // four an SM by its registers
    projectBackwardKernel<<<blocks, 128, 0, stream>>>(F, I, list, listed, grads, gMeans, gScales, gQuats, gSh);
    return cudaGetLastError();
}

cudaError_t launchL2Loss(const float4* colour, const float* target, uint32_t pixels, float4* dLdColour, float* loss,
                         cudaStream_t stream) {
    if (pixels == 0) return cudaSuccess;
    const uint32_t blocks = std::min((pixels + kLossThreads - 1) / kLossThreads, kLossBlocks);
    l2LossKernel<<<(blocks + kLossCluster - 1) / kLossCluster * kLossCluster, kLossThreads, 0, stream>>>(
        colour, target, pixels, 1.0f / (3.0f * (float)pixels), dLdColour, loss);
    return cudaGetLastError();
}

}   // namespace ath
