// Stage (d): per-tile front-to-back blending -- splat/splat_blend.slang:236-578
// (splatBlend = blendPixel<composite=false, matte=false, traced=false>) -- with
// the P layer (usd/aov_position.slang:34-52) as its epilogue.
//
// One block a 16x16 tile, its warps independent: each owns a box of pixels
// (walk.cuh), reads the tile's list 32 records at a time, a lane a record, keeps
// those that can reach its box in slots of its own (in list order) and walks
// them. A pixel stops at T < 1e-4 after accumulating (:501-505), a warp once all
// its pixels have. Per pixel the walk is sequential in the tile's (depth key,
// slot) order and every value it blends is rounded as the CPU restatement does
// (built with --fmad=false; see splat_math.cuh), so the result is the
// restatement's to the bit: the box test skips only records no pixel of the box
// passes, and a pixel that does not blend a visited record takes alpha 0, which
// leaves its sums and its transmittance as they were.
//
// Bound by instruction issue. Against one thread a pixel over every record of the
// tile, staged for the whole block behind barriers: 1.5M splats at 1920x1080 0.50 -> 0.30 ms, 6M at
// 3840x2160 1.53 -> 0.96, 500k Gaussians at 1280x720 (training) 0.30 -> 0.18.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "kernels.h"
#include "raster_types.cuh"
#include "splat_math.cuh"
#include "walk.cuh"

namespace ath {
namespace {

constexpr float kColourGradScale = 256.0f;   // frame.slang:36
constexpr uint32_t kCryptoSlots = 6;         // splat_blend.slang:82

// A pixel's Cryptomatte ranks (splat_blend.slang:88-143): the ids that covered
// it most and their summed weights. Id 0 names nothing and is never kept; a full
// list gives its lightest slot up to a heavier id. Written ranked by weight,
// descending (a stable insertion sort), as 3 float4 (id bits, weight, id bits,
// weight).
// The trace's list (splat_trace.slang:33-128): the kTraceSlots heaviest splats
// of a pixel's walk by weight, the lightest rank kept so that a splat too light
// for the list costs one comparison, and everything the walk blended.
constexpr uint32_t kTraceSlots = 4;
constexpr uint32_t kTraceWords = kTraceSlots * 2 + kTraceSlots / 2 + 1;
constexpr uint32_t kTraceNone = 0xFFFFFFFFu, kTraceEmpty = 0xFFFFFFFEu;

__device__ __forceinline__ uint32_t halfBits(float v) { return (uint32_t)__half_as_ushort(__float2half_rn(v)); }

struct TraceList {
    uint32_t slots[kTraceSlots];
    float weights[kTraceSlots];
    float total, floor;
    uint32_t lightest;

    __device__ __forceinline__ void clear() {
#pragma unroll
        for (uint32_t k = 0; k < kTraceSlots; ++k) {
            slots[k] = kTraceNone;
            weights[k] = 0.0f;
        }
        total = floor = 0.0f;
        lightest = 0;
    }
    // a splat heavier than the lightest rank takes its place
    __device__ __forceinline__ void enter(uint32_t slot, float weight) {
#pragma unroll
        for (uint32_t k = 0; k < kTraceSlots; ++k)
            if (k == lightest) {
                slots[k] = slot;
                weights[k] = weight;
            }
        lightest = 0;
        float w = weights[0];
#pragma unroll
        for (uint32_t k = 1; k < kTraceSlots; ++k)
            if (weights[k] < w) {
                lightest = k;
                w = weights[k];
            }
        floor = w;
    }
    // planes of `pixels` words: the slots heaviest first, their view depths (as
    // the floats' bits), the weights as halves two a word, and (rest, under) as
    // halves; a pixel nothing reached writes kTraceEmpty in its first word alone
    __device__ void write(uint32_t* trace, uint32_t at, uint32_t pixels, float under,
                          const float4* __restrict__ recs) const {
        if (!(total > 0.0f) && !(under > 0.0f)) {
            trace[at] = kTraceEmpty;
            return;
        }
        uint32_t order[kTraceSlots];
#pragma unroll
        for (uint32_t k = 0; k < kTraceSlots; ++k) order[k] = k;
        for (uint32_t i = 1; i < kTraceSlots; ++i) {
            const uint32_t pick = order[i];
            uint32_t j = i;
            while (j > 0 && weights[order[j - 1]] < weights[pick]) {
                order[j] = order[j - 1];
                --j;
            }
            order[j] = pick;
        }
        float held = 0.0f;
        for (uint32_t k = 0; k < kTraceSlots; ++k) {
            const uint32_t from = order[k];
            const bool some = weights[from] > 0.0f;
            trace[k * pixels + at] = some ? slots[from] : kTraceNone;
            trace[(kTraceSlots + k) * pixels + at] = some ? __float_as_uint(recs[(size_t)slots[from] * 3].z) : 0u;
            held = held + weights[from];
        }
        for (uint32_t pair = 0; pair < kTraceSlots / 2; ++pair)
            trace[(kTraceSlots * 2 + pair) * pixels + at] =
                halfBits(weights[order[pair * 2]]) | (halfBits(weights[order[pair * 2 + 1]]) << 16);
        trace[(kTraceWords - 1) * pixels + at] = halfBits(fmaxf(total - held, 0.0f)) | (halfBits(fmaxf(under, 0.0f)) << 16);
    }
};

struct CryptoList {
    uint32_t ids[kCryptoSlots];
    float weights[kCryptoSlots];

    __device__ __forceinline__ void clear() {
#pragma unroll
        for (uint32_t k = 0; k < kCryptoSlots; ++k) {
            ids[k] = 0;
            weights[k] = 0.0f;
        }
    }
    // `weight` of `id` (where `on`): added to the id's slot, or in the place of the lightest
    // when the id is new and heavier. Without branches: a warp's pixels differ in which of
    // these they take, and an id is in at most one slot.
    __device__ __forceinline__ void add(bool on, uint32_t id, float weight) {
        on = on && weight > 0.0f && id != 0;
        bool found = false;
        uint32_t lightest = 0;
        float lightestWeight = weights[0];
#pragma unroll
        for (uint32_t k = 0; k < kCryptoSlots; ++k) {
            const bool here = ids[k] == id && weights[k] > 0.0f;
            const bool less = weights[k] < lightestWeight;
            lightest = less ? k : lightest;
            lightestWeight = less ? weights[k] : lightestWeight;
            found = found || here;
            weights[k] = on && here ? weights[k] + weight : weights[k];
        }
        const bool enter = on && !found && weight > lightestWeight;
#pragma unroll
        for (uint32_t k = 0; k < kCryptoSlots; ++k) {
            const bool here = enter && k == lightest;
            ids[k] = here ? id : ids[k];
            weights[k] = here ? weight : weights[k];
        }
    }
    __device__ __forceinline__ void write(float4* out, uint32_t at, uint32_t pixels) const {
        uint32_t order[kCryptoSlots];
#pragma unroll
        for (uint32_t k = 0; k < kCryptoSlots; ++k) order[k] = k;
        for (uint32_t i = 1; i < kCryptoSlots; ++i) {
            const uint32_t pick = order[i];
            uint32_t j = i;
            while (j > 0 && weights[order[j - 1]] < weights[pick]) {
                order[j] = order[j - 1];
                --j;
            }
            order[j] = pick;
        }
        for (uint32_t layer = 0; layer < kCryptoSlots / 2; ++layer) {
            const uint32_t a = order[layer * 2], b = order[layer * 2 + 1];
            out[(size_t)layer * pixels + at] =
                make_float4(weights[a] > 0.0f ? __uint_as_float(ids[a]) : 0.0f, fmaxf(weights[a], 0.0f),
                            weights[b] > 0.0f ? __uint_as_float(ids[b]) : 0.0f, fmaxf(weights[b], 0.0f));
        }
    }
};

// Which of the matte's layers a blend makes: Cryptomatte alone, or any of it (Cryptomatte,
// the lifted matte, the trace), whose lists take more registers.
enum MatteKind : uint32_t { kNoMatte = 0, kCryptomatte = 1, kAnyMatte = 2 };

// kContribution: the contributionMode hooks of splat_blend.slang:364-407 (modes
// 1 to 4). kUnder: the composite over an opaque layer under the splats
// (:249-251,329-333,516-523,555-575): a pixel's walk stops at the first record
// at or behind the layer's depth, and the layer takes the rest of the pixel.
// kMatte: Cryptomatte, the lifted matte and the trace. The plain frame builds
// without any; kTrain also keeps what the backward needs. The hooks run a pixel at
// a time, so those kernels take one pixel a lane.
template <int kPx, bool kTrain, bool kContribution, bool kUnder, MatteKind kMatte>
__global__ void __launch_bounds__(Box<kPx>::kThreads)
    blendKernel(const FrameConst F, uint32_t pairs, uint32_t slots, const uint2* __restrict__ ranges,
                const uint64_t* __restrict__ sorted, const float4* __restrict__ recs, float4* __restrict__ colour,
                float* __restrict__ depth, float4* __restrict__ position, float* __restrict__ finalT,
                uint32_t* __restrict__ lastContrib, uint32_t* __restrict__ live, uint32_t* __restrict__ status,
                Contribution contrib, Under under, Matte matte) {
    static_assert(kPx == 1 || !(kContribution || kMatte), "the hooks take one pixel a lane");
    __shared__ WalkRecord<kPx> sRecords[Box<kPx>::kCount][32];
    __shared__ uint32_t sIds[kMatte ? Box<kPx>::kCount : 1][kMatte ? 32 : 1];   // the records' Cryptomatte ids
    CryptoList list;
    if (kMatte) list.clear();
    TraceList trace;
    if (kMatte == kAnyMatte && matte.trace) trace.clear();

    const uint32_t tile = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t boxX = (tile % F.tilesX) * kTile + Box<kPx>::x0(warp);
    const uint32_t boxY = (tile / F.tilesX) * kTile + Box<kPx>::y0(warp);
    const uint32_t py = boxY + Box<kPx>::laneY(lane);
    uint32_t px[kPx];
    bool inside[kPx], done[kPx];
    float underZ[kPx];
    bool underHit[kPx];
    Px<kPx> xc;
    const Px<kPx> yc = both<kPx>((float)py + 0.5f);
    float nearestUnder = 3.4e38f;
#pragma unroll
    for (int p = 0; p < kPx; ++p) {
        px[p] = boxX + Box<kPx>::laneX(lane) + 4u * (uint32_t)p;
        inside[p] = px[p] < F.width && py < F.height;
        done[p] = !inside[p];
        xc.v[p] = (float)px[p] + 0.5f;
        underZ[p] = kUnder && inside[p] ? under.depth[py * F.width + px[p]] : 0.0f;
        underHit[p] = kUnder && underZ[p] > 0.0f;
        if (kUnder && underHit[p]) nearestUnder = fminf(nearestUnder, underZ[p]);
    }
    if (kUnder) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) nearestUnder = fminf(nearestUnder, __shfl_xor_sync(0xFFFFFFFFu, nearestUnder, o));
    }
    uint2 range = ranges[tile];
    if (range.y > pairs || range.x > range.y) {   // never, for ranges the sort wrote
        if (threadIdx.x == 0) atomicOr(status, kStatusIndexRange);
        range = make_uint2(0, 0);
    }
    const bool thresholded = F.depthMode != 0;

    Px<kPx> r = both<kPx>(0.0f), g = r, bl = r, depthSum = r, T = both<kPx>(1.0f);
    float depthAt[kPx];
    float matteKnown = 0.0f, matteInside = 0.0f, matteUntold = 0.0f;   // the lifted matte's sums
    uint32_t last[kPx];
#pragma unroll
    for (int p = 0; p < kPx; ++p) {
        depthAt[p] = -1.0f;
        last[p] = 0;
    }
    auto allDone = [&]() {
        bool d = true;
#pragma unroll
        for (int p = 0; p < kPx; ++p) d = d && done[p];
        return __all_sync(0xFFFFFFFFu, d);
    };
    // the list a chunk ahead: lane l's record of the next chunk is loaded while this one is walked
    uint32_t slot = 0, id = 0;
    float4 screen, conic, tint;
    screen = conic = tint = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto load = [&](uint32_t first) {
        if (first + lane >= range.y) return;
        slot = (uint32_t)sorted[first + lane];
        if (slot >= slots) {
            atomicOr(status, kStatusIndexRange);
            slot = 0;
        }
        screen = recs[(size_t)slot * 3 + 0];
        conic = recs[(size_t)slot * 3 + 1];
        tint = recs[(size_t)slot * 3 + 2];
        if (kMatte && matte.out) id = matte.ids[slot];
    };
    load(range.x);
    for (uint32_t first = range.x; first < range.y; first += 32) {
        if (allDone()) break;
        // a record at or behind the layer ends pixels' walks wherever it lies: such a chunk is walked whole
        const bool real = first + lane < range.y;
        bool hit = real && reachesBox(screen, conic, (float)boxX + 0.5f, (float)boxY + 0.5f,
                                      (float)(Box<kPx>::kWidth - 1), (float)(Box<kPx>::kHeight - 1));
        if (kUnder && __any_sync(0xFFFFFFFFu, real && screen.z >= nearestUnder)) hit = real;
        const uint32_t hits = __ballot_sync(0xFFFFFFFFu, hit);
        const uint32_t rank = __popc(hits & ((1u << lane) - 1u));
        const uint32_t count = __popc(hits);
        __syncwarp();   // the walk of the chunk before has read its slots
        if (hit) sRecords[warp][rank].set(screen, conic, tint, slot, first - range.x + lane + 1u);
        if (kMatte && hit) sIds[warp][rank] = id;
        if ((count & 1u) && lane == 0) sRecords[warp][count].setNone();   // the last pair's second
        __syncwarp();
        const bool odd = __any_sync(0xFFFFFFFFu, hit && sRecords[warp][rank].odd != 0u);
        load(first + 32);
        uint32_t laneBits = 0;   // the walked records some pixel of this lane blended
        // one record blended into the lane's pixels; kOdd: some record of the chunk is odd;
        // kThreshold: the depth layer's threshold crossing is wanted
        auto blendOne = [&](uint32_t j, const WalkRecord<kPx>& R, const auto& at, auto oddHere, auto thresholdHere) {
            constexpr bool kOdd = decltype(oddHere)::value, kThreshold = decltype(thresholdHere)::value;
            Px<kPx> alpha;
            bool blend[kPx], any = false;
#pragma unroll
            for (int p = 0; p < kPx; ++p) {
                if (kUnder) done[p] = done[p] || (underHit[p] && R.z[0] >= underZ[p]);
                const float a = fminf(0.99f, at.raw.v[p]);
                blend[p] = !done[p] && !(at.power.v[p] > R.cutoff) && !(a < kFaint);
                alpha.v[p] = blend[p] ? a : 0.0f;
                any = any || blend[p];
            }
            const Px<kPx> weight = T * alpha;
            if (kContribution && blend[0]) {
                const uint32_t s = R.slot, pixel = py * F.width + px[0];
                const float w = weight.v[0];
                if (contrib.mode == 1u) {
                    atomicAdd(&contrib.words[s], (uint32_t)(w * 4096.0f + 0.5f));
                } else if (contrib.mode == 2u) {
                    // splat_blend.slang:366-380: the pixel with the splat taken away shows what is
                    // behind it, recovered from the whole frame; the squared change, capped at one,
                    // in 2^-24 into a 64-bit sum of two words (low, then its carries)
                    const float4 whole = reinterpret_cast<const float4*>(contrib.finalColour)[pixel];
                    const float after = fmaxf(T.v[0] * (1.0f - alpha.v[0]), 1.0e-4f);
                    const float cx = w * (R.r[0] - (whole.x - (r.v[0] + w * R.r[0])) / after);
                    const float cy = w * (R.g[0] - (whole.y - (g.v[0] + w * R.g[0])) / after);
                    const float cz = w * (R.bl[0] - (whole.z - (bl.v[0] + w * R.bl[0])) / after);
                    const float d2 = (cx * cx + cy * cy) + cz * cz;
                    const uint32_t add = (uint32_t)(fminf(d2, 1.0f) * 16777216.0f + 0.5f);
                    const uint32_t before = atomicAdd(&contrib.words[s * 2], add);
                    if (before + add < before) atomicAdd(&contrib.words[s * 2 + 1], 1u);
                } else if (contrib.mode == 3u) {
                    // splat_blend.slang:399-407: the weight, and the weight times the mask, in 1/1024
                    const uint32_t seen = (uint32_t)(w * 1024.0f + 0.5f);
                    if (seen != 0u) {
                        atomicAdd(&contrib.words[s * 2 + 1], seen);
                        const float m = fminf(fmaxf(contrib.liftMask[pixel], 0.0f), 1.0f);
                        const uint32_t within = (uint32_t)((w * m) * 1024.0f + 0.5f);
                        if (within != 0u) atomicAdd(&contrib.words[s * 2], within);
                    }
                } else {
                    const float4 dl = reinterpret_cast<const float4*>(contrib.finalColour)[pixel];
                    const float dls[3] = {dl.x, dl.y, dl.z};
                    for (uint32_t ch = 0; ch < 3; ++ch) {
                        const float gc = (w * dls[ch]) * kColourGradScale;
                        const int step = (int)floorf(gc + hash01((pixel * 3u + ch) ^ (s * 2654435761u)));
                        if (step != 0) atomicAdd(&contrib.words[s * 4 + ch], (uint32_t)step);
                    }
                    atomicAdd(&contrib.words[s * 4 + 3], (uint32_t)(w * kColourGradScale + 0.5f));
                }
            }
            if (kMatte && matte.out) list.add(blend[0], sIds[warp][j], weight.v[0]);
            if (kMatte == kAnyMatte && blend[0] && (matte.trace || matte.lifted)) {
                const float w = weight.v[0];
                if (matte.trace) {
                    // splat_blend.slang:445-451
                    trace.total = trace.total + w;
                    if (w > trace.floor) trace.enter(R.slot, w);
                }
                if (matte.lifted) {
                    // splat_blend.slang:423-435: the share a lift told the splat, or, for one no
                    // lifting camera saw, its weight kept aside
                    const uint32_t told = R.slot * 2u;
                    const uint32_t seen = matte.liftSums[told + 1u];
                    if (seen != 0u) {
                        float share = (float)matte.liftSums[told] / (float)seen;
                        if (matte.hard) share = share > matte.threshold ? 1.0f : 0.0f;
                        matteKnown = matteKnown + w;
                        matteInside = matteInside + w * share;
                    } else {
                        matteUntold = matteUntold + w;
                    }
                }
            }
            using Rec = WalkRecord<kPx>;
            if (kOdd && R.odd) {   // a colour that is not finite stays out of the pixels that do not blend it
#pragma unroll
                for (int p = 0; p < kPx; ++p)
                    if (blend[p]) {
                        const float w = weight.v[p];
                        r.v[p] = r.v[p] + w * R.r[0];
                        g.v[p] = g.v[p] + w * R.g[0];
                        bl.v[p] = bl.v[p] + w * R.bl[0];
                        depthSum.v[p] = depthSum.v[p] + w * R.z[0];
                    }
            } else {
                r = r + weight * Rec::px(R.r);
                g = g + weight * Rec::px(R.g);
                bl = bl + weight * Rec::px(R.bl);
                depthSum = depthSum + weight * Rec::px(R.z);
            }
            T = T * fused(alpha, both<kPx>(-1.0f), both<kPx>(1.0f));   // T (1 - alpha)
            if (kThreshold) {
#pragma unroll
                for (int p = 0; p < kPx; ++p)
                    if (blend[p] && depthAt[p] < 0.0f && 1.0f - T.v[p] >= F.depthThreshold) depthAt[p] = R.z[0];
            }
#pragma unroll
            for (int p = 0; p < kPx; ++p) {
                if (kTrain) last[p] = blend[p] ? R.place : last[p];
                done[p] = done[p] || T.v[p] < 1e-4f;
            }
            if (kTrain) laneBits |= any ? 1u << j : 0u;
        };
        // the chunk's walk, two records at a time: the second's power and exponential do not
        // wait for the first's transmittance (a long chain that a warp alone on its scheduler
        // waits out)
        auto walk = [&](auto oddHere, auto thresholdHere) {
            constexpr bool kOdd = decltype(oddHere)::value;
            if (kContribution || kMatte) {
                for (uint32_t j = 0; j < count; ++j) {
                    const WalkRecord<kPx>& R = sRecords[warp][j];
                    blendOne(j, R, WalkPoint<kPx, kOdd>(R, xc, yc), oddHere, thresholdHere);
                }
            } else {
                for (uint32_t j = 0; j < count; j += 2) {
                    const WalkRecord<kPx>& R = sRecords[warp][j];
                    const WalkRecord<kPx>& S = sRecords[warp][j + 1];
                    const WalkPoint<kPx, kOdd> first(R, xc, yc), second(S, xc, yc);
                    blendOne(j, R, first, oddHere, thresholdHere);
                    blendOne(j + 1, S, second, oddHere, thresholdHere);
                }
            }
        };
        if (odd) walk(std::true_type(), std::true_type());
        else if (thresholded) walk(std::false_type(), std::true_type());
        else walk(std::false_type(), std::false_type());
        if (kTrain) {
            const uint32_t walked = __reduce_or_sync(0xFFFFFFFFu, laneBits);
            const uint32_t word = __ballot_sync(0xFFFFFFFFu, hit && ((walked >> rank) & 1u));
            if (lane == 0)
                live[((size_t)(range.x >> 5) + tile + ((first - range.x) >> 5)) * Box<kPx>::kCount + warp] = word;
        }
    }
#pragma unroll
    for (int p = 0; p < kPx; ++p) {
        if (!inside[p]) continue;
        const uint32_t at = py * F.width + px[p];
        const float left = T.v[p], coverage = 1.0f - left;
        float4 behind = make_float4(F.bg[0], F.bg[1], F.bg[2], F.bg[3]);
        if (kUnder && underHit[p]) {
            behind = reinterpret_cast<const float4*>(under.colour)[at];
            depthSum.v[p] = depthSum.v[p] + left * underZ[p];
            if (depthAt[p] < 0.0f) depthAt[p] = underZ[p];
        }
        const float total = kUnder && underHit[p] ? 1.0f : coverage;
        if (kMatte == kAnyMatte && matte.trace)   // splat_blend.slang:545-551: what closed the walk from behind is `under`
            trace.write(matte.trace, at, F.width * F.height, kUnder && underHit[p] ? left : 0.0f, recs);
        if (kMatte == kAnyMatte && matte.lifted) {
            // splat_blend.slang:536-539: the untold weight at the share of the known
            const float share = matteKnown > 0.0f ? matteInside / matteKnown : 0.0f;
            matte.lifted[at] = fminf(fmaxf(matteInside + matteUntold * share, 0.0f), 1.0f);
        }
        if (kMatte && matte.out) {
            // what closed the walk takes the rest of the pixel (splat_blend.slang:525-534)
            if (kUnder && underHit[p] && matte.underIds) list.add(true, matte.underIds[at], left);
            list.write(reinterpret_cast<float4*>(matte.out), at, F.width * F.height);
        }
        colour[at] = make_float4(r.v[p] + left * behind.x, g.v[p] + left * behind.y, bl.v[p] + left * behind.z,
                                 coverage + left * behind.w);
        const float z = F.depthMode == 0 ? (total > 1e-6f ? depthSum.v[p] / total : 0.0f) : fmaxf(depthAt[p], 0.0f);
        depth[at] = z;
        if (kTrain) {
            finalT[at] = left;
            lastContrib[at] = last[p];
        }
        if (position) {
            // usd/aov_position.slang:40-51
            if (!(z > 0.0f)) {
                position[at] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            } else {
                const float scale = F.orthographic != 0 ? 1.0f : z;
                const float v0 = ((xc.v[p] - F.centreX) / F.focalX) * scale;
                const float v1 = ((yc.v[p] - F.centreY) / F.focalY) * scale;
                const float* m = F.viewToWorld;
                position[at] = make_float4(((m[0] * v0 + m[1] * v1) + m[2] * z) + m[3] * 1.0f,
                                           ((m[4] * v0 + m[5] * v1) + m[6] * z) + m[7] * 1.0f,
                                           ((m[8] * v0 + m[9] * v1) + m[10] * z) + m[11] * 1.0f, 1.0f);
            }
        }
    }
}

}   // namespace

bool trainingOnePixel(const FrameConst& F, int sms, const Contribution& contrib, const Matte& matte) {
    return contrib.mode != 0u || matte.out != nullptr || matte.lifted != nullptr || matte.trace != nullptr ||
           onePixelBoxes(F.tilesX * F.tilesY, (uint32_t)sms, true);
}
size_t trainingLiveWords(const FrameConst& F, uint64_t pairs) { return frameLiveWords(pairs, F.tilesX * F.tilesY); }

cudaError_t launchBlend(const FrameConst& F, uint32_t pairs, uint32_t slots, const uint2* ranges,
                        const uint64_t* sorted, const float4* recs, float4* colour, float* depth, float4* position,
                        const TrainingState* training, int sms, uint32_t* status, cudaStream_t stream,
                        const Contribution& contrib, const Under& under, const Matte& matte) {
    const uint32_t tiles = F.tilesX * F.tilesY;
    if (tiles == 0) return cudaSuccess;
    const TrainingState keep = training ? *training : TrainingState{};
#define ATH_BLEND(P_, T_, C_, U_, M_)                                                                              \
    blendKernel<P_, T_, C_, U_, M_><<<tiles, Box<P_>::kThreads, 0, stream>>>(                                      \
        F, pairs, slots, ranges, sorted, recs, colour, depth, position, keep.finalT, keep.lastContrib, keep.live, \
        status, contrib, under, matte)
    const bool c = contrib.mode != 0u, u = under.depth != nullptr,
               m = matte.out != nullptr || matte.lifted != nullptr || matte.trace != nullptr;
    // an under-layer is never part of a differentiable frame
    const bool one = training ? keep.onePixel : onePixelBoxes(tiles, (uint32_t)sms, false);
    if (m && !c && !training && matte.lifted == nullptr && matte.trace == nullptr) {
        if (u) ATH_BLEND(1, false, false, true, kCryptomatte);
        else ATH_BLEND(1, false, false, false, kCryptomatte);
    } else if (m) {
        if (c && training) ATH_BLEND(1, true, true, false, kAnyMatte);
        else if (training) ATH_BLEND(1, true, false, false, kAnyMatte);
        else if (c && u) ATH_BLEND(1, false, true, true, kAnyMatte);
        else if (c) ATH_BLEND(1, false, true, false, kAnyMatte);
        else if (u) ATH_BLEND(1, false, false, true, kAnyMatte);
        else ATH_BLEND(1, false, false, false, kAnyMatte);
    } else if (c) {
        if (training) ATH_BLEND(1, true, true, false, kNoMatte);
        else if (u) ATH_BLEND(1, false, true, true, kNoMatte);
        else ATH_BLEND(1, false, true, false, kNoMatte);
    } else if (training) {
        if (one) ATH_BLEND(1, true, false, false, kNoMatte);
        else ATH_BLEND(2, true, false, false, kNoMatte);
    } else if (u) {
        if (one) ATH_BLEND(1, false, false, true, kNoMatte);
        else ATH_BLEND(2, false, false, true, kNoMatte);
    } else {
        if (one) ATH_BLEND(1, false, false, false, kNoMatte);
        else ATH_BLEND(2, false, false, false, kNoMatte);
    }
#undef ATH_BLEND
    return cudaGetLastError();
}

}   // namespace ath
