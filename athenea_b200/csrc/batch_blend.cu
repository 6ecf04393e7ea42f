// The batched path's blends: a training step's forward blend, loss and blend
// adjoint in one persistent kernel over every view's tiles. This file builds
// with FMA contraction (the other kernels of the plain and batched paths do
// not): nothing here has to match the reference's FP32 to the bit, only the
// forward and the adjoint each other, and both are compiled alike. Which records
// a pixel blends is decided per pixel, the same way in both, whatever the tile
// size.
#include <cstdint>

#include <cuda_runtime.h>

#include "batch_kernels.cuh"
#include "walk.cuh"

namespace ath {
namespace {

// A warp's box of pixels: 8x8, two pixels a lane.
constexpr uint32_t kBox = 8;
// The pixels a block takes of a tile: a span of kBlendSpan x kBlendSpan (or the
// whole tile when it is smaller), so that a block's barriers wait on fewer boxes
// and a span whose pixels are done stops staging the tile's records.
constexpr uint32_t kBlendSpan = 16;

// Bit b set when box b of the tile (boxes row-major, T/8 a row) may hold a pixel centre
// inside the footprint: unless the footprint's least power over the box's pixel centres is
// past the cutoff. The least power lies on an edge facing the centre (walk.cuh's reachesBox,
// here for the factored conic). Conservative: the limit carries a margin over the per-pixel
// test's rounding, in absolute and relative terms and for the cancellation in t = dx + fr dy
// (an error of 2 ca t over the roundings of dx and fr dy, with ca t^2 near the limit).
template <uint32_t T>
__device__ __forceinline__ uint32_t boxMask(float tileX0, float tileY0, float4 screen, float ca, float fr, float fs) {
    constexpr int kAcross = (int)(T / kBox);
    const float cc = __fmaf_rn(ca * fr, fr, fs);
    if (!(cc > 1e-12f)) return (1u << (kAcross * kAcross)) - 1u;
    const float perX = __fdividef(-ca * fr, cc);   // an edge at x: the least power's y over x
    const float limit = screen.w * 1.0001f + 1e-4f;
    const float cancel = 3e-7f * __fsqrt_rn(ca * limit);
    uint32_t mask = 0;
#pragma unroll
    for (int r = 0; r < kAcross; ++r) {
        const float loy = (tileY0 + (float)(r * (int)kBox) + 0.5f) - screen.y, hiy = loy + (float)(kBox - 1);
        const float ey = clampf(0.0f, loy, hiy), Y = fmaxf(fabsf(loy), fabsf(hiy));
#pragma unroll
        for (int c = 0; c < kAcross; ++c) {
            const float lox = (tileX0 + (float)(c * (int)kBox) + 0.5f) - screen.x, hix = lox + (float)(kBox - 1);
            const float ex = clampf(0.0f, lox, hix), X = fmaxf(fabsf(lox), fabsf(hix));
            const float y = clampf(perX * ex, loy, hiy), x = clampf(-fr * ey, lox, hix);
            const float t = __fmaf_rn(fr, y, ex), u = __fmaf_rn(fr, ey, x);
            const float onX = ex != 0.0f ? __fmaf_rn(ca * t, t, (fs * y) * y) : 3.4e38f;
            const float onY = ey != 0.0f ? __fmaf_rn(ca * u, u, (fs * ey) * ey) : 3.4e38f;
            const float least = ex == 0.0f && ey == 0.0f ? 0.0f : fminf(onX, onY);
            if (!(least > __fmaf_rn(cancel, __fmaf_rn(fabsf(fr), Y, X), limit))) mask |= 1u << (r * kAcross + c);
        }
    }
    return mask;
}

// A walk's exponent e = log2(opacity) - power / (2 ln 2), so that alpha =
// min(0.99, 2^e) takes no multiply a pixel: each staged record carries
// log2(opacity) in place of its opacity (every record's opacity is at least 1/255).
__device__ __forceinline__ float log2Of(float x) {
    float lg;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(lg) : "f"(x));
    return lg;
}
// The least such exponent at which a pixel blends a record: the larger of the
// cutoff's (power at the cutoff) and log2(1/255), where alpha reaches 1/255. One
// comparison a pixel then stands for both tests. Both walks take it from the same
// record values, so the forward and the adjoint decide alike.
__device__ __forceinline__ float blendFloor(float cutoffExp, float lgOpacity) {
    constexpr float kLog2Faint = -7.99435344f;   // log2(1/255)
    return fmaxf(cutoffExp + lgOpacity, kLog2Faint);
}

// The adjoint's sums over a warp, kSumRecords records at a time through shared memory:
// each lane stores six values of a record in six columns (a column: one value of one
// record, the warp's 32 lanes side by side), then lane k sums column k by eight 16-byte
// loads and adds the record's words into global memory. A lane's two pixels and a column's
// runs of four share their row, so the moments in dy come from the row sums (walk.cuh's
// rowSums) and need no columns: six values for nine words. Shared memory bounds this (its
// pipe 76% busy with nine columns); summing by shuffles (a transposed reduction) took 12
// shuffles, 12 adds and 16 selects a record.
constexpr uint32_t kSumValues = 6;    // of -2 dL/dpower: its sum, its moments t and t t; dL/dcolour r g b
constexpr uint32_t kSumRecords = 4;   // 24 of 32 lanes take a column: five records' would cost a block an SM

// ---- the blends of a training step: forward, loss and adjoint, a tile at a time ----
// One block of T*T/2 threads takes tiles off a queue (heaviest first: `order`,
// by the bit length of their pair counts, so the queue ends on light tiles)
// and, for each, runs the
// forward blend, the loss of its pixels, and the blend's adjoint, so that each
// pixel's final transmittance, last contributor and loss gradient stay in
// registers between the two walks.
//
// Forward: warp w owns an 8x8 box of the tile and each lane two pixels of it,
// (x, y) and (x + 4, y): one dy a lane, so that the terms in dy alone, and in the
// adjoint the factors dy of the moments, are formed once for both. Staging a batch of records, the block marks for each
// record the boxes its footprint can reach (a conservative test: the box's least
// power against the cutoff, with a margin); a warp then walks only the records
// marked for its box, found 32 at a time by a ballot, in list order. A pixel
// blends exactly the records it would blend walking the whole list: the
// per-pixel test decides, the box test only skips records no pixel of the box can
// pass. So the image does not depend on the tile size.
//
// Adjoint: each warp on its own once its pixels' loss gradients are known (no
// block barrier): the forward marked, for each 32-record chunk of the tile's list
// a warp walked, the records some pixel of its box blended (`live`, one word a
// chunk and box); the warp gathers those records, last first, 32 at a time into
// slots of its own (shared memory that the forward's staged records held) and walks them
// from its pixels' last contributor down. What a lane sums over its two pixels, and the
// warp over its 64 (kSumRecords records at a time), are moments of
// dP = -2 dL/dpower over the pixel offsets in the factored frame (t = dx + fr dy,
// dy): sum dP t, sum dP dy, sum dP t^2, sum dP t dy, sum dP dy^2. Each visit's warp
// sums are added into the record's gradient words in global memory as they are
// (moments, opacity times dL/dopacity, dL/dcolour); the projection's adjoint turns
// the moments into the centre and conic gradients (batchMomentsToRecordGrad, which
// applies the -1/2) and divides the opacity's word by the opacity, once a record. The loss
// has no alpha term, so dL/d(alpha out) is 0 and the colour behind a record enters
// only through S.dC, one value a pixel.
//
// kTrain false: the forward blend alone (a batched render: colour and, when
// given, depth as the plain blend makes it; no target, loss or gradients).
// kCount: also count the walks' work (evaluations and warp visits) into the
// batch's words; a step timed stage by stage counts, the captured steps do not.
template <uint32_t T, uint32_t S, uint32_t NB, bool kTrain, bool kCount>
__global__ void __launch_bounds__(S * S / 2, S == 32 ? 2 : S == 16 ? (kTrain ? 8 : 7) : 16)   // 16x16 spans: no spill
    blendStepKernel(const BatchConst B, const BatchView* __restrict__ views, const uint2* __restrict__ ranges,
                    const uint64_t* __restrict__ pairs, const uint32_t* __restrict__ values,
                    const float4* __restrict__ recs, float4* __restrict__ colour, const float* __restrict__ target,
                    float* __restrict__ loss, float* __restrict__ grads, float* __restrict__ depth,
                    uint32_t* __restrict__ words, const uint32_t* __restrict__ order, uint32_t* __restrict__ live,
                    uint8_t* __restrict__ seen) {
    constexpr uint32_t kThreads = S * S / 2;
    constexpr uint32_t kAcross = S / kBox;            // boxes across a block's span
    constexpr uint32_t kSpans = (T / S) * (T / S);    // spans (blocks' work units) a tile
    constexpr uint32_t kBoxes = (T / kBox) * (T / kBox);   // boxes a tile (the live words' row)
    // The forward's staged records: 48 bytes at one address, centre (cx, cy, depth); conic
    // (ca, fs pre-scaled, fr; log2 of the opacity); colour (r g b; the least exponent that
    // blends); then each record's boxes and index. The adjoint's, a warp's own, in the same
    // memory after the forward: 32 gathered records, what the packed arithmetic of a lane's
    // two pixels takes stored twice, so that a broadcast load gives the pair; then the
    // columns of the sums.
    struct Forward {
        float4 staged[NB][3];
        uint32_t mask[NB], rec[NB];
    };
    struct alignas(16) Gathered {   // 80 bytes: with the columns, eight blocks' fit an SM
        float nx[2], ny[2];         // minus the centre
        float ca[2], fr[2];         // the conic, its weights pre-scaled
        float fs[2], lgo[2];        // and log2 of the opacity
        float r[2], g[2], bl[2];    // the colour
        float least;                // the least exponent that blends
        uint32_t rel;               // its place in the tile's list
    };
    struct Adjoint {
        Gathered records[32];
        uint32_t rec[32];           // their records
        float sums[kSumRecords * kSumValues * kColumnStride];
    };
    constexpr size_t kAdjointBytes = kTrain ? kThreads / 32 * sizeof(Adjoint) : 0;
    constexpr size_t kBytes = sizeof(Forward) > kAdjointBytes ? sizeof(Forward) : kAdjointBytes;
    __shared__ __align__(16) unsigned char sRaw[kBytes];
    Forward& sF = *reinterpret_cast<Forward*>(sRaw);
    __shared__ uint32_t sTileBase[kMaxBatchViews];
    __shared__ uint32_t sTile;
    for (uint32_t k = threadIdx.x; k < B.views; k += kThreads) sTileBase[k] = views[k].tileBase;
    const uint64_t slotMask = (1ull << B.slotBits) - 1ull;
    const float kScale = -0.5f * 1.4426950408889634f;   // power -> base-2 exponent
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t lx = (warp % kAcross) * kBox + (lane & 3u), ly = (warp / kAcross) * kBox + (lane >> 2);
    const uint32_t sumRecord = lane / kSumValues, sumValue = lane % kSumValues;   // the column this lane sums
    uint32_t evaluated = 0;   // (pixel, record) evaluations of the forward this thread made
    uint32_t blended = 0;     // of them, those that blended
    uint32_t adjVisited = 0, adjLive = 0;   // the adjoint's evaluations, and those that blended
    uint32_t fwdVisits = 0, adjVisits = 0, adjSummed = 0;   // a warp's record visits (counted by lane 0)
    uint32_t staged = 0;      // records this thread staged
    float lossSum = 0.0f;     // this thread's pixels' share of the loss
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) {
            const uint32_t ticket = atomicAdd(&words[kBatchBlendTicket], 1u);
            sTile = ticket < B.totalTiles * kSpans ? order[ticket / kSpans] * kSpans + ticket % kSpans : 0xFFFFFFFFu;
        }
        __syncthreads();
        if (sTile == 0xFFFFFFFFu) break;
        const uint32_t tile = sTile / kSpans, span = sTile % kSpans;   // the block's span of the tile
        const uint32_t v = viewOf(sTileBase, B.views, tile);
        const BatchView& V = views[v];
        const uint32_t local = tile - V.tileBase;
        const uint32_t tx = local % V.tilesX, ty = local / V.tilesX;
        const uint32_t spanX = tx * T + (span % (T / S)) * S, spanY = ty * T + (span / (T / S)) * S;
        const float tileX0 = (float)spanX, tileY0 = (float)spanY;   // the span's first pixel
        const uint32_t px[2] = {spanX + lx, spanX + lx + 4}, py = spanY + ly;
        const uint2 range = ranges[tile];
        const float pxc[2] = {(float)px[0] + 0.5f, (float)px[1] + 0.5f}, pyc = (float)py + 0.5f;
        const size_t recBase = (size_t)v * B.count;
        // record s of this view into slot k: the factored conic's two weights pre-scaled
        // to base-2 exponent units, log2 of its opacity, the least exponent that blends,
        // and the boxes it can reach
        auto stage = [&](uint32_t k, uint32_t s) {
            if constexpr (kCount) ++staged;
            sF.rec[k] = s;
            const size_t at = (recBase + s) * 3;
            const float4 sc = recs[at + 0];
            const float4 c = recs[at + 1];
            const float4 rgb = recs[at + 2];
            sF.staged[k][0] = make_float4(sc.x, sc.y, sc.z, 0.0f);
            const float lgo = log2Of(c.w);
            sF.staged[k][1] = make_float4(c.x * kScale, c.y, c.z * kScale, lgo);
            sF.staged[k][2] = make_float4(rgb.x, rgb.y, rgb.z, blendFloor(kScale * sc.w, lgo));
            sF.mask[k] = boxMask<S>(tileX0, tileY0, sc, c.x, c.y, c.z);
        };

        // ---- forward
        float r[2] = {0.0f, 0.0f}, g[2] = {0.0f, 0.0f}, bl[2] = {0.0f, 0.0f}, Tr[2] = {1.0f, 1.0f};
        float depthSum[2] = {0.0f, 0.0f}, depthAt[2] = {-1.0f, -1.0f};   // a render's depth
        uint32_t last[2] = {0, 0};
        bool done[2];
#pragma unroll
        for (int p = 0; p < 2; ++p) done[p] = !(px[p] < V.width && py < V.height);
        for (uint32_t first = range.x; first < range.y; first += NB) {
            if (__syncthreads_count(done[0] && done[1]) == kThreads) break;
            const uint32_t count = min(NB, range.y - first);
            for (uint32_t k = threadIdx.x; k < count; k += kThreads) stage(k, gaussianOf(pairs, values, slotMask, first + k));
            __syncthreads();
            if (__all_sync(0xFFFFFFFFu, done[0] && done[1])) continue;
            for (uint32_t base = 0; base < count; base += 32) {
                const uint32_t m = base + lane < count ? sF.mask[base + lane] : 0u;
                uint32_t todo = __ballot_sync(0xFFFFFFFFu, (m >> warp) & 1u);
                uint32_t laneBits = 0;   // the records of this chunk a pixel of this lane blended
                while (todo) {
                    const uint32_t j = base + (uint32_t)__ffs(todo) - 1u;
                    todo &= todo - 1u;
                    if constexpr (kCount) ++fwdVisits;
                    const float4 ce = sF.staged[j][0];
                    const float4 k = sF.staged[j][1];
                    const float4 cc = sF.staged[j][2];
                    const float dy = pyc - ce.y;
                    const float ey = __fmaf_rn(k.z * dy, dy, k.w);
                    bool hit = false;
                    // both pixels evaluated without branching: a pixel that does not blend the
                    // record (done, outside the cutoff, or under 1/255) takes alpha 0, which
                    // leaves its sums and transmittance as they were
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        const float t = __fmaf_rn(k.y, dy, pxc[p] - ce.x);
                        const float e = __fmaf_rn(k.x * t, t, ey);
                        const float a0 = fminf(0.99f, fastExp2(e));
                        const bool blend = !done[p] && e >= cc.w;
                        if constexpr (kCount) { evaluated += done[p] ? 0u : 1u; blended += blend ? 1u : 0u; }
                        const float alpha = blend ? a0 : 0.0f;
                        const float w = Tr[p] * alpha;
                        r[p] = __fmaf_rn(w, cc.x, r[p]);
                        g[p] = __fmaf_rn(w, cc.y, g[p]);
                        bl[p] = __fmaf_rn(w, cc.z, bl[p]);
                        if constexpr (!kTrain) depthSum[p] = __fmaf_rn(w, ce.z, depthSum[p]);
                        Tr[p] = __fmaf_rn(-Tr[p], alpha, Tr[p]);   // T (1 - alpha), one rounding
                        last[p] = blend ? first - range.x + j + 1 : last[p];
                        if constexpr (!kTrain)
                            if (blend && depthAt[p] < 0.0f && 1.0f - Tr[p] >= B.depthThreshold) depthAt[p] = ce.z;
                        done[p] = done[p] || Tr[p] < 1e-4f;
                        hit = hit || blend;
                    }
                    if constexpr (kTrain) laneBits |= hit ? 1u << (j - base) : 0u;
                }
                // the records of this chunk some pixel of the box blended
                const uint32_t liveWord = kTrain ? __reduce_or_sync(0xFFFFFFFFu, laneBits) : 0u;
                if constexpr (kTrain) {
                    if (lane == 0)
                        live[((size_t)(range.x >> 5) + tile + ((first - range.x + base) >> 5)) * kBoxes +
                             span * (kAcross * kAcross) + warp] = liveWord;
                    // the records some pixel blended take a gradient in the adjoint: mark them
                    // (lane l for record base + l; a plain store, every writer stores 1), by which
                    // the projection's adjoint groups Gaussians
                    if ((liveWord >> lane) & 1u) seen[recBase + sF.rec[base + lane]] = 1u;
                }
                if (__all_sync(0xFFFFFFFFu, done[0] && done[1])) break;
            }
        }

        if constexpr (!kTrain) {
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                if (!(px[p] < V.width && py < V.height)) continue;
                const float coverage = 1.0f - Tr[p];
                const uint32_t at = V.pixelBase + py * V.width + px[p];
                colour[at] = make_float4(r[p] + Tr[p] * B.bg[0], g[p] + Tr[p] * B.bg[1], bl[p] + Tr[p] * B.bg[2],
                                         coverage + Tr[p] * B.bg[3]);
                if (depth)
                    depth[at] = B.depthMode == 0 ? (coverage > 1e-6f ? depthSum[p] / coverage : 0.0f)
                                                 : fmaxf(depthAt[p], 0.0f);
            }
            continue;
        }

        // ---- the pixels' colour, the loss (the view's mean L2 over its pixels and r g b) and its gradient
        Px<2> sd, dR, dG, dB;
        bool wild = false;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            dR.v[p] = dG.v[p] = dB.v[p] = 0.0f;
            if (px[p] < V.width && py < V.height) {
                const uint32_t at = V.pixelBase + py * V.width + px[p];
                const float coverage = 1.0f - Tr[p];
                const float4 c = make_float4(r[p] + Tr[p] * B.bg[0], g[p] + Tr[p] * B.bg[1],
                                             bl[p] + Tr[p] * B.bg[2], coverage + Tr[p] * B.bg[3]);
                colour[at] = c;
                const float er = c.x - target[(size_t)at * 3 + 0], eg = c.y - target[(size_t)at * 3 + 1],
                            eb = c.z - target[(size_t)at * 3 + 2];
                lossSum += (er * er + eg * eg + eb * eb) * V.lossScale;
                const float k2 = 2.0f * V.lossScale;
                if (last[p] != 0u) {   // a pixel that blended nothing gives no gradient, whatever its target holds
                    dR.v[p] = k2 * er;
                    dG.v[p] = k2 * eg;
                    dB.v[p] = k2 * eb;
                }
            }
            sd.v[p] = (B.bg[0] * dR.v[p] + B.bg[1] * dG.v[p]) + B.bg[2] * dB.v[p];   // S.dC, S the colour behind
            wild = wild || !(((fabsf(dR.v[p]) + fabsf(dG.v[p])) + fabsf(dB.v[p])) + fabsf(sd.v[p]) < kWalkLimit);
        }
        // a gradient that is not finite, or whose products may not be: the box's walk then leaves the
        // pixels that do not blend a record out of its sums one by one, as alpha 0 does not
        wild = __any_sync(0xFFFFFFFFu, wild);

        // ---- adjoint: each warp on its own, over the records its box blended, last first
        // (the forward's live bits), gathered 32 at a time into the warp's own slots; no
        // block barrier, no staging and no box tests
        __syncthreads();   // the block's warps are done with the staged records, whose memory the adjoint takes
        Adjoint& sA = reinterpret_cast<Adjoint*>(sRaw)[warp];
        const Px<2> xc{{pxc[0], pxc[1]}}, yc = both<2>(pyc);
        const float boxRow = tileY0 + (float)((warp / kAcross) * kBox) + 0.5f;   // the box's first row
        Px<2> light{{Tr[0], Tr[1]}};   // the pixels' transmittance, from the last record back
        const uint32_t warpLast = __reduce_max_sync(0xFFFFFFFFu, max(last[0], last[1]));
        const uint32_t nChunks = (warpLast + 31u) >> 5;
        const uint32_t* liveOf = live + ((size_t)(range.x >> 5) + tile) * kBoxes + span * (kAcross * kAcross) + warp;
        for (int32_t hi = (int32_t)nChunks - 1; hi >= 0; hi -= 32) {
            // lane l: the live bits of chunk hi - l (records 32 c .. 32 c + 31 of the tile)
            const int32_t ch = hi - (int32_t)lane;
            const uint32_t word = ch >= 0 ? liveOf[(size_t)ch * kBoxes] : 0u;
            const uint32_t n = __popc(word);
            uint32_t incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= (uint32_t)o) incl += u;
            }
            const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
            const uint32_t excl = incl - n;
            for (uint32_t r0 = 0; r0 < total; r0 += 32) {
                // the records of ranks r0 .. r0 + 31 (ranked last first) into the warp's slots:
                // lane q takes rank r0 + q
                const uint32_t want = r0 + lane;
                uint32_t c, bit;
                liveRecord(word, excl, want, c, bit);
                const uint32_t cnt = min(32u, total - r0);   // lane < cnt exactly when want < total
                if (lane < cnt) {
                    const uint32_t rel = (uint32_t)(hi - (int32_t)c) * 32u + bit;
                    const uint32_t gs = gaussianOf(pairs, values, slotMask, range.x + rel);
                    const size_t at = (recBase + gs) * 3;
                    const float4 sc = recs[at + 0];
                    const float4 k = recs[at + 1];
                    const float4 rgb = recs[at + 2];
                    const float lgo = log2Of(k.w), ca = k.x * kScale, fs = k.z * kScale;
                    Gathered& G = sA.records[lane];
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        G.nx[p] = -sc.x; G.ny[p] = -sc.y;
                        G.ca[p] = ca; G.fr[p] = k.y; G.fs[p] = fs; G.lgo[p] = lgo;
                        G.r[p] = rgb.x; G.g[p] = rgb.y; G.bl[p] = rgb.z;
                    }
                    G.least = blendFloor(kScale * sc.w, lgo);
                    G.rel = rel;
                    sA.rec[lane] = (uint32_t)(recBase + gs);
                }
                __syncwarp();
                auto walk = [&](auto wildHere) {
                constexpr bool kWild = decltype(wildHere)::value;
                for (uint32_t q0 = 0; q0 < cnt; q0 += kSumRecords) {
                    const uint32_t batch = min(kSumRecords, cnt - q0);
                    float* column = sA.sums + lane;
                    for (uint32_t q = q0; q < q0 + batch; ++q, column += kSumValues * kColumnStride) {
                        if constexpr (kCount) { ++adjVisits; ++adjSummed; }
                        const Gathered& G = sA.records[q];
                        auto pair = [](const float (&v)[2]) { return Px<2>{{v[0], v[1]}}; };
                        const Px<2> dy = yc + pair(G.ny);
                        const Px<2> t = fused(pair(G.fr), dy, xc + pair(G.nx));
                        const Px<2> e = fused(pair(G.ca) * t, t, fused(pair(G.fs) * dy, dy, pair(G.lgo)));
                        Px<2> alpha, raw, inv;
                        bool on[2];
                        // as the forward, without branching: a pixel past its last contributor or
                        // that does not blend the record takes alpha 0 (T unchanged, no terms)
#pragma unroll
                        for (int p = 0; p < 2; ++p) {
                            raw.v[p] = fastExp2(e.v[p]);
                            const float a0 = fminf(0.99f, raw.v[p]);
                            on[p] = G.rel < last[p] && e.v[p] >= G.least;
                            if constexpr (kCount) { adjVisited += G.rel < last[p] ? 1u : 0u; adjLive += on[p] ? 1u : 0u; }
                            alpha.v[p] = on[p] ? a0 : 0.0f;
                        }
                        const Px<2> om = fused(alpha, both<2>(-1.0f), both<2>(1.0f));
#pragma unroll
                        for (int p = 0; p < 2; ++p) inv.v[p] = fastRcp(om.v[p]);
                        light = light * inv;
                        const Px<2> w = light * alpha;
                        Px<2> vR = dR, vG = dG, vB = dB;
                        if constexpr (kWild) {
#pragma unroll
                            for (int p = 0; p < 2; ++p)
                                if (!on[p]) vR.v[p] = vG.v[p] = vB.v[p] = 0.0f;
                        }
                        const Px<2> cd = fused(pair(G.bl), vB, fused(pair(G.g), vG, pair(G.r) * vR));
                        // alpha dL/dalpha where alpha is not clamped (dL/dalpha = T before it
                        // times (c - S).dC): the opacity times dL/dopacity, and -2 dL/dpower
                        Px<2> u = fused(sd, both<2>(-1.0f), cd);
                        if constexpr (kWild) {
#pragma unroll
                            for (int p = 0; p < 2; ++p)
                                if (!on[p]) u.v[p] = 0.0f;
                        }
                        Px<2> dP = w * u;
                        sd = fused(alpha, u, sd);
#pragma unroll
                        for (int p = 0; p < 2; ++p) dP.v[p] = raw.v[p] < 0.99f ? dP.v[p] : 0.0f;
                        const Px<2> dPt = dP * t, dPtt = dPt * t, wr = w * vR, wg = w * vG, wb = w * vB;
                        column[0 * kColumnStride] = dP.v[0] + dP.v[1];
                        column[1 * kColumnStride] = dPt.v[0] + dPt.v[1];
                        column[2 * kColumnStride] = dPtt.v[0] + dPtt.v[1];
                        column[3 * kColumnStride] = wr.v[0] + wr.v[1];
                        column[4 * kColumnStride] = wg.v[0] + wg.v[1];
                        column[5 * kColumnStride] = wb.v[0] + wb.v[1];
                    }
                    __syncwarp();
                    // lane k sums column k and adds what it gives into the record's words in global
                    // memory (reductions, not read back): the five moments, dL/dalpha and dL/dcolour,
                    // which the projection's adjoint turns into centre and conic gradients (linear in
                    // the moments, so sums from every box, tile and batch add up). A gathered record's
                    // forward live bit says a pixel of this box blended it; sums that come to zero
                    // (all its pixels clamped) are not added.
                    if (lane < batch * kSumValues) {
                        const Gathered& G = sA.records[q0 + sumRecord];
                        const RowSums v = rowSums<8>(sA.sums + lane * kColumnStride, boxRow, G.ny[0]);
                        float* words = grads + (size_t)sA.rec[q0 + sumRecord] * kGradWords;
                        // an opacity over 1 takes no geometry or opacity gradient (its kernel has no moments)
                        const bool some = v.sum != 0.0f || v.first != 0.0f || v.second != 0.0f;
                        if (some && (sumValue >= 3 || G.lgo[0] <= 0.0f)) {
                            // words: moments t, dy, t t, t dy, dy dy; the opacity's; the colour's
                            atomicAdd(words + (sumValue == 0 ? 5u : sumValue == 1 ? 0u : sumValue == 2 ? 2u : 3u + sumValue),
                                      v.sum);
                            if (sumValue < 2) atomicAdd(words + (sumValue == 0 ? 1u : 3u), v.first);
                            if (sumValue == 0) atomicAdd(words + 4, v.second);
                        }
                    }
                    __syncwarp();   // the next records' values overwrite the columns
                }
                };
                // out of the way: laid out among the other it cost the 16 mixed views 1.7%, here 0.3%
                if (__builtin_expect(wild, 0)) walk(std::true_type());
                else walk(std::false_type());
                __syncwarp();   // the next round's gathers overwrite the slots
            }
        }
    }
    if constexpr (kTrain) {
        // the loss: the threads' shares summed in 64 bits (a warp, the batch's word, and the last
        // block to finish writes it): thousands of 32-bit atomic additions into one word each
        // rounded it, which cost it up to 2e-6 of its value
        double sum = (double)lossSum;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
        double* total = reinterpret_cast<double*>(words + kBatchLoss);
        if (lane == 0 && sum != 0.0) atomicAdd(total, sum);
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0 && atomicAdd(&words[kBatchLossBlocks], 1u) == gridDim.x - 1) {
            __threadfence();
            *loss = (float)*reinterpret_cast<volatile double*>(total);
        }
    }
    if constexpr (!kCount) return;
    // the work counts: a warp's sums, one atomic each
    const uint32_t visits = lane == 0;   // a warp's visits, once
    const uint32_t counts[8] = {evaluated, blended, adjVisited, adjLive, fwdVisits * visits, adjVisits * visits,
                                adjSummed * visits, staged};
    const uint32_t at[8] = {kBatchEvaluated, kBatchBlended, kBatchAdjVisited, kBatchAdjLive, kBatchFwdVisits,
                            kBatchAdjVisits, kBatchAdjSummed, kBatchStaged};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        uint64_t e = counts[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xFFFFFFFFu, e, o);
        if (lane == 0 && e) atomicAdd(reinterpret_cast<unsigned long long*>(words + at[c]), (unsigned long long)e);
    }
}

template <typename K>
int residentGrid(K kernel, int threads, int sms) {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0);
    return (n > 0 ? n : 1) * sms;
}

template <uint32_t T, uint32_t S, uint32_t NB>
cudaError_t stepWith(const BatchConst& B, const BlendLaunch& L, cudaStream_t stream, float4* colour,
                     const float* target, float* loss, float* grads, float* depth) {
    if (target && L.count) {
        const int grid = residentGrid(blendStepKernel<T, S, NB, true, true>, S * S / 2, L.sms);
        blendStepKernel<T, S, NB, true, true><<<grid, S * S / 2, 0, stream>>>(
            B, L.views, L.ranges, L.pairs, L.values, L.recs, colour, target, loss, grads, nullptr, L.words, L.order,
            L.live, L.seen);
    } else if (target) {
        const int grid = residentGrid(blendStepKernel<T, S, NB, true, false>, S * S / 2, L.sms);
        blendStepKernel<T, S, NB, true, false><<<grid, S * S / 2, 0, stream>>>(
            B, L.views, L.ranges, L.pairs, L.values, L.recs, colour, target, loss, grads, nullptr, L.words, L.order,
            L.live, L.seen);
    } else {
        const int grid = residentGrid(blendStepKernel<T, S, NB, false, false>, S * S / 2, L.sms);
        blendStepKernel<T, S, NB, false, false><<<grid, S * S / 2, 0, stream>>>(
            B, L.views, L.ranges, L.pairs, L.values, L.recs, colour, nullptr, nullptr, nullptr, depth, L.words,
            L.order, nullptr, nullptr);
    }
    return cudaGetLastError();
}

}   // namespace

#define ATH_BLEND_CASES(CALL)                                                                              \
    CALL(8, 64) CALL(8, 128) CALL(8, 256) CALL(8, 512) CALL(16, 64) CALL(16, 128) CALL(16, 256) CALL(16, 512)     \
    CALL(32, 64) CALL(32, 128) CALL(32, 256) CALL(32, 512)

cudaError_t launchBatchBlendStep(const BatchConst& B, const BlendLaunch& L, cudaStream_t stream, float4* colour,
                                 const float* target, float* loss, float* grads, float* depth) {
#define ATH_CASE(T_, NB_) \
    if (L.tile == T_ && L.blockBatch == NB_) \
        return stepWith<T_, (T_ > kBlendSpan ? kBlendSpan : T_), NB_>(B, L, stream, colour, target, loss, grads, depth);
    ATH_BLEND_CASES(ATH_CASE)
#undef ATH_CASE
    return cudaErrorInvalidValue;
}

}   // namespace ath
