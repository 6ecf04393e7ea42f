// Stage (a): per-Gaussian projection -- splat/splat_project.slang:497-785 and
// :1080-1129 (projectSplat<0>, the plain entry splatProjectPlain) -- with the
// tiles each splat touches.
// Stage (b): the pairs, (tile, slot), in depth order (splat/splat_emit.slang:17-50 over
// the depth sort's slots, as the reference; the scan of their counts, which the reference
// runs as PrefixSum::apply, TileRasterizer.cpp:1088-1089, is fused in), whose stable sort by
// tile (sort.cu) gives each tile its splats front to back; and the tiles' ranges
// (splat/splat_ranges.slang:11-25).
//
// Built with --fmad=false: see splat_math.cuh.
#include <algorithm>

#include <cuda_runtime.h>

#include "gauss.cuh"
#include "kernels.h"
#include "raster_types.cuh"
#include "splat_math.cuh"

namespace ath {
namespace {

struct Fate {
    bool removed, graded;
    float opacity;
};

// common/edit.slang:46-78
__device__ Fate editFate(const EditConst& e, float px, float py, float pz, float opacity, const float s[3]) {
    Fate fate{false, false, opacity};
    if (e.active == 0) return fate;
    if (e.minOpacity > 0.0f && opacity < e.minOpacity) {
        fate.removed = true;
        return fate;
    }
    if (e.maxScale > 0.0f && fmaxf(fmaxf(fabsf(s[0]), fabsf(s[1])), fabsf(s[2])) > e.maxScale) {
        fate.removed = true;
        return fate;
    }
    const float rx = px - e.centre[0], ry = py - e.centre[1], rz = pz - e.centre[2];
    bool inside = e.shape == 1 ? ((rx * rx + ry * ry) + rz * rz) <= e.size[0] * e.size[0]
                               : (fabsf(rx) <= e.size[0] && fabsf(ry) <= e.size[1] && fabsf(rz) <= e.size[2]);
    if (e.invert != 0) inside = !inside;
    if ((e.mode == 0 && !inside) || (e.mode == 1 && inside)) {
        fate.removed = true;
        return fate;
    }
    if (inside) {
        fate.graded = true;
        fate.opacity = opacity * e.opacity;
        fate.removed = !(fate.opacity >= kFaint);
    }
    return fate;
}

// common/edit.slang:86-90
__device__ void editGrade(const EditConst& e, float c[3]) {
    float g[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) g[k] = (c[k] * e.tint[k]) * e.brightness;
    const float luma = (g[0] * 0.2126f + g[1] * 0.7152f) + g[2] * 0.0722f;
#pragma unroll
    for (int k = 0; k < 3; ++k) c[k] = fmaxf(luma + (g[k] - luma) * e.saturation, 0.0f);
}

// common/sh.slang:25-51, the view-dependent part of the colour, its three channels side by
// side: B(k, ch), the coefficient of basis k, is asked for in the order of the row, once.
template <typename Coefficient>
__device__ __forceinline__ void evaluateRest(uint32_t degree, float x, float y, float z, Coefficient B, float out[3]) {
    const float kC1 = 0.4886025119029199f;
    out[0] = out[1] = out[2] = 0.0f;
    if (degree == 0) return;
    // a run of bases: the sum of weight k times its coefficient, left to right
    auto run = [&](uint32_t first, const auto& weights, float sum[3]) {
        constexpr uint32_t n = sizeof(weights) / sizeof(weights[0]);
#pragma unroll
        for (uint32_t k = 0; k < n; ++k)
#pragma unroll
            for (uint32_t ch = 0; ch < 3; ++ch) {
                const float term = weights[k] * B(first + k, ch);
                sum[ch] = k == 0 ? term : sum[ch] + term;
            }
    };
    const float one[3] = {(-kC1) * y, kC1 * z, -(kC1 * x)};   // a - b c is a + (-b) c
    run(0, one, out);
    if (degree >= 2) {
        const float xx = x * x, yy = y * y, zz = z * z;
        const float xy = x * y, yz = y * z, xz = x * z;
        const float two[5] = {1.0925484305920792f * xy, -1.0925484305920792f * yz,
                              0.31539156525252005f * ((2.0f * zz - xx) - yy), -1.0925484305920792f * xz,
                              0.5462742152960396f * (xx - yy)};
        float t[3];
        run(3, two, t);
#pragma unroll
        for (uint32_t ch = 0; ch < 3; ++ch) out[ch] = out[ch] + t[ch];
        if (degree >= 3) {
            const float three[7] = {(-0.5900435899266435f * y) * (3.0f * xx - yy), (2.890611442640554f * xy) * z,
                                    (-0.4570457994644658f * y) * ((4.0f * zz - xx) - yy),
                                    (0.3731763325901154f * z) * ((2.0f * zz - 3.0f * xx) - 3.0f * yy),
                                    (-0.4570457994644658f * x) * ((4.0f * zz - xx) - yy), (1.445305721320277f * z) * (xx - yy),
                                    (-0.5900435899266435f * x) * (xx - 3.0f * yy)};
            float u[3];
            run(8, three, u);
#pragma unroll
            for (uint32_t ch = 0; ch < 3; ++ch) out[ch] = out[ch] + u[ch];
        }
    }
}

constexpr uint32_t kProjectThreads = 256;

// A tile of the rect (rx0, ry0, cols) at row-major index `local`: the row from a
// float quotient corrected to the exact one.
__device__ __forceinline__ void rectTile(uint32_t local, uint32_t cols, uint32_t& c, uint32_t& r) {
    r = (uint32_t)__fdividef((float)local + 0.5f, (float)cols);
    if (r * cols > local) --r;
    else if ((r + 1) * cols <= local) ++r;
    c = local - r * cols;
}

// A lane's tiles of a rect `cols` wide, 32 apart in its row-major order.
struct RectWalk {
    uint32_t cols, col, row, stepCol, stepRow;
    __device__ __forceinline__ RectWalk(uint32_t width, uint32_t lane) : cols(width) {
        rectTile(lane, cols, col, row);
        rectTile(32, cols, stepCol, stepRow);
    }
    __device__ __forceinline__ void next() {
        col += stepCol;
        row += stepRow;
        if (col >= cols) {
            col -= cols;
            ++row;
        }
    }
};

// The least lane k whose inclusive sum `incl` passes q (q below the warp's total).
__device__ __forceinline__ uint32_t ownerOf(uint32_t incl, uint32_t q) {
    uint32_t lo = 0;
#pragma unroll
    for (uint32_t step = 16; step >= 1; step >>= 1)
        if (__shfl_sync(0xFFFFFFFFu, incl, lo + step - 1u) <= q) lo += step;
    return lo;
}

__device__ __forceinline__ uint32_t warpInclusive(uint32_t v) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= (uint32_t)o) v += u;
    }
    return v;
}

// What the emit reads of a slot, 16 bytes, so that its walk in depth order touches one
// sector a splat: the rect (x0 | y0 << 16, x1 | y1 << 16) and the tiles of it the splat
// touches, bit k of (z, w) for tile k, row-major. A rect of more than kMaskTiles tiles has
// their number in z, and its tiles are tested again where its pairs are written. A culled
// slot is all zeros.
constexpr uint32_t kMaskTiles = 64;
// A rect of more than kListTiles tiles the projection counts by itself, kLargeRun tiles a lane
// at once: the list's search and loads, one after another a tile, are a large rect's whole time,
// for its warp is alone with it. Below, rects of all sizes share the list's lanes without a gap.
// 3000 splats over most of 1920x1080: 3.63 ms by the list, 1.03 now (a thread a footprint 1.66).
constexpr uint32_t kListTiles = 512, kLargeRun = 4;
__device__ __forceinline__ void spanShape(uint4 s, uint32_t& cols, uint32_t& area, uint32_t& touched) {
    cols = (s.y & 0xFFFFu) - (s.x & 0xFFFFu) + 1;
    area = cols * ((s.y >> 16) - (s.x >> 16) + 1);
    touched = area > kMaskTiles ? s.z : __popc(s.z) + __popc(s.w);
}

// One thread a slot: projectSplat<0>, its record, rect and key. The tiles are tested by
// warps: the candidates of a warp's 32 footprints (each footprint's screen rect, row-major)
// are one list, lane l taking entry 32 c + l, so a warp's work is the sum of its rects,
// where a thread a footprint took 32 times the largest (rects of hundreds of tiles apart: kListTiles). The warps of a block wait for each
// other nowhere (but where a frame counts): the last to end adds the block's sums. 1.5M
// splats at 1920x1080: 406 us, by lists 201, without a scan among the blocks 154; 6M at
// 3840x2160: 4.52 ms, 1.23, 1.07.
// kOne: a single instance, its constants among the kernel's.
template <uint32_t L, bool kOne>
__global__ void __launch_bounds__(kProjectThreads, 5)   // as its main path fits without a spill
    projectKernel(const FrameConst F, const __grid_constant__ InstanceConst one, const InstanceConst* __restrict__ inst,
                  uint32_t nInst, uint32_t slots,
                  uint32_t countCulls, float4* __restrict__ recs, uint4* __restrict__ spans,
                  uint32_t* __restrict__ keys, uint32_t* __restrict__ words) {
    __shared__ unsigned long long sPairs;
    __shared__ uint32_t sKept, sEnded;
    __shared__ uint32_t sCulled[8];
    __shared__ uint32_t sCloud[2 * kMaxClouds];   // count_splats: (visible, pairs) a cloud, this block's share
    __shared__ float4 sFoot[kProjectThreads];     // cx cy ca cb
    __shared__ float2 sFootRest[kProjectThreads]; // cc cutoff
    __shared__ uint4 sRect[kProjectThreads];      // rx0 ry0 cols rows
    if (threadIdx.x == 0) sPairs = 0, sKept = sEnded = 0;
    if (threadIdx.x < 8) sCulled[threadIdx.x] = 0;
    if (countCulls && threadIdx.x < 2 * kMaxClouds) sCloud[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t slot = blockIdx.x * kProjectThreads + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t area = 0, key = kCulledKey, cloud = 0;
    uint2 rect = make_uint2(0, 0);
    bool graded = false;
    if (slot < slots) {
        if (!kOne)
            while (cloud + 1 < nInst && slot >= inst[cloud + 1].base) ++cloud;
        const InstanceConst& I = kOne ? one : inst[cloud];
        const Gauss g = loadGauss<L>(I, slot - I.base);
        const Fate fate = editFate(I.edit, g.px, g.py, g.pz, g.opacity, g.scale);
        if (fate.removed) {
            key = kCulledKey | kCullEdit;
        } else {
            graded = fate.graded;
            const Geometry G = projectGeometry(F, I, g, fate.opacity);
            uint32_t rx0, ry0, rx1, ry1;
            if (G.cull) {
                key = kCulledKey | G.cull;
            } else if (!tileRectOf(F, G, rx0, ry0, rx1, ry1)) {
                key = kCulledKey | kCullOffscreen;
            } else {
                key = __float_as_uint(G.tz) >> 7;
                area = (rx1 - rx0 + 1) * (ry1 - ry0 + 1);
                rect = make_uint2(rx0 | (ry0 << 16), rx1 | (ry1 << 16));
                sFoot[threadIdx.x] = make_float4(G.cx, G.cy, G.ca, G.cb);
                sFootRest[threadIdx.x] = make_float2(G.cc, G.cutoff);
                sRect[threadIdx.x] = make_uint4(rx0, ry0, rx1 - rx0 + 1, ry1 - ry0 + 1);
                recs[(size_t)slot * 3 + 0] = make_float4(G.cx, G.cy, G.tz, G.cutoff);
                recs[(size_t)slot * 3 + 1] = make_float4(G.ca, G.cb, G.cc, G.alpha);
            }
        }
    }
    // the tiles touched: the warp's candidates, 32 at a time
    uint32_t touched = 0;
    unsigned long long mask = 0;
    {
        const uint32_t listed = area > kListTiles ? 0u : area;
        const uint32_t incl = warpInclusive(listed), excl = incl - listed;
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        __syncwarp();
        for (uint32_t q0 = 0; q0 < total; q0 += 32) {
            const uint32_t q = q0 + lane;
            const uint32_t owner = ownerOf(incl, min(q, total - 1u));
            const uint32_t start = __shfl_sync(0xFFFFFFFFu, excl, owner);
            bool hit = false;
            if (q < total) {
                const uint32_t k = warp * 32 + owner;
                const float4 f = sFoot[k];
                const float2 rest = sFootRest[k];
                const uint4 r = sRect[k];
                uint32_t col, row;
                rectTile(q - start, r.z, col, row);
                hit = tileTouched(F.width, F.height, f.x, f.y, f.z, f.w, rest.x, rest.y, r.x + col, r.y + row);
            }
            const uint32_t hits = __ballot_sync(0xFFFFFFFFu, hit);
            // this lane's own candidates among the 32
            const uint32_t lo = max(excl, q0), hi = min(incl, q0 + 32);
            if (lo < hi) {
                const uint32_t own = (hits >> (lo - q0)) & (0xFFFFFFFFu >> (32 - (hi - lo)));
                touched += __popc(own);
                if (lo - excl < kMaskTiles) mask |= (unsigned long long)own << (lo - excl);
            }
        }
    }
    for (uint32_t left = __ballot_sync(0xFFFFFFFFu, area > kListTiles); left; left &= left - 1u) {
        const uint32_t owner = (uint32_t)__ffs((int)left) - 1u, k = warp * 32 + owner;
        const float4 f = sFoot[k];
        const float2 rest = sFootRest[k];
        const uint4 r = sRect[k];
        RectWalk at(r.z, lane);
        uint32_t mine = 0;
        for (uint32_t q0 = lane; q0 < r.z * r.w; q0 += 32 * kLargeRun) {
            uint32_t near = 0;
#pragma unroll
            for (uint32_t j = 0; j < kLargeRun; ++j, at.next()) {
                const TileBox t(F.width, F.height, f.x, f.y, r.x + at.col, r.y + at.row);
                const int estimate = powerEstimate(f.z, f.w, rest.x, rest.y, t.lox, t.loy, t.hix, t.hiy);
                const bool here = q0 + 32 * j < r.z * r.w;
                mine += here && estimate > 0 ? 1u : 0u;
                near |= here && estimate == 0 ? 1u << j : 0u;
            }
            for (; near; near &= near - 1u) {
                uint32_t col, row;
                rectTile(q0 + 32 * ((uint32_t)__ffs((int)near) - 1u), r.z, col, row);
                mine += tileTouched(F.width, F.height, f.x, f.y, f.z, f.w, rest.x, rest.y, r.x + col, r.y + row) ? 1u : 0u;
            }
        }
        const uint32_t found = __reduce_add_sync(0xFFFFFFFFu, mine);
        if (lane == owner) touched = found;
    }
    if (area && touched == 0) key = kCulledKey | kCullNoTile;
    const bool kept = touched != 0;
    if (kept) {
        const InstanceConst& I = kOne ? one : inst[cloud];
        const uint32_t i = slot - I.base;
        const Gauss g = loadGauss<L>(I, i);
        const uint32_t degree = min(degreeOf(I.restPerColour), F.shLimit);
        const float dx = g.px - I.eye[0], dy = g.py - I.eye[1], dz = g.pz - I.eye[2];
        const float len = sqrtf((dx * dx + dy * dy) + dz * dz);
        const float x = dx / len, y = dy / len, z = dz / len;
        float rest[3];
        if constexpr (L == kLayoutPacked) {
            const uint32_t* row = I.sh + (size_t)i * I.shWords;
            evaluateRest(degree, x, y, z, [&](uint32_t k, uint32_t ch) {
                    const uint32_t word = __ldg(row + (k * 3 + ch) / 2);
                    return ((k * 3 + ch) & 1u) == 0u ? lowHalf(word) : highHalf(word);
                }, rest);
        } else if ((I.shStride & 3u) == 0 && (reinterpret_cast<uintptr_t>(I.shf) & 15u) == 0) {
            // a lane reads its own row, 192 bytes from its neighbours' at degree 3: 16 bytes a
            // load, for each load takes a line a lane
            const float4* row = reinterpret_cast<const float4*>(I.shf + (size_t)i * I.shStride);
            evaluateRest(degree, x, y, z, [&](uint32_t k, uint32_t ch) {
                    const uint32_t at = 3 + k * 3 + ch;
                    const float4 four = __ldg(row + at / 4);
                    return at % 4 == 0 ? four.x : at % 4 == 1 ? four.y : at % 4 == 2 ? four.z : four.w;
                }, rest);
        } else {
            evaluateRest(degree, x, y, z, [&](uint32_t k, uint32_t ch) { return restAt<L>(I, i, k * 3 + ch); }, rest);
        }
        float colour[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float v = g.base[k] + rest[k];
            colour[k] = I.linear != 0 ? fmaxf(v, 0.0f) : srgbToLinear(v);
        }
        if (graded) editGrade(I.edit, colour);
        recs[(size_t)slot * 3 + 2] = make_float4(colour[0], colour[1], colour[2], 0.0f);
    }
    if (slot < slots) {
        keys[slot] = key;
        const uint2 bits = area > kMaskTiles ? make_uint2(touched, 0) : make_uint2((uint32_t)mask, (uint32_t)(mask >> 32));
        spans[slot] = kept ? make_uint4(rect.x, rect.y, bits.x, bits.y) : make_uint4(0, 0, 0, 0);
        if (countCulls && !kept) atomicAdd(&sCulled[key & 7u], 1u);
        // splatCountersCloud's rows (TileRasterizer.cpp:1335-1346): the first 64 clouds one by one
        if (countCulls && kept && cloud < kMaxClouds) {
            atomicAdd(&sCloud[2 * cloud], 1u);
            atomicAdd(&sCloud[2 * cloud + 1], touched);
        }
    }
    // the block's sums, added by the last of its warps to get here
    const uint32_t warpKept = __popc(__ballot_sync(0xFFFFFFFFu, kept));
    const uint32_t warpPairs = __reduce_add_sync(0xFFFFFFFFu, touched);
    if (lane == 0) {
        if (warpKept) {
            atomicAdd(&sPairs, (unsigned long long)warpPairs);
            atomicAdd(&sKept, warpKept);
        }
        __threadfence_block();
        if (atomicAdd(&sEnded, 1u) == kProjectThreads / 32 - 1) {
            __threadfence_block();
            if (const uint32_t all = atomicAdd(&sKept, 0u)) {
                atomicAdd(&words[kWordVisible], all);
                atomicAdd(reinterpret_cast<unsigned long long*>(&words[kWordPairsLo]), atomicAdd(&sPairs, 0ull));
            }
        }
    }
    if (!countCulls) return;
    const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, touched);
    if (lane == 0 && most) atomicMax(&words[kWordMaxTiles], most);
    __syncthreads();
    if (threadIdx.x < 7 && sCulled[threadIdx.x]) atomicAdd(&words[kWordCulled + threadIdx.x], sCulled[threadIdx.x]);
    if (threadIdx.x < 2 * kMaxClouds && sCloud[threadIdx.x]) atomicAdd(&words[kWordClouds + threadIdx.x], sCloud[threadIdx.x]);
}

// Bit `k` (counted from the least) of the set bits of a 64-bit word.
__device__ __forceinline__ uint32_t setBit(uint32_t lo, uint32_t hi, uint32_t k) {
    uint32_t w = lo, at = 0;
    const uint32_t inLow = __popc(lo);
    if (k >= inLow) {
        k -= inLow;
        w = hi;
        at = 32;
    }
#pragma unroll
    for (uint32_t step = 16; step; step >>= 1) {
        const uint32_t below = __popc(w & ((1u << step) - 1u));
        if (k >= below) {
            k -= below;
            w >>= step;
            at += step;
        }
    }
    return at;
}

// splat_emit.slang:17-50 over the depth sort's slots: a pair (tile << 32 | slot) a
// touched tile, row-major over the splat's rect. A stable sort by tile then leaves each
// tile its splats in (depth key, slot) order (splat/frame.slang:17-20). A warp writes its
// 32 splats' pairs as one list, lane l pair 32 c + l, from the masks of the tiles they
// touch; where the splats' pairs start comes from a look-back over the blocks. Bound by
// the splats' records, a sector each in depth order, and the pairs' writes. With rects,
// masks, keys and offsets apart 1.5M splats took 102 us, now 73; 6M 692, now 498.
__global__ void __launch_bounds__(kProjectThreads, 8)   // it waits, mostly: by five blocks an SM 91 and 619 us
    emitKernel(const FrameConst F, uint32_t slots, const uint32_t* __restrict__ order, const float4* __restrict__ recs,
               const uint4* __restrict__ spans, uint64_t* __restrict__ flags, uint32_t* __restrict__ words,
               uint64_t capacity, uint64_t* __restrict__ pairs) {
    __shared__ uint32_t sTicket;
    __shared__ uint32_t sWarp[kProjectThreads / 32];
    __shared__ uint64_t sPrefix;
    const uint32_t visible = min(slots, words[kWordVisible]);
    if (threadIdx.x == 0) sTicket = atomicAdd(&words[kWordEmitTicket], 1u);
    __syncthreads();
    const uint32_t b = sTicket;
    if (b != 0 && b * kProjectThreads >= visible) return;   // past the visible slots: no block waits for this one
    const uint32_t i = b * kProjectThreads + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t all = (uint64_t)words[kWordPairsLo] | ((uint64_t)words[kWordPairsHi] << 32);
    if (b == 0 && threadIdx.x == 0) {
        // what the sort, the ranges and the blends take: the pairs the buffers hold
        words[kWordPairsKept] = (uint32_t)min(all, capacity);
        if (all > capacity) atomicOr(&words[kWordSticky], kStatusPairOverflow);
    }
    uint32_t slot = 0, touched, cols, area;
    uint4 span = make_uint4(0, 0, 0, 0);
    if (i < visible) {
        slot = order[i];
        if (slot < slots) span = spans[slot];
    }
    spanShape(span, cols, area, touched);
    const uint32_t incl = warpInclusive(touched), excl = incl - touched;
    if (lane == 31) sWarp[warp] = incl;
    __syncthreads();
    uint32_t warpBase = 0, blockTotal = 0;
#pragma unroll
    for (uint32_t w = 0; w < kProjectThreads / 32; ++w) {
        const uint32_t v = sWarp[w];
        warpBase += w < warp ? v : 0u;
        blockTotal += v;
    }
    if (warp == 0) {
        const uint64_t prefix = lookbackExclusive(flags, b, blockTotal, &words[kWordSticky]);
        if (lane == 0) sPrefix = prefix;
    }
    __syncthreads();
    const uint64_t base = sPrefix + warpBase;
    const bool large = area > kMaskTiles;
    const uint32_t anyLarge = __ballot_sync(0xFFFFFFFFu, large);
    const uint32_t rect0 = span.x, maskLo = span.z, maskHi = span.w;
    // the list leaves out rects too large for a mask, whose pairs lie between the others' (walking past
    // them there was a third of the kernel where splats cover the image: 4.0 ms for 3000, now 2.8)
    uint32_t listIncl = incl, gap = 0;
    if (anyLarge) {
        listIncl = warpInclusive(large ? 0u : touched);
        gap = incl - listIncl;
    }
    const uint32_t listExcl = listIncl - (large ? 0u : touched), total = __shfl_sync(0xFFFFFFFFu, listIncl, 31);
    for (uint32_t q0 = 0; q0 < total; q0 += 32) {
        const uint32_t q = q0 + lane;
        const uint32_t owner = ownerOf(listIncl, min(q, total - 1u));
        const uint32_t k = q - __shfl_sync(0xFFFFFFFFu, listExcl, owner);
        const uint32_t oRect = __shfl_sync(0xFFFFFFFFu, rect0, owner), oCols = __shfl_sync(0xFFFFFFFFu, cols, owner);
        const uint32_t oLo = __shfl_sync(0xFFFFFFFFu, maskLo, owner), oHi = __shfl_sync(0xFFFFFFFFu, maskHi, owner);
        const uint32_t oSlot = __shfl_sync(0xFFFFFFFFu, slot, owner);
        const uint32_t skipped = anyLarge ? __shfl_sync(0xFFFFFFFFu, gap, owner) : 0u;
        if (q >= total) continue;
        uint32_t col, row;
        rectTile(setBit(oLo, oHi, k), oCols, col, row);
        const uint32_t tile = ((oRect >> 16) + row) * F.tilesX + (oRect & 0xFFFFu) + col;
        const uint64_t at = base + skipped + q;
        if (at < capacity) pairs[at] = ((uint64_t)tile << 32) | oSlot;
    }
    // rects too large for a mask: the warp tests their tiles again, one splat after another
    for (uint32_t left = anyLarge; left; left &= left - 1u) {
        const uint32_t owner = (uint32_t)__ffs((int)left) - 1u;
        const uint32_t oSlot = __shfl_sync(0xFFFFFFFFu, slot, owner), oRect = __shfl_sync(0xFFFFFFFFu, rect0, owner);
        const uint32_t oCols = __shfl_sync(0xFFFFFFFFu, cols, owner), oArea = __shfl_sync(0xFFFFFFFFu, area, owner);
        const uint32_t expected = __shfl_sync(0xFFFFFFFFu, touched, owner);
        uint64_t at = base + __shfl_sync(0xFFFFFFFFu, excl, owner);
        const float4 s = recs[(size_t)oSlot * 3 + 0], k = recs[(size_t)oSlot * 3 + 1];
        uint32_t written = 0;
        for (uint32_t q0 = 0; q0 < oArea && written < expected; q0 += 32) {
            uint32_t col, row;
            rectTile(min(q0 + lane, oArea - 1u), oCols, col, row);
            const uint32_t tx = (oRect & 0xFFFFu) + col, ty = (oRect >> 16) + row;
            const bool hit = q0 + lane < oArea && tileTouched(F.width, F.height, s.x, s.y, k.x, k.y, k.z, s.w, tx, ty);
            const uint32_t hits = __ballot_sync(0xFFFFFFFFu, hit);
            const uint32_t n = written + __popc(hits & ((1u << lane) - 1u));
            if (hit && n < expected && at + n < capacity) pairs[at + n] = ((uint64_t)(ty * F.tilesX + tx) << 32) | oSlot;
            written += __popc(hits);
        }
    }
}

// The slots' rects, and the exclusive scan of the tiles they touch, for inspection.
__global__ void __launch_bounds__(kProjectThreads)
    inspectSlotsKernel(const uint4* __restrict__ spans, uint32_t slots, uint64_t* __restrict__ flags,
                       uint32_t* __restrict__ ticketAndStatus, uint2* __restrict__ rects, uint32_t* __restrict__ offsets) {
    __shared__ uint32_t sTicket;
    __shared__ uint32_t sWarp[kProjectThreads / 32];
    __shared__ uint64_t sPrefix;
    if (threadIdx.x == 0) sTicket = atomicAdd(&ticketAndStatus[0], 1u);
    __syncthreads();
    const uint32_t b = sTicket, slot = b * kProjectThreads + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint4 span = slot < slots ? spans[slot] : make_uint4(0, 0, 0, 0);
    uint32_t cols, area, touched;
    spanShape(span, cols, area, touched);
    const uint32_t incl = warpInclusive(touched);
    if (lane == 31) sWarp[warp] = incl;
    __syncthreads();
    uint32_t warpBase = 0, blockTotal = 0;
#pragma unroll
    for (uint32_t w = 0; w < kProjectThreads / 32; ++w) {
        const uint32_t v = sWarp[w];
        warpBase += w < warp ? v : 0u;
        blockTotal += v;
    }
    if (warp == 0) {
        const uint64_t prefix = lookbackExclusive(flags, b, blockTotal, &ticketAndStatus[1]);
        if (lane == 0) sPrefix = prefix;
    }
    __syncthreads();
    if (slot >= slots) return;
    rects[slot] = make_uint2(span.x, span.y);
    offsets[slot] = (uint32_t)(sPrefix + (incl - touched) + warpBase);
}

// The sorted pairs as frame.slang's two sorts have them, for inspection: (tile << 24 |
// depth key) and the slot of each.
__global__ void __launch_bounds__(256)
    inspectPairsKernel(const uint64_t* __restrict__ pairs, uint32_t count, const uint32_t* __restrict__ keys,
                       uint32_t slots, uint64_t* __restrict__ pairKeys, uint32_t* __restrict__ pairSplats) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const uint32_t slot = (uint32_t)pairs[i];
    pairKeys[i] = ((pairs[i] >> 32) << 24) | (slot < slots ? keys[slot] : 0u);
    pairSplats[i] = slot;
}

// splat_ranges.slang:11-25 over the sorted pairs; ranges were cleared first
// (splat_tiles_clear.slang). A thread takes a run of eight pairs (four 16-byte loads)
// and the pair before it, and writes a range's start and the previous range's end where
// the tile changes. `pairsDevice` holds the pair count (at most `pairs`, the grid's bound).
constexpr uint32_t kRangeRun = 8;

__global__ void __launch_bounds__(256)
    rangesKernel(uint32_t pairs, const uint32_t* __restrict__ pairsDevice, uint32_t tiles,
                 const uint64_t* __restrict__ sorted, uint2* __restrict__ ranges, uint32_t* __restrict__ status) {
    pairs = min(pairs, *pairsDevice);
    const uint64_t first = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * kRangeRun;
    if (first >= pairs) return;
    uint32_t tile[kRangeRun];
    if (first + kRangeRun <= pairs) {
        const ulonglong2* at = reinterpret_cast<const ulonglong2*>(sorted + first);
#pragma unroll
        for (uint32_t k = 0; k < kRangeRun / 2; ++k) {
            const ulonglong2 two = at[k];
            tile[2 * k] = (uint32_t)(two.x >> 32);
            tile[2 * k + 1] = (uint32_t)(two.y >> 32);
        }
    } else {
#pragma unroll
        for (uint32_t k = 0; k < kRangeRun; ++k) tile[k] = first + k < pairs ? (uint32_t)(sorted[first + k] >> 32) : 0u;
    }
    uint32_t before = first == 0 ? 0xFFFFFFFFu : (uint32_t)(sorted[first - 1] >> 32);
#pragma unroll
    for (uint32_t k = 0; k < kRangeRun; ++k) {
        const uint64_t i = first + k;
        if (i >= pairs) break;
        uint32_t t = tile[k];
        if (t >= tiles) {
            atomicOr(status, kStatusIndexRange);
            t = 0xFFFFFFFFu;
        }
        if (t != before) {
            if (t != 0xFFFFFFFFu) ranges[t].x = (uint32_t)i;
            if (before < tiles) ranges[before].y = (uint32_t)i;
        }
        if (i + 1 == pairs && t != 0xFFFFFFFFu) ranges[t].y = pairs;
        before = t;
    }
}

}   // namespace

cudaError_t launchProject(const FrameConst& F, const InstanceConst& one, const InstanceConst* inst, uint32_t nInst, uint32_t slots,
                          uint32_t layout, bool countCulls, float4* recs, uint4* spans, uint32_t* keys, uint32_t* words,
                          cudaStream_t stream) {
    if (slots == 0) return cudaSuccess;
    const uint32_t cc = countCulls ? 1u : 0u;
#define ATH_PROJECT(L_, O_)                                                                                        \
    projectKernel<L_, O_><<<projectBlocks(slots), kProjectThreads, 0, stream>>>(F, one, inst, nInst, slots, cc, recs, \
                                                                               spans, keys, words)
    if (layout == kLayoutPacked && nInst == 1) ATH_PROJECT(kLayoutPacked, true);
    else if (layout == kLayoutPacked) ATH_PROJECT(kLayoutPacked, false);
    else ATH_PROJECT(kLayoutParams, true);
#undef ATH_PROJECT
    return cudaGetLastError();
}

uint32_t projectBlocks(uint32_t slots) { return (slots + kProjectThreads - 1) / kProjectThreads; }

cudaError_t launchEmit(const FrameConst& F, uint32_t slots, const uint32_t* order, const float4* recs,
                       const uint4* spans, uint64_t* flags, uint32_t* words, uint64_t capacity, uint64_t* pairs,
                       cudaStream_t stream) {
    emitKernel<<<std::max(1u, projectBlocks(slots)), kProjectThreads, 0, stream>>>(
        F, slots, order, recs, spans, flags, words, capacity, pairs);
    return cudaGetLastError();
}

cudaError_t launchInspectSlots(const uint4* spans, uint32_t slots, uint64_t* flags, uint32_t* ticketAndStatus,
                               uint2* rects, uint32_t* offsets, cudaStream_t stream) {
    if (slots == 0) return cudaSuccess;
    inspectSlotsKernel<<<projectBlocks(slots), kProjectThreads, 0, stream>>>(spans, slots, flags, ticketAndStatus, rects, offsets);
    return cudaGetLastError();
}

cudaError_t launchInspectPairs(const uint64_t* pairs, uint32_t count, const uint32_t* keys, uint32_t slots,
                               uint64_t* pairKeys, uint32_t* pairSplats, cudaStream_t stream) {
    if (count == 0) return cudaSuccess;
    inspectPairsKernel<<<(count + 255) / 256, 256, 0, stream>>>(pairs, count, keys, slots, pairKeys, pairSplats);
    return cudaGetLastError();
}

cudaError_t launchRanges(uint32_t pairs, const uint32_t* pairsDevice, uint32_t tiles, const uint64_t* sorted,
                         uint2* ranges, uint32_t* status, cudaStream_t stream) {
    if (pairs == 0) return cudaSuccess;
    const uint32_t run = 256 * kRangeRun;
    rangesKernel<<<(uint32_t)(((uint64_t)pairs + run - 1) / run), 256, 0, stream>>>(pairs, pairsDevice, tiles, sorted,
                                                                                   ranges, status);
    return cudaGetLastError();
}

}   // namespace ath
