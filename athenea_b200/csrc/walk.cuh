// What the plain path's two walks over a tile's list share: the blend (blend.cu)
// and its adjoint (backward.cu). A warp owns a box of pixels, kPx of them a lane,
// and walks only the records of its tile that can reach the box. Which records a
// pixel blends, and every rounding of what it blends, are the reference's: both
// files build with --fmad=false, and where a product and a sum are fused here it
// is written, and either exact or outside what the reference computes.
#pragma once

#include <cstdint>
#include <type_traits>

#include "raster_types.cuh"
#include "splat_math.cuh"

namespace ath {

// ---- a lane's pixels: one, or two handled as packed pairs of 32-bit numbers ------
// sm_100a multiplies and adds two 32-bit pairs in one instruction, each lane of the
// pair rounded on its own; the walks are bound by instruction issue.
template <int kPx>
struct Px {
    float v[kPx];
};
template <int kPx>
__device__ __forceinline__ Px<kPx> both(float a) {
    Px<kPx> r;
#pragma unroll
    for (int p = 0; p < kPx; ++p) r.v[p] = a;
    return r;
}
__device__ __forceinline__ Px<1> operator*(Px<1> a, Px<1> b) { return {{a.v[0] * b.v[0]}}; }
__device__ __forceinline__ Px<1> operator+(Px<1> a, Px<1> b) { return {{a.v[0] + b.v[0]}}; }
__device__ __forceinline__ Px<1> fused(Px<1> a, Px<1> b, Px<1> c) { return {{__fmaf_rn(a.v[0], b.v[0], c.v[0])}}; }
// A packed product is a fused multiply-add of -0 that the compiler cannot see is one (its
// rounding is the product's, the sign of a zero included): a plain packed product it fuses
// with the sum it goes into, even where contraction is off.
static __constant__ float2 kMinusZero = {-0.0f, -0.0f};
__device__ __forceinline__ Px<2> operator*(Px<2> a, Px<2> b) {
    const float2 r = __ffma2_rn(make_float2(a.v[0], a.v[1]), make_float2(b.v[0], b.v[1]), kMinusZero);
    return {{r.x, r.y}};
}
__device__ __forceinline__ Px<2> operator+(Px<2> a, Px<2> b) {
    const float2 r = __fadd2_rn(make_float2(a.v[0], a.v[1]), make_float2(b.v[0], b.v[1]));
    return {{r.x, r.y}};
}
__device__ __forceinline__ Px<2> fused(Px<2> a, Px<2> b, Px<2> c) {
    const float2 r = __ffma2_rn(make_float2(a.v[0], a.v[1]), make_float2(b.v[0], b.v[1]), make_float2(c.v[0], c.v[1]));
    return {{r.x, r.y}};
}

// The box of a warp, and its boxes in a 16x16 tile: 8x8 pixels with two a lane, (x, y)
// and (x + 4, y); 8x4 with one.
template <int kPx>
struct Box {
    static constexpr uint32_t kWidth = 8, kHeight = 4 * kPx;
    static constexpr uint32_t kCount = (kTile / kWidth) * (kTile / kHeight);
    static constexpr uint32_t kThreads = kCount * 32;
    // the box's first pixel in its tile, and the lane's first pixel in the box
    static __device__ __forceinline__ uint32_t x0(uint32_t box) { return (box % (kTile / kWidth)) * kWidth; }
    static __device__ __forceinline__ uint32_t y0(uint32_t box) { return (box / (kTile / kWidth)) * kHeight; }
    static __device__ __forceinline__ uint32_t laneX(uint32_t lane) { return kPx == 2 ? lane & 3u : lane & 7u; }
    static __device__ __forceinline__ uint32_t laneY(uint32_t lane) { return kPx == 2 ? lane >> 2 : lane >> 3; }
};

// Images whose boxes of two pixels a lane are fewer than this many an SM take boxes of
// one pixel a lane: half the work a warp, twice the warps, where warps are too few to
// hide each other's latency and the longest lists' boxes end last. A training pass, whose
// adjoint reads and tests each record once a box, does so up to 64 boxes an SM, a frame up to 128.
// By one and by two: frames of 100k splats at 960x540 (55 an SM) 218 and 246 us, of 1.5M at
// 1280x720 (97) 613 and 626, at 1920x1080 (221) 818 and 813; passes over 500k Gaussians at
// 960x540 708 and 729 us, at 1280x720 828 and 789.
inline bool onePixelBoxes(uint32_t tiles, uint32_t sms, bool training) {
    return tiles * Box<2>::kCount < sms * (training ? 64u : 128u);
}

// The live bits a differentiable frame keeps: chunk c of tile t's list (its records 32 c
// to 32 c + 31) and box b at word ((range start >> 5) + t + c) * boxes + b, bit k set when
// some pixel of the box blended the chunk's record k. Tiles never overlap.
inline size_t frameLiveWords(uint64_t pairs, uint32_t tiles) {
    return (size_t)(pairs / 32 + tiles + 2) * Box<1>::kCount;
}

// The live record of rank `want` among those of a warp's 32 chunks, last first: lane l
// holds `word`, the live bits of the l-th chunk from the end, and `excl`, how many live
// records the chunks of the lanes before it hold. `chunk` is the lane whose chunk the
// record is in (the last whose count is at most the rank, a search over the lanes'
// counts), `bit` its bit there (the set bit of the remaining rank, counted down from bit
// 31, a search over the word's halves, quarters, ...). Called by all 32 lanes.
__device__ __forceinline__ void liveRecord(uint32_t word, uint32_t excl, uint32_t want, uint32_t& chunk, uint32_t& bit) {
    chunk = 0;
#pragma unroll
    for (uint32_t step = 16; step; step >>= 1)
        if (__shfl_sync(0xFFFFFFFFu, excl, chunk + step) <= want) chunk += step;
    const uint32_t w = __shfl_sync(0xFFFFFFFFu, word, chunk);
    uint32_t rem = want - __shfl_sync(0xFFFFFFFFu, excl, chunk);
    bit = 31;
#pragma unroll
    for (uint32_t step = 16; step; step >>= 1) {
        const uint32_t below = __popc((w >> (bit - step + 1u)) & ((1u << step) - 1u));
        if (below <= rem) {
            rem -= below;
            bit -= step;
        }
    }
}

// The sums of a column: 32 floats, the warp's lanes side by side, four lanes a row of the
// box. `sum`, and with each value times its row's dy, the offset from the record's centre,
// and dy dy (`first`, `second`): a lane's pixels share their row, so a moment in y is taken
// over rows here rather than a pixel at a time. About the centre from the start, each row's
// dy rounded as the pixels' own: moments about another row, shifted to the centre
// afterwards, cancel for a footprint of about a pixel (sigma 0.55: the conic's c off by
// 1.4e-6 of the sum of its terms' sizes, here 6.5e-8). Two rows at a time.
struct RowSums {
    float sum, first, second;
};
template <int kRows>
__device__ __forceinline__ RowSums rowSums(const float* column, float firstRow, float minusCentre) {
    static_assert(kRows == 8 || kRows == 4, "8x8 boxes take four lanes a row, 8x4 ones eight");
    const float4* in = reinterpret_cast<const float4*>(column);
    const float firstDy = firstRow + minusCentre;   // exact, as the whole numbers added are, where the centre is near
    Px<2> dy{{firstDy, firstDy + 1.0f}}, sum, first, second;
#pragma unroll
    for (int row = 0; row < kRows; row += 2) {
        Px<2> s;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            float4 v = in[(row + k) * (8 / kRows)];
            if (kRows == 4) {
                const float4 u = in[(row + k) * 2 + 1];
                v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
            }
            const Px<2> two = Px<2>{{v.x, v.y}} + Px<2>{{v.z, v.w}};
            s.v[k] = two.v[0] + two.v[1];
        }
        if (row) dy = dy + both<2>(2.0f);
        const Px<2> moment = s * dy;
        sum = row ? sum + s : s;
        first = row ? first + moment : moment;
        second = row ? fused(moment, dy, second) : moment * dy;
    }
    return {sum.v[0] + sum.v[1], first.v[0] + first.v[1], second.v[0] + second.v[1]};
}
constexpr uint32_t kColumnStride = 36;   // floats: 16-byte aligned, eight lanes' loads in eight banks of four

// ---- can a record reach a box? ---------------------------------------------------
// False only when no pixel centre of [x0, x0 + w] x [y0, y0 + h] passes the walks' test
// power <= cutoff, as they round it. The least power over the box lies on an edge that
// faces the centre; the margin (1e-5 of the largest term the power can have over the
// box, some 80 roundings) covers the rounding of the walks' power, whose terms cancel
// for a thin footprint, and of this one.
__device__ __forceinline__ bool reachesBox(float4 screen, float4 conic, float x0, float y0, float w, float h) {
    const float a = conic.x, b = conic.y, c = conic.z;
    const float lox = x0 - screen.x, hix = lox + w, loy = y0 - screen.y, hiy = loy + h;
    const float ex = clampf(0.0f, lox, hix), ey = clampf(0.0f, loy, hiy);   // the box's point nearest the centre
    if (!(a > 1e-12f && c > 1e-12f)) return true;
    const float X = fmaxf(fabsf(lox), fabsf(hix)), Y = fmaxf(fabsf(loy), fabsf(hiy));
    const float most = __fmaf_rn(a * X, X, __fmaf_rn(2.0f * fabsf(b) * X, Y, (c * Y) * Y));
    const float limit = __fmaf_rn(1e-5f, most, __fmaf_rn(screen.w, 1.0001f, 1e-4f));
    float least = ex == 0.0f && ey == 0.0f ? 0.0f : 3.4e38f;
    if (ex != 0.0f) {
        const float y = clampf(__fdividef(-b * ex, c), loy, hiy);
        least = __fmaf_rn(a * ex, ex, y * __fmaf_rn(c, y, 2.0f * b * ex));
    }
    if (ey != 0.0f) {
        const float x = clampf(__fdividef(-b * ey, a), lox, hix);
        least = fminf(least, __fmaf_rn(c * ey, ey, x * __fmaf_rn(a, x, 2.0f * b * ey)));
    }
    return !(least > limit);
}

// Colours and gradients below this have finite products, so that a factor of 0 takes a
// pixel's term out of a sum; past it the walks choose the pixels one by one.
constexpr float kWalkLimit = 1e18f;

// ---- a record as a warp's walk holds it ------------------------------------------
// Values the packed arithmetic takes are stored once a pixel of the lane, so that a
// broadcast load gives the pair.
template <int kPx>
struct alignas(16) WalkRecord {
    float nx[kPx], ny[kPx];        // minus the centre
    float a[kPx], b2[kPx];         // the conic's a, and twice its b
    float c[kPx], alpha[kPx];      // its c; the opacity
    float r[kPx], g[kPx];
    float bl[kPx], z[kPx];
    float cutoff;
    uint32_t odd;                  // 1: an opacity over 1, or a colour that is not finite or past kWalkLimit
    uint32_t slot, place;          // the record's slot; its place in the tile's list

    __device__ __forceinline__ void set(float4 screen, float4 conic, float4 colour, uint32_t atSlot, uint32_t atPlace) {
        const float opacity = fabsf(conic.w);
#pragma unroll
        for (int p = 0; p < kPx; ++p) {
            nx[p] = -screen.x; ny[p] = -screen.y;
            a[p] = conic.x; b2[p] = 2.0f * conic.y; c[p] = conic.z; alpha[p] = opacity;
            r[p] = colour.x; g[p] = colour.y; bl[p] = colour.z; z[p] = screen.z;
        }
        cutoff = screen.w;
        const float sum = ((fabsf(colour.x) + fabsf(colour.y)) + fabsf(colour.z)) + fabsf(screen.z);
        odd = opacity <= 1.0f && sum < kWalkLimit ? 0u : 1u;
        slot = atSlot;
        place = atPlace;
    }
    // A record no pixel blends.
    __device__ __forceinline__ void setNone() {
        set(make_float4(0.0f, 0.0f, 0.0f, -3.4e38f), make_float4(0.0f, 0.0f, 0.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f),
            0u, 0u);
    }
    static __device__ __forceinline__ Px<kPx> px(const float (&m)[kPx]) {
        Px<kPx> o;
#pragma unroll
        for (int p = 0; p < kPx; ++p) o.v[p] = m[p];
        return o;
    }
};

// exp_f for a walk's argument -power / 2, of a pixel inside the cutoff (power at most 34):
// the same reduction, polynomial and roundings, without the cases outside [-86, 88] and
// with the scaling by 2^n as one integer addition to the exponent. A power below -176, or
// one that is not a number, gives 2^127 or so: an alpha of 0.99, as exp_f's infinity does
// (and as min(0.99, not a number) does). n ln2's high part is exact, so its subtraction
// can be fused.
template <int kPx>
__device__ __forceinline__ Px<kPx> expWalk(Px<kPx> power) {
    Px<kPx> x;
#pragma unroll
    for (int p = 0; p < kPx; ++p) x.v[p] = fminf(-0.5f * power.v[p], 88.0f);
    const Px<kPx> magic = both<kPx>(12582912.0f);   // 1.5 2^23: the sum rounds to a whole number
    const Px<kPx> t = x * both<kPx>(1.44269502162933349609375f) + magic;
    const Px<kPx> n = t + both<kPx>(-12582912.0f);
    Px<kPx> r = fused(n, both<kPx>(-0.693115234375f), x);
    r = r + n * both<kPx>(-3.1946183298714458942413330078125e-05f);
    Px<kPx> p = both<kPx>(1.98412701138295233249664306641e-04f);
    p = p * r + both<kPx>(1.38888892251998186111450195312e-03f);
    p = p * r + both<kPx>(8.33333376795053482055664062500e-03f);
    p = p * r + both<kPx>(4.16666679084300994873046875000e-02f);
    p = p * r + both<kPx>(1.66666671633720397949218750000e-01f);
    p = p * r + both<kPx>(0.5f);
    p = p * r + both<kPx>(1.0f);
    p = p * r + both<kPx>(1.0f);
#pragma unroll
    for (int k = 0; k < kPx; ++k)
        p.v[k] = __uint_as_float(__float_as_uint(p.v[k]) + (__float_as_uint(t.v[k]) << 23));
    return p;
}

// A record at a lane's pixels: the offsets, the power, the unclamped alpha and its
// Gaussian, each rounded as splat_blend.slang:340-362 has them. kOdd: the record may be one
// of WalkRecord::odd.
template <int kPx, bool kOdd>
struct WalkPoint {
    Px<kPx> dx, dy, power, raw;

    __device__ __forceinline__ WalkPoint(const WalkRecord<kPx>& R, Px<kPx> xc, Px<kPx> yc) {
        using Rec = WalkRecord<kPx>;
        dx = xc + Rec::px(R.nx);
        dy = yc + Rec::px(R.ny);
        power = ((Rec::px(R.a) * dx) * dx + (Rec::px(R.b2) * dx) * dy) + (Rec::px(R.c) * dy) * dy;
        const Px<kPx> gauss = expWalk<kPx>(power);
        raw = Rec::px(R.alpha) * gauss;
        if (kOdd && R.alpha[0] > 1.0f) {   // Spark's harder kernel (frame.slang:337-348)
#pragma unroll
            for (int p = 0; p < kPx; ++p) raw.v[p] = falloffAlpha(R.alpha[0], gauss.v[p]);
        }
    }
};

}   // namespace ath
