// Host-side entry points of the stage kernels (one .cu each), called by the
// rasteriser's host code (host.cu).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/athenea_raster.h"

namespace ath {

struct FrameConst;
struct InstanceConst;

// host.cu: FrameParams' setters (modules/render/src/FrameParams.h:32-117)
FrameConst frameConstFor(const ath_projection& p, const ath_settings& s);
InstanceConst instanceConstFor(const ath_projection& p, const ath_settings& s, const ath_instance& in, uint32_t base);

// project.cu
uint32_t projectBlocks(uint32_t slots);   // also the look-back words of the emit
// spans: 16 bytes a slot, its rect and the tiles of it that it touches (project.cu).
// inst: the instances in device memory; a single one is passed by value, `one`, and needs none.
cudaError_t launchProject(const FrameConst& F, const InstanceConst& one, const InstanceConst* inst, uint32_t nInst, uint32_t slots,
                          uint32_t layout, bool countCulls, float4* recs, uint4* spans, uint32_t* keys, uint32_t* words,
                          cudaStream_t stream);
// The pairs (tile << 32 | slot) of the visible slots in `order` (the depth sort's; words[kWordVisible] of
// them, at most `slots`). Writes the pairs the
// buffers hold, min(pairs, capacity), into words[kWordPairsKept], and raises kStatusPairOverflow in
// words[kWordSticky] past the capacity. flags: projectBlocks(slots) words, zeroed by the caller.
cudaError_t launchEmit(const FrameConst& F, uint32_t slots, const uint32_t* order, const float4* recs,
                       const uint4* spans, uint64_t* flags, uint32_t* words, uint64_t capacity, uint64_t* pairs,
                       cudaStream_t stream);
// Ranges over the sorted pairs, *pairsDevice of them, at most `pairs`.
cudaError_t launchRanges(uint32_t pairs, const uint32_t* pairsDevice, uint32_t tiles, const uint64_t* sorted,
                         uint2* ranges, uint32_t* status, cudaStream_t stream);
// The slots' rects and first pairs, for inspection. flags (projectBlocks(slots) words) and
// ticketAndStatus (two): zeroed by the caller.
cudaError_t launchInspectSlots(const uint4* spans, uint32_t slots, uint64_t* flags, uint32_t* ticketAndStatus,
                               uint2* rects, uint32_t* offsets, cudaStream_t stream);
// The sorted pairs as (tile << 24 | depth key) and slot, for inspection.
cudaError_t launchInspectPairs(const uint64_t* pairs, uint32_t count, const uint32_t* keys, uint32_t slots,
                               uint64_t* pairKeys, uint32_t* pairSplats, cudaStream_t stream);

// sort.cu
constexpr uint32_t kSortTileKeys = 8192;   // keys a onesweep block ranks (the look-back's unit) in a large sort
uint32_t sortPasses(uint32_t bits);      // 8-bit passes, or 9-bit ones where that saves a pass
uint32_t sortHistWords();                // the words of a sort's digit histograms (every pass)
// The look-back words of any sort of at most n keys (or of n keys in tiles of tileKeys); pairs:
// 64-bit keys with values.
size_t sortFlagWords(uint32_t n, uint32_t bits, bool pairs = false, uint32_t tileKeys = 0);
uint32_t sortResultIndex(uint32_t n, uint32_t bits);
// Allows the kernels of the sorts an owner runs their shared memory.
enum SortUse : uint32_t { kSortsKeys = 1, kSortsPairs = 2, kSortsDepths = 4 };   // 64-bit keys without and with values, a frame's depths
cudaError_t sortPrepare(uint32_t uses);
// What of its histograms, look-back words and tickets a sort clears: all; the histograms
// (the words carry epochs, the tickets are the caller's); or none (the caller cleared them).
enum SortClear : uint32_t { kClearAll, kClearHistograms, kClearNone };
cudaError_t launchSort(uint64_t* keys[2], uint32_t* vals[2], uint32_t n, uint32_t bits, uint32_t* hist,
                       uint64_t* flags, uint32_t* tickets, uint32_t* status, cudaStream_t stream,
                       SortClear clear = kClearAll, uint32_t tileKeys = 0);
// The same over bits [firstBit, firstBit + bits), with the key count on the device (at most n) and,
// when epochDevice is given, epoch-tagged look-back words that need no clearing (a captured step).
cudaError_t launchSortDevice(uint64_t* keys[2], uint32_t* vals[2], uint32_t n, const uint32_t* nDevice,
                             const uint32_t* epochDevice, uint32_t firstBit, uint32_t bits, uint32_t* hist,
                             uint64_t* flags, uint32_t* tickets, uint32_t* status, cudaStream_t stream,
                             SortClear clear = kClearAll, uint32_t tileKeys = 0);

// A frame's visible splats front to back: the slots sorted stably by the low 24 bits of `keys` (left
// as they are), into slots[0], *visible of them (the culled ones, keys of kCulledKey and a reason,
// are left out; past the visible ones slots[0] holds nothing of use). sortKeys and slots: room for n
// each. hist (three passes' worth), flags and tickets: zeroed by the caller.
cudaError_t launchSortDepths(const uint32_t* keys, uint32_t* sortKeys[2], uint32_t* slots[2], uint32_t n,
                             const uint32_t* visible, uint32_t* hist, uint64_t* flags, uint32_t* tickets, uint32_t* status,
                             cudaStream_t stream);
constexpr uint32_t kDepthBits = 24;

// blend.cu
// The reference's contributionMode hooks of the blend (modes 1 and 4).
struct Contribution {
    uint32_t mode = 0;                   // 0 none, 1 weights, 2 squared change, 3 lifted mask, 4 colour gradients
    uint32_t* words = nullptr;
    const float* finalColour = nullptr;  // float4 a pixel: mode 2 the whole frame, mode 4 dL/dpixel
    const float* liftMask = nullptr;     // mode 3: a float a pixel
};

// An opaque layer under the splats (TileRasterizer::render's `under`): its
// colour (float4) and depth (float, 0 where it has nothing) a pixel.
struct Under {
    const float* colour = nullptr;
    const float* depth = nullptr;
};

// Cryptomatte: a uint id a slot in, 3 float4 layers a pixel out.
struct Matte {
    const uint32_t* ids = nullptr;        // Cryptomatte: the id a slot, the layers out, the under layer's ids
    float* out = nullptr;
    const uint32_t* underIds = nullptr;
    const uint32_t* liftSums = nullptr;   // the matte a lift told the splats: two words a slot (inside, seen)
    float* lifted = nullptr;              // and the matte a pixel it sums to
    uint32_t hard = 0;
    float threshold = 0.5f;
    uint32_t* trace = nullptr;            // the splats a pixel is made of (splat_trace.slang), kTraceWords planes
};

// What a differentiable frame keeps for its backward: per pixel the final transmittance
// and one past the last record blended; per box of pixels the records of the tile's list
// some pixel blended (walk.cuh).
struct TrainingState {
    float* finalT = nullptr;
    uint32_t* lastContrib = nullptr;
    uint32_t* live = nullptr;
    bool onePixel = false;
};

cudaError_t launchBlend(const FrameConst& F, uint32_t pairs, uint32_t slots, const uint2* ranges,
                        const uint64_t* sorted, const float4* recs, float4* colour, float* depth, float4* position,
                        const TrainingState* training, int sms, uint32_t* status, cudaStream_t stream,
                        const Contribution& contrib = Contribution{}, const Under& under = Under{},
                        const Matte& matte = Matte{});
// Whether a differentiable frame's boxes hold one pixel a lane (onePixelBoxes; always with the
// contribution or matte hooks), and the words its live bits take.
bool trainingOnePixel(const FrameConst& F, int sms, const Contribution& contrib, const Matte& matte);
size_t trainingLiveWords(const FrameConst& F, uint64_t pairs);

// backward.cu
cudaError_t launchBlendBackward(const FrameConst& F, uint32_t pairs, uint32_t slots, const uint2* ranges,
                                const uint64_t* sorted, const float4* recs, const TrainingState& training,
                                const float4* dLdColour, const float* dLdDepth,
                                const float* depthOut, float* grads, uint32_t* status, cudaStream_t stream);
// list: room for a slot each; *listed: zeroed by the caller.
cudaError_t launchProjectBackward(const FrameConst& F, const InstanceConst& I, const uint32_t* keys,
                                  const float* grads, uint32_t* list, uint32_t* listed, float4* gMeans, float4* gScales,
                                  float4* gQuats, float* gSh, int sms, cudaStream_t stream);
cudaError_t launchL2Loss(const float4* colour, const float* target, uint32_t pixels, float4* dLdColour, float* loss,
                         cudaStream_t stream);

// decode.cu
uint32_t decodeBlocks(uint32_t count);
cudaError_t launchDecode(const float* records, uint32_t count, const ath_encoding& E, float4* positions, uint4* shape,
                         uint32_t* sh, uint64_t* flags, uint32_t* words, cudaStream_t stream);

}   // namespace ath
