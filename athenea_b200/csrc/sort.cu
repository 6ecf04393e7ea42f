// Stage (c): a stable LSD radix sort of 64-bit keys (32-bit for a frame's depths)
// with 32-bit values, eight (or nine) bits a pass, in the onesweep form (Adinets and Merrill, "Onesweep: A Faster
// Least Significant Digit Radix Sort for GPUs", 2022): one read of the keys
// makes every pass's digit histogram, then each pass is a single kernel whose
// tiles rank their keys in shared memory, find where each digit of theirs
// starts by a decoupled look-back over the tiles before them, and scatter.
//
// It replaces the reference's RadixSort (modules/gpu/src/algo/RadixSort.cpp:
// 95-261; shaders/athenea/algo/radix_*.slang), which the rasteriser runs twice
// (24-bit depth keys, then tile keys). Same contract: stable, so equal keys
// keep their input order (algo/radix_common.slang:18-22), and only the low
// `bits` of a key take part.
#include <cuda_runtime.h>

#include "kernels.h"
#include "raster_types.cuh"
#include "splat_math.cuh"

namespace ath {
namespace {

constexpr uint32_t kMaxRadix = 512;     // a 9-bit pass's digits: the histograms' stride a pass
constexpr uint32_t kSortThreads = 512;
constexpr uint32_t kWarps = kSortThreads / 32;
// Keys a thread: 16 (8192-key tiles: fewer tiles for the look-back to walk), or 4 where
// 8192-key tiles would leave most SMs idle and one block's ranking would be the pass.
// 64-bit keys with values take 12: with 16 their keys, places and destinations do not fit the
// registers that two blocks an SM leave.
constexpr uint32_t kItems = 16, kSmallItems = 4, kPairItems = 12;
static_assert(kSortThreads * kItems == kSortTileKeys, "kernels.h states the sort's tile size");
// A warp ranks its items in independent chains (an 8-bit pass of 8192-key tiles: items
// 0-7 and 8-15), each with its own digit counters, so the chains' shared-memory round
// trips overlap instead of queueing behind each other; the chains are ordered
// after each other like warps.
constexpr uint32_t kMaxPasses = 8;

// `nDevice`, when given, holds the key count (a count only the device knows, as
// in a step captured in a CUDA graph); `n` is then a bound on it.
__device__ __forceinline__ uint32_t countOf(uint32_t n, const uint32_t* nDevice) {
    return nDevice ? min(n, *nDevice) : n;
}

// Digit d's slot in a per-digit table in shared memory: d with its low five bits
// XORed with the next five (a permutation within each run of 32). A warp's keys
// often hold digits 32 or 64 apart and little else (a pass over an exponent byte's
// few values beside a tile index's low bits); unswizzled, those all fall in one
// bank and their counter reads serialise.
__device__ __forceinline__ uint32_t digitSlot(uint32_t d) { return d ^ ((d >> 5) & 31u); }

// A sort's passes over bits [firstBit, firstBit + bits): `wide` digits of nine bits, then
// eights. Worked out where it is asked for: with arrays among a kernel's constants, looked up
// by pass, the one-block sort of 5k depths took 16.9 us, now 12.8.
struct SortPlan {
    uint32_t passes, bits, wide;
    __host__ __device__ uint32_t width(uint32_t p) const { return p < wide ? 9u : 8u; }
    __host__ __device__ uint32_t shift(uint32_t p) const { return 8u * p + min(p, wide); }   // from firstBit
    // a digit's bits that take part: the last one's past the sort's do not
    __host__ __device__ uint32_t mask(uint32_t p) const { return (1u << min(width(p), bits - shift(p))) - 1u; }
};

template <typename K>
__global__ void __launch_bounds__(256)
    histogramKernel(const K* __restrict__ keys, uint32_t n, const uint32_t* __restrict__ nDevice,
                    uint32_t firstBit, const SortPlan plan, uint32_t* __restrict__ hist) {
    __shared__ uint32_t sHist[kMaxPasses * kMaxRadix];
    n = countOf(n, nDevice);
    for (uint32_t j = threadIdx.x; j < plan.passes * kMaxRadix; j += blockDim.x) sHist[j] = 0;
    __syncthreads();
    // A thread takes a run of eight keys, all in flight before their counts, and counts equal
    // digits that follow each other at once: the high digits of pairs written splat by splat are
    // alike, and lanes that count the same digit wait for each other. 6M
    // splats' pairs at 3840x2160: 249 us, now 157; 8M random keys 33, now 30.
    constexpr uint32_t kRun = 8, kVector = 16 / sizeof(K);
    const bool aligned = (reinterpret_cast<uintptr_t>(keys) & 15u) == 0;
    const uint64_t threads = (uint64_t)gridDim.x * blockDim.x, me = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t first = me * kRun; first < n; first += threads * kRun) {
        const uint32_t count = (uint32_t)min((uint64_t)kRun, n - first);
        K key[kRun];
        if (aligned && count == kRun) {
#pragma unroll
            for (uint32_t k = 0; k < kRun / kVector; ++k) {
                const uint4 four = __ldg(reinterpret_cast<const uint4*>(keys + first) + k);
                if constexpr (sizeof(K) == 8) {
                    key[2 * k] = ((K)four.y << 32) | four.x;
                    key[2 * k + 1] = ((K)four.w << 32) | four.z;
                } else {
                    key[4 * k] = four.x, key[4 * k + 1] = four.y, key[4 * k + 2] = four.z, key[4 * k + 3] = four.w;
                }
            }
        } else {
#pragma unroll
            for (uint32_t k = 0; k < kRun; ++k) key[k] = k < count ? keys[first + k] : (K)0;
        }
#pragma unroll
        for (uint32_t p = 0; p < kMaxPasses; ++p) {
            if (p >= plan.passes) break;
            const uint32_t shift = firstBit + plan.shift(p), mask = plan.mask(p);
            // a frame's depths: a culled slot's key counts as no digit (a run with some of them counted by
            // a second copy of this costs more, 12 us for 1.5M slots: lanes differ; this 8.8, without 7.3)
            auto digitOf = [&](K k) {
                const uint32_t d = (uint32_t)(k >> shift) & mask;
                return sizeof(K) == 4 && k >= (K)kCulledKey ? kMaxRadix : d;
            };
            auto add = [&](uint32_t d, uint32_t times) {
                if (sizeof(K) == 8 || d < kMaxRadix) atomicAdd(&sHist[p * kMaxRadix + digitSlot(d)], times);
            };
            uint32_t run = digitOf(key[0]), length = 1;
#pragma unroll
            for (uint32_t k = 1; k < kRun; ++k) {
                if (k >= count) break;
                const uint32_t d = digitOf(key[k]);
                if (d == run) {
                    ++length;
                } else {
                    add(run, length);
                    run = d;
                    length = 1;
                }
            }
            add(run, length);
        }
    }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < plan.passes * kMaxRadix; j += blockDim.x) {
        const uint32_t c = sHist[(j / kMaxRadix) * kMaxRadix + digitSlot(j % kMaxRadix)];
        if (c) atomicAdd(&hist[j], c);
    }
}

// Exclusive scan of one value a thread over the block (kSortThreads threads).
__device__ __forceinline__ uint32_t blockExclusiveScan(uint32_t v, uint32_t* sWarp) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (uint32_t)o) incl += u;
    }
    if (lane == 31) sWarp[warp] = incl;
    __syncthreads();
    uint32_t base = 0;
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w) base += w < warp ? sWarp[w] : 0u;
    __syncthreads();
    return base + incl - v;
}

// What a pass carries beside its keys.
enum SortValues : uint32_t { kNoValues = 0, kReadValues = 1, kIndexValues = 2 };   // index: a key's place in the input

// A pass's shared memory: its keys, their place taken by its chains' digit masks while it
// ranks; then its chains' digit counters.
template <uint32_t kBits, uint32_t kPerThread>
__host__ __device__ constexpr uint32_t rankChains() { return kWarps * (kBits == 8 && kPerThread >= 16 ? 2 : 1); }
template <typename K, uint32_t kBits, uint32_t kPerThread>
__host__ __device__ constexpr size_t rankSmem() {
    const size_t keys = (size_t)kSortThreads * kPerThread * sizeof(K), masks = ((size_t)rankChains<kBits, kPerThread>() << kBits) * 4;
    return keys > masks ? keys : masks;
}
template <typename K, uint32_t kBits, uint32_t kPerThread>
constexpr size_t onesweepSmem() {
    return rankSmem<K, kBits, kPerThread>() + ((size_t)rankChains<kBits, kPerThread>() << kBits) * 4;
}

// kBits: the pass's digit width, 8 or 9 (its digits one thread each in the
// digit phase; a 9-bit pass ranks in one chain, so that its counters fit beside the keys).
// The values take the keys' shared memory once the keys are out, each thread keeping its
// items' places in the tile and its outputs' destinations in registers: with values as
// without, two blocks an SM (values beside the keys, 128 KB, left one). 8M pairs of
// 40 bits: 605 -> 549 us with the masks below. 64-bit keys with values in 8192-key tiles, the
// static sort's, are at most 128 tiles for more SMs: one block an SM, and no spill (1M pairs
// of 40 bits 136 -> 119 us, 20k 108 -> 92).
template <typename K, uint32_t kValues, uint32_t kBits, uint32_t kPerThread>
__global__ void __launch_bounds__(kSortThreads, sizeof(K) == 8 && kValues != kNoValues && kPerThread == kItems ? 1 : 2)
    onesweepKernel(const K* __restrict__ keysIn, const uint32_t* __restrict__ valsIn, K* __restrict__ keysOut,
                   uint32_t* __restrict__ valsOut, uint32_t n, uint32_t shift, uint32_t digitMask,
                   const uint32_t* __restrict__ globalHist, uint64_t* __restrict__ flags, uint32_t* __restrict__ ticket,
                   uint32_t* __restrict__ status, const uint32_t* __restrict__ nDevice,
                   const uint32_t* __restrict__ epochDevice) {
    constexpr uint32_t kRadix = 1u << kBits;
    constexpr uint32_t kCounters = rankChains<kBits, kPerThread>(), kChains = kCounters / kWarps;
    constexpr uint32_t kChainItems = kPerThread / kChains;
    constexpr uint32_t kTileKeys = kSortThreads * kPerThread;
    // The first pass of a frame's depths leaves culled slots out: the passes after it, and the emit,
    // take the visible ones alone.
    constexpr bool kDrop = kValues == kIndexValues;
    extern __shared__ __align__(16) unsigned char smem[];
    K* sKeys = reinterpret_cast<K*>(smem);
    uint32_t* sVals = reinterpret_cast<uint32_t*>(smem);
    uint32_t* sMasks = reinterpret_cast<uint32_t*>(smem);   // kCounters x kRadix, while the keys are ranked
    uint32_t* sWarpCnt = reinterpret_cast<uint32_t*>(smem + rankSmem<K, kBits, kPerThread>());   // kCounters x kRadix
    __shared__ uint32_t sTile, sKept;
    __shared__ uint32_t sStart[kRadix];
    __shared__ uint32_t sAdjust[kRadix];
    __shared__ uint32_t sScan[kWarps];

    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    n = countOf(n, nDevice);
    // Look-back words are [epoch:30][status:2][value:32]; a word of another
    // epoch reads as not ready. Without an epoch (0) the caller clears them.
    const uint32_t epoch = epochDevice ? (*epochDevice & 0x3FFFFFFFu) : 0u;
    if (tid == 0) sTile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = sTile;
    const uint32_t base = tile * kTileKeys;
    if (base >= n) return;   // a tile past the keys (the grid was sized for a bound): out before any work
#pragma unroll
    for (uint32_t j = tid; j < kCounters * kRadix / 4; j += kSortThreads) {
        reinterpret_cast<uint4*>(sWarpCnt)[j] = make_uint4(0, 0, 0, 0);
        reinterpret_cast<uint4*>(sMasks)[j] = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    const uint32_t ltMask = (1u << lane) - 1u;

    // Rank: warp `warp` owns keys [base + warp*32*kPerThread, +32*kPerThread), item k of
    // lane l being the (k*32 + l)-th; walking k then l is input order, so the
    // ranks are stable. A key's peers, the warp's keys of its digit, are the bits their lanes
    // set in the digit's mask: __match_any_sync takes some 240 cycles of an SM's quarter where
    // 32 digits differ, and was most of a pass; the masks take 35 there, 130 where all agree. (A
    // warp's ranking by masks of lanes is the warp-level multisplit of S. Ashkiani et al., "GPU
    // Multisplit", PPoPP 2016, which makes them by ballots.)
    const uint32_t mine = base + warp * 32 * kPerThread + lane;
    K key[kPerThread];
    uint32_t rank[kPerThread];
#pragma unroll
    for (uint32_t k = 0; k < kPerThread; ++k) key[k] = mine + k * 32 < n ? keysIn[mine + k * 32] : (K)(kDrop ? kCulledKey : 0u);
    auto takes = [&](uint32_t k) { return kDrop ? key[k] < (K)kCulledKey : mine + k * 32 < n; };
#pragma unroll
    for (uint32_t i = 0; i < kChainItems; ++i) {
        uint32_t at[kChains], peers[kChains], before[kChains];
        bool valid[kChains];
#pragma unroll
        for (uint32_t c = 0; c < kChains; ++c) {
            const uint32_t k = c * kChainItems + i;
            valid[c] = takes(k);
            at[c] = (warp * kChains + c) * kRadix + digitSlot((uint32_t)((key[k] >> shift) & digitMask));
            if (valid[c]) atomicOr(&sMasks[at[c]], 1u << lane);
        }
        __syncwarp();
#pragma unroll
        for (uint32_t c = 0; c < kChains; ++c) {
            peers[c] = valid[c] ? sMasks[at[c]] : 0u;
            before[c] = valid[c] ? sWarpCnt[at[c]] : 0u;
        }
        __syncwarp();
#pragma unroll
        for (uint32_t c = 0; c < kChains; ++c)
            if (valid[c] && (peers[c] & ltMask) == 0) {   // the digit's first lane
                sMasks[at[c]] = 0;
                sWarpCnt[at[c]] = before[c] + __popc(peers[c]);
            }
        __syncwarp();
#pragma unroll
        for (uint32_t c = 0; c < kChains; ++c) rank[c * kChainItems + i] = before[c] + __popc(peers[c] & ltMask);
    }
    __syncthreads();

    // One thread a digit (the first kRadix threads): the warps' counts to exclusive
    // offsets, the tile's count; every thread takes part in the block scans.
    const bool digit = tid < kRadix;
    const uint32_t t = digit ? tid : 0u;
    uint32_t count = 0;
    if (digit) {
#pragma unroll
        for (uint32_t w = 0; w < kCounters; ++w) {
            const uint32_t c = sWarpCnt[w * kRadix + digitSlot(t)];
            sWarpCnt[w * kRadix + digitSlot(t)] = count;
            count += c;
        }
    }
    // Where this tile's share of digit t starts in the output.
    uint64_t* flag = flags + (size_t)tile * kRadix + t;
    uint32_t exclusive = 0;
    const uint64_t tag = (uint64_t)epoch << 34;
    if (tile == 0) {
        exclusive = blockExclusiveScan(digit ? globalHist[t] : 0u, sScan);
        if (digit) storeRelaxed(flag, tag | (2ull << 32) | (uint64_t)(exclusive + count));
    } else if (digit) {
        storeRelaxed(flag, tag | (1ull << 32) | (uint64_t)count);
        uint64_t sum = 0;
        int64_t j = (int64_t)tile - 1;
        uint32_t spins = 0;
        while (j >= 0) {
            const uint64_t v = loadRelaxed(flags + (size_t)j * kRadix + t);
            const uint32_t st = (uint32_t)(v >> 34) == epoch ? (uint32_t)(v >> 32) & 3u : 0u;
            if (st == 0) {
                if (++spins > kSpinLimit || ((spins & 255u) == 0 && gaveUp(status))) {
                    atomicOr(status, kStatusLookbackTimeout);
                    break;
                }
                __nanosleep(32);
                continue;
            }
            sum += v & 0xFFFFFFFFull;
            if (st == 2) break;
            --j;
        }
        exclusive = (uint32_t)sum;
        storeRelaxed(flag, tag | (2ull << 32) | (uint64_t)(exclusive + count));
    }
    const uint32_t start = blockExclusiveScan(count, sScan);
    if (digit) {
        sStart[digitSlot(t)] = start;
        sAdjust[digitSlot(t)] = exclusive - start;
    }
    if (kDrop && tid == kRadix - 1) sKept = start + count;
    __syncthreads();

    // Scatter into shared memory in the tile's sorted order, then out.
    uint32_t place[kPerThread / 2];   // the items' places in that order, two a word (at most 8191)
#pragma unroll
    for (uint32_t k = 0; k < kPerThread; ++k) {
        uint32_t s = 0;
        if (takes(k)) {
            const uint32_t at = digitSlot((uint32_t)((key[k] >> shift) & digitMask));
            s = sStart[at] + sWarpCnt[(warp * kChains + k / kChainItems) * kRadix + at] + rank[k];
            sKeys[s] = key[k];
        }
        place[k / 2] = k & 1u ? place[k / 2] | (s << 16) : s;
    }
    __syncthreads();
    const uint32_t tileN = kDrop ? sKept : min(kTileKeys, n - base);
    uint32_t to[kValues == kNoValues ? 1 : kPerThread];
#pragma unroll
    for (uint32_t k = 0; k < kPerThread; ++k) {
        const uint32_t s = tid + k * kSortThreads;
        uint32_t dst = 0xFFFFFFFFu;
        if (s < tileN) {
            const K out = sKeys[s];
            dst = sAdjust[digitSlot((uint32_t)((out >> shift) & digitMask))] + s;
            if (dst < n) {
                if (keysOut) keysOut[dst] = out;
            } else {
                atomicOr(status, kStatusIndexRange);
                dst = 0xFFFFFFFFu;
            }
        }
        if constexpr (kValues != kNoValues) to[k] = dst;
    }
    if constexpr (kValues != kNoValues) {
        uint32_t val[kPerThread];
#pragma unroll
        for (uint32_t k = 0; k < kPerThread; ++k)
            val[k] = kValues == kIndexValues ? mine + k * 32 : mine + k * 32 < n ? valsIn[mine + k * 32] : 0u;
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kPerThread; ++k)
            if (takes(k)) sVals[(place[k / 2] >> (16 * (k & 1u))) & 0xFFFFu] = val[k];
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kPerThread; ++k)
            if (to[k] != 0xFFFFFFFFu) valsOut[to[k]] = sVals[tid + k * kSortThreads];
    }
}

// A whole sort of at most kSortTileKeys keys in one block: the passes of `plan` one after
// another, the keys (and values) carried in registers and reordered through shared memory.
// A small sort's passes are latency alone, each some 6 us as a kernel; in one block they
// need no histograms, look-back, tickets or clearing either. A frame of 5k splats: 144 -> 140 us
// (128 now: the masks below, and SortPlan). Every key is read before the first is written, so the
// output may be the input.
template <typename K, uint32_t kValues>
__host__ __device__ constexpr size_t smallKeysSmem() { return kSortTileKeys * (sizeof(K) + (kValues == kNoValues ? 0 : 4)); }
template <typename K, uint32_t kValues>
__global__ void __launch_bounds__(kSortThreads)
    smallSortKernel(const K* keysIn, const uint32_t* valsIn, K* keysOut, uint32_t* valsOut, uint32_t n,
                    const uint32_t* __restrict__ nDevice, uint32_t firstBit, const SortPlan plan) {
    extern __shared__ __align__(16) unsigned char smem[];
    static_assert(smallKeysSmem<K, kValues>() >= (size_t)kWarps * kMaxRadix * 4, "the masks take the keys' place");
    K* sKeys = reinterpret_cast<K*>(smem);
    uint32_t* sVals = reinterpret_cast<uint32_t*>(sKeys + kSortTileKeys);
    uint32_t* sMasks = reinterpret_cast<uint32_t*>(smem);   // kWarps x kMaxRadix at most, while the keys are ranked
    uint32_t* sWarpCnt = reinterpret_cast<uint32_t*>(smem + smallKeysSmem<K, kValues>());   // kWarps x kMaxRadix at most
    __shared__ uint32_t sStart[kMaxRadix];
    __shared__ uint32_t sScan[kWarps];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    n = min(countOf(n, nDevice), kSortTileKeys);
    // only the warps that hold keys rank them; item k of lane l is key mine + 32 k
    const uint32_t perThread = (n + kSortThreads - 1) / kSortThreads;
    const uint32_t mine = warp * 32 * perThread + lane;
    K key[kItems];
    uint32_t val[kValues == kNoValues ? 1 : kItems];
    uint32_t rank[kItems];
#pragma unroll
    for (uint32_t k = 0; k < kItems; ++k) {
        const uint32_t i = mine + k * 32;
        const bool valid = k < perThread && i < n;
        key[k] = valid ? keysIn[i] : (K)0;
        if (kValues == kIndexValues && key[k] >= (K)kCulledKey) key[k] = (K)((1u << kDepthBits) - 1u);   // past any depth: last
        if constexpr (kValues == kReadValues) val[k] = valid ? valsIn[i] : 0u;
        if constexpr (kValues == kIndexValues) val[k] = i;
    }
    for (uint32_t p = 0; p < plan.passes; ++p) {
        const uint32_t radix = 1u << plan.width(p), digitMask = plan.mask(p), shift = firstBit + plan.shift(p);
        for (uint32_t j = tid; j < kWarps * radix / 4; j += kSortThreads) {
            reinterpret_cast<uint4*>(sWarpCnt)[j] = make_uint4(0, 0, 0, 0);
            reinterpret_cast<uint4*>(sMasks)[j] = make_uint4(0, 0, 0, 0);
        }
        __syncthreads();
        uint32_t *counts = sWarpCnt + warp * radix, *masks = sMasks + warp * radix;
#pragma unroll
        for (uint32_t k = 0; k < kItems; ++k) {
            if (k >= perThread) break;
            const bool valid = mine + k * 32 < n;
            const uint32_t at = digitSlot((uint32_t)((key[k] >> shift) & digitMask));
            if (valid) atomicOr(&masks[at], 1u << lane);
            __syncwarp();
            const uint32_t peers = valid ? masks[at] : 0u, before = valid ? counts[at] : 0u;
            const uint32_t lower = peers & ((1u << lane) - 1u);
            __syncwarp();
            if (valid && lower == 0) {   // the digit's first lane
                masks[at] = 0;
                counts[at] = before + __popc(peers);
            }
            __syncwarp();
            rank[k] = before + __popc(lower);
        }
        __syncthreads();
        uint32_t count = 0;
        if (tid < radix) {
#pragma unroll
            for (uint32_t w = 0; w < kWarps; ++w) {
                uint32_t& at = sWarpCnt[w * radix + digitSlot(tid)];
                const uint32_t c = at;
                at = count;
                count += c;
            }
        }
        const uint32_t start = blockExclusiveScan(count, sScan);
        if (tid < radix) sStart[digitSlot(tid)] = start;
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kItems; ++k) {
            if (k >= perThread) break;
            if (mine + k * 32 < n) {
                const uint32_t at = digitSlot((uint32_t)((key[k] >> shift) & digitMask));
                const uint32_t s = sStart[at] + counts[at] + rank[k];
                sKeys[s] = key[k];
                if constexpr (kValues != kNoValues) sVals[s] = val[k];
            }
        }
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kItems; ++k) {
            if (k >= perThread) break;
            const uint32_t i = mine + k * 32;
            if (i < n) {
                key[k] = sKeys[i];
                if constexpr (kValues != kNoValues) val[k] = sVals[i];
            }
        }
        __syncthreads();   // the next pass clears its masks over the keys
    }
#pragma unroll
    for (uint32_t k = 0; k < kItems; ++k) {
        if (k >= perThread) break;
        const uint32_t i = mine + k * 32;
        if (i < n) {
            if (keysOut) keysOut[i] = key[k];
            if constexpr (kValues != kNoValues) valsOut[i] = val[k];
        }
    }
}
template <typename K, uint32_t kValues>
constexpr size_t smallSortSmem() {
    return smallKeysSmem<K, kValues>() + (size_t)kWarps * kMaxRadix * 4;
}

template <typename K, uint32_t kValues, uint32_t kBits, uint32_t kPerThread>
cudaError_t allowSmem() {
    return cudaFuncSetAttribute(onesweepKernel<K, kValues, kBits, kPerThread>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)onesweepSmem<K, kBits, kPerThread>());
}
// what a block takes without asking, its static arrays included
static_assert(onesweepSmem<uint64_t, 8, kSmallItems>() <= 44 * 1024, "small tiles of eight bits ask for no more");
template <typename K, uint32_t kValues>
cudaError_t allowSmallSmem() {
    return cudaFuncSetAttribute(smallSortKernel<K, kValues>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smallSortSmem<K, kValues>());
}

// The passes of a sort of `bits` bits: eight bits a pass, or, where that takes a
// pass fewer, nine bits in as many passes as needed and eight in the rest
// (34 bits: 9 + 9 + 8 + 8 in four passes, not five).
SortPlan planSort(uint32_t bits) {
    const uint32_t eights = (bits + 7) / 8, nines = (bits + 8) / 9;
    SortPlan p{nines < eights ? nines : eights, bits, 0};
    if (nines < eights && bits > 8 * p.passes) p.wide = bits - 8 * p.passes;
    return p;
}

}   // namespace

uint32_t sortPasses(uint32_t bits) { return planSort(bits).passes; }
// Small tiles up to the count at which 2048-key tiles fill two blocks on every SM.
constexpr uint32_t kSmallTile = kSortThreads * kSmallItems, kSmallSort = 2u * 148u * kSmallTile;
uint32_t sortTileKeys(uint32_t n, bool pairs) {
    return n <= kSmallSort ? kSmallTile : pairs ? kSortThreads * kPairItems : kSortTileKeys;
}
size_t sortFlagWords(uint32_t n, uint32_t bits, bool pairs, uint32_t tileKeys) {
    const SortPlan p = planSort(bits);
    auto words = [&](uint32_t count, uint32_t keys) {
        size_t w = 0;
        for (uint32_t k = 0; k < p.passes; ++k) w += (size_t)((count + keys - 1) / keys) << p.width(k);
        return w;
    };
    if (tileKeys) return words(n, tileKeys);
    // room for any sort of at most n keys: a smaller one may take the small tiles
    const size_t most = words(n, sortTileKeys(n, pairs));
    return n > kSmallSort ? max(most, words(kSmallSort, kSmallTile)) : most;
}

// Each some 6 us: an owner asks for the sorts it runs.
cudaError_t sortPrepare(uint32_t uses) {
    cudaError_t err = cudaSuccess;
    auto also = [&](cudaError_t (*allow)()) { if (err == cudaSuccess) err = allow(); };
    if (uses & kSortsKeys) {
        also(allowSmem<uint64_t, kNoValues, 8, kItems>);
        also(allowSmem<uint64_t, kNoValues, 9, kItems>);
        also(allowSmem<uint64_t, kNoValues, 9, kSmallItems>);
        also(allowSmallSmem<uint64_t, kNoValues>);
    }
    if (uses & kSortsPairs) {
        also(allowSmem<uint64_t, kReadValues, 8, kItems>);
        also(allowSmem<uint64_t, kReadValues, 9, kItems>);
        also(allowSmem<uint64_t, kReadValues, 8, kPairItems>);
        also(allowSmem<uint64_t, kReadValues, 9, kPairItems>);
        also(allowSmem<uint64_t, kReadValues, 9, kSmallItems>);
        also(allowSmallSmem<uint64_t, kReadValues>);
    }
    if (uses & kSortsDepths) {
        also(allowSmem<uint32_t, kIndexValues, 8, kItems>);
        also(allowSmem<uint32_t, kReadValues, 8, kItems>);
        also(allowSmallSmem<uint32_t, kIndexValues>);
    }
    return err;
}

namespace {

template <typename K, uint32_t kValues, uint32_t kBits>
void launchPass(uint32_t tileKeys, uint32_t tiles, const K* keysIn, const uint32_t* valsIn, K* keysOut,
                uint32_t* valsOut, uint32_t n, uint32_t shift, const uint32_t* hist, uint64_t* flags, uint32_t* ticket,
                uint32_t* status, const uint32_t* nDevice, const uint32_t* epochDevice, uint32_t digitMask,
                cudaStream_t stream) {
#define ATH_TILE(I_)                                                                                                 \
    onesweepKernel<K, kValues, kBits, I_><<<tiles, kSortThreads, onesweepSmem<K, kBits, I_>(), stream>>>(            \
        keysIn, valsIn, keysOut, valsOut, n, shift, digitMask, hist, flags, ticket, status, nDevice, epochDevice)
    if constexpr (sizeof(K) == 8 && kValues != kNoValues)
        if (tileKeys == kSortThreads * kPairItems) return (void)(ATH_TILE(kPairItems));
    if (tileKeys == kSortTileKeys) ATH_TILE(kItems);
    else ATH_TILE(kSmallItems);
#undef ATH_TILE
}

// What the sorts share: the clearing, the digit histograms of `in`, then `pass` for each pass.
template <typename K, typename Pass>
cudaError_t runSort(uint32_t n, const uint32_t* nDevice, const uint32_t* epochDevice, uint32_t firstBit, uint32_t bits,
                    uint32_t tileKeys, SortClear clear, uint32_t* hist, uint64_t* flags, uint32_t* tickets,
                    cudaStream_t stream, const K* in, bool pairs, Pass pass) {
    const SortPlan plan = planSort(bits);
    if (plan.passes > kMaxPasses || firstBit + bits > 8 * sizeof(K)) return cudaErrorInvalidValue;
    const uint32_t keys = tileKeys ? tileKeys : sortTileKeys(n, pairs);
    const uint32_t tiles = (n + keys - 1) / keys;
    cudaError_t err = cudaSuccess;
    if (clear != kClearNone) err = cudaMemsetAsync(hist, 0, sizeof(uint32_t) * kMaxRadix * plan.passes, stream);
    if (err == cudaSuccess && clear == kClearAll) {
        err = cudaMemsetAsync(flags, 0, sizeof(uint64_t) * sortFlagWords(n, bits, pairs, keys), stream);
        if (err == cudaSuccess) err = cudaMemsetAsync(tickets, 0, sizeof(uint32_t) * plan.passes, stream);
    }
    if (err != cudaSuccess) return err;
    int device = 0, sms = 148;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    histogramKernel<K><<<min((n + 255) / 256, (uint32_t)sms * 4), 256, 0, stream>>>(in, n, nDevice, firstBit, plan, hist);
    for (uint32_t p = 0; p < plan.passes; ++p) {
        pass(p, plan, keys, tiles, firstBit + plan.shift(p), hist + p * kMaxRadix, flags, tickets + p,
             plan.mask(p));
        flags += (size_t)tiles << plan.width(p);
    }
    return cudaGetLastError();
}

}   // namespace

// keys/vals[0] hold the input; the sorted result lands in keys/vals[sortResultIndex(n, bits)]
// (n as given here, also where nDevice holds the count). vals may be null (keys only). The passes
// sort bits [firstBit, firstBit + bits) of the keys, eight or nine at a time
// (planSort). hist: kMaxPasses * kMaxRadix words, flags: sortFlagWords
// words, tickets: one word a pass; all three start at zero (`clear`: what of them is
// zeroed here). tileKeys: kSortTileKeys for callers whose flags hold no more than that
// takes; 0 by the count.
cudaError_t launchSortDevice(uint64_t* keys[2], uint32_t* vals[2], uint32_t n, const uint32_t* nDevice,
                             const uint32_t* epochDevice, uint32_t firstBit, uint32_t bits, uint32_t* hist,
                             uint64_t* flags, uint32_t* tickets, uint32_t* status, cudaStream_t stream,
                             SortClear clear, uint32_t tileKeys) {
    if (n <= 1 && !nDevice) return cudaSuccess;
    const bool withValues = vals != nullptr && vals[0] != nullptr;
    if (n <= kSortTileKeys) {   // one block, in place
        if (firstBit + bits > 64) return cudaErrorInvalidValue;
        const SortPlan plan = planSort(bits);
        if (withValues)
            smallSortKernel<uint64_t, kReadValues><<<1, kSortThreads, smallSortSmem<uint64_t, kReadValues>(), stream>>>(
                keys[0], vals[0], keys[0], vals[0], n, nDevice, firstBit, plan);
        else
            smallSortKernel<uint64_t, kNoValues><<<1, kSortThreads, smallSortSmem<uint64_t, kNoValues>(), stream>>>(
                keys[0], nullptr, keys[0], nullptr, n, nDevice, firstBit, plan);
        return cudaGetLastError();
    }
    auto pass = [&](uint32_t p, const SortPlan& plan, uint32_t tileKeysHere, uint32_t tiles, uint32_t shift,
                    const uint32_t* h, uint64_t* f, uint32_t* ticket, uint32_t mask) {
        const uint32_t in = p & 1u, out = in ^ 1u;
        const uint32_t* vi = withValues ? vals[in] : nullptr;
        uint32_t* vo = withValues ? vals[out] : nullptr;
#define ATH_PASS(V_, W_)                                                                                            \
    launchPass<uint64_t, V_, W_>(tileKeysHere, tiles, keys[in], vi, keys[out], vo, n, shift, h, f, ticket, status, \
                                 nDevice, epochDevice, mask, stream)
        if (withValues && plan.width(p) == 9) ATH_PASS(kReadValues, 9);
        else if (withValues) ATH_PASS(kReadValues, 8);
        else if (plan.width(p) == 9) ATH_PASS(kNoValues, 9);
        else ATH_PASS(kNoValues, 8);
#undef ATH_PASS
    };
    return runSort<uint64_t>(n, nDevice, epochDevice, firstBit, bits, tileKeys, clear, hist, flags, tickets, stream, keys[0],
                             withValues, pass);
}

cudaError_t launchSort(uint64_t* keys[2], uint32_t* vals[2], uint32_t n, uint32_t bits, uint32_t* hist,
                       uint64_t* flags, uint32_t* tickets, uint32_t* status, cudaStream_t stream, SortClear clear,
                       uint32_t tileKeys) {
    return launchSortDevice(keys, vals, n, nullptr, nullptr, 0, bits, hist, flags, tickets, status, stream, clear, tileKeys);
}

cudaError_t launchSortDepths(const uint32_t* keys, uint32_t* sortKeys[2], uint32_t* slots[2], uint32_t n,
                             const uint32_t* visible, uint32_t* hist, uint64_t* flags, uint32_t* tickets, uint32_t* status,
                             cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    if (n <= kSortTileKeys) {
        smallSortKernel<uint32_t, kIndexValues><<<1, kSortThreads, smallSortSmem<uint32_t, kIndexValues>(), stream>>>(
            keys, nullptr, nullptr, slots[0], n, nullptr, 0, planSort(kDepthBits));
        return cudaGetLastError();
    }
    // three 8-bit passes: keys -> [0] -> [1] -> [0], the first carrying its keys' places and leaving
    // the culled ones out, the last writing the slots alone
    auto pass = [&](uint32_t p, const SortPlan& plan, uint32_t tileKeys, uint32_t tiles, uint32_t shift, const uint32_t* h,
                    uint64_t* f, uint32_t* ticket, uint32_t mask) {
        const uint32_t out = p & 1u, in = out ^ 1u;
        uint32_t* ko = p + 1 == plan.passes ? nullptr : sortKeys[out];
        if (p == 0)
            launchPass<uint32_t, kIndexValues, 8>(tileKeys, tiles, keys, nullptr, ko, slots[out], n, shift, h, f, ticket,
                                                  status, nullptr, nullptr, mask, stream);
        else
            launchPass<uint32_t, kReadValues, 8>(tileKeys, tiles, sortKeys[in], slots[in], ko, slots[out], n, shift, h, f,
                                                 ticket, status, visible, nullptr, mask, stream);
    };
    static_assert(kDepthBits == 24, "three 8-bit passes");
    return runSort<uint32_t>(n, nullptr, nullptr, 0, kDepthBits, 0, kClearNone, hist, flags, tickets, stream, keys, false, pass);
}

uint32_t sortResultIndex(uint32_t n, uint32_t bits) { return n <= kSortTileKeys ? 0u : (sortPasses(bits) & 1u); }
uint32_t sortHistWords() { return kMaxPasses * kMaxRadix; }

}   // namespace ath
