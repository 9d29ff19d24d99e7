// Onesweep LSD radix sort of 32-bit keys with 8-bit digits: stable and ascending, the
// contract of splatkit-ios/.../metal/sort/MetalRadixSort.h:13-19 (an argsort whose first pass
// takes each key's position as its value; the last pass skips the key write unless asked).
//
// The reference runs histogram -> scan -> scatter per pass (SplatRadixSort.metal:17-171). Here:
//   1. one upfront pass reads every key once and builds all digit histograms; the block that
//      finishes last turns them into exclusive digit bases;
//   2. one scatter pass per digit. Each tile (2048, 4096 or 6144 keys, 4096 by default) ranks
//      its keys per warp with ballot matching (8 ballots per row, rows in source order, so
//      ranking is stable), publishes its per-digit counts, stages keys and values in digit order in
//      shared memory, learns how many keys of each digit the tiles before it hold by decoupled
//      look-back (bounded waits, four predecessors at a time) and writes each digit run contiguously.
//      A large sort's pass is bound by its instructions (about 120 per 32 keys): 40M keys, 4 passes
//      340 -> 240 us each with one staging round instead of two, no bounds tests between the loads and
//      the writes, and the wider look-back; HBM's share is 98 us. A pass of up to 1.2M keys is one
//      tile's latency: a million keys 22 -> 13 us.
// Tiles are handed out by an atomic counter, so a tile only waits on tiles already running.
#include <cuda_runtime.h>

#include "sk_device.cuh"
#include "sk_kernels.h"
#include "sk_launch.cuh"

namespace sk {
namespace {

constexpr uint32_t kThreads = 256;
constexpr uint32_t kWarps = kThreads / 32;
constexpr uint32_t kTileKeys = 4096;  // keys per scatter tile unless asked otherwise
constexpr uint32_t kBins = 256;
constexpr uint32_t kMaxPasses = 4;

__device__ __forceinline__ uint32_t clampCount(const uint32_t* count, uint32_t capacity) {
  return min(*count, capacity);
}

// ---- 1. all-digit histogram ------------------------------------------------------------
__global__ void __launch_bounds__(kThreads)
    histogramKernel(const uint32_t* __restrict__ keys, const uint32_t* count, uint32_t capacity,
                    uint32_t passes, uint32_t* accum, uint32_t* bases, uint32_t* counters) {
  chainedKernelStart();
  __shared__ uint32_t h[kMaxPasses][kBins];
  for (uint32_t i = threadIdx.x; i < kMaxPasses * kBins; i += kThreads) (&h[0][0])[i] = 0;
  __syncthreads();
  const uint32_t n = clampCount(count, capacity);
  const uint32_t stride = gridDim.x * kThreads * 4;  // keys per grid step of one uint4 per thread
  // four 16-byte loads in flight per thread, then their 16 keys counted
  for (uint32_t base = (blockIdx.x * kThreads + threadIdx.x) * 4; base < n; base += stride * 4) {
    uint4 v[4];
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      const uint32_t i = base + q * stride;
      if (i + 3 < n) {
        v[q] = __ldg(reinterpret_cast<const uint4*>(keys + i));
      } else {
        v[q].x = i < n ? keys[i] : 0u;
        v[q].y = i + 1 < n ? keys[i + 1] : 0u;
        v[q].z = i + 2 < n ? keys[i + 2] : 0u;
        v[q].w = i + 3 < n ? keys[i + 3] : 0u;
      }
    }
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      const uint32_t i = base + q * stride;
      const uint32_t k[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
      for (uint32_t j = 0; j < 4; ++j) {
        if (i + j >= n) break;
        for (uint32_t p = 0; p < passes; ++p) atomicAdd(&h[p][(k[j] >> (8 * p)) & 0xffu], 1u);
      }
    }
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < passes * kBins; i += kThreads) {
    const uint32_t v = (&h[0][0])[i];
    if (v) atomicAdd(&accum[i], v);
  }
  if (finishTile(counters)) finishDigitHistograms(accum, bases, passes);
}

// ---- 2. onesweep scatter ----------------------------------------------------------------
// Lanes of this warp whose digit equals this lane's: 8 ballots.
__device__ __forceinline__ uint32_t matchDigit(uint32_t digit) {
  uint32_t peers = 0xffffffffu;
#pragma unroll
  for (uint32_t b = 0; b < 8; ++b) {
    const bool bit = (digit >> b) & 1u;
    const uint32_t vote = __ballot_sync(0xffffffffu, bit);
    peers &= bit ? vote : ~vote;
  }
  return peers;
}

// A scatter block has one group of 256 threads (a thread per digit), or two.
template <uint32_t kGroups>
struct ScatterSmem {
  uint32_t warpCount[kGroups * kWarps][kBins];  // per warp and digit: its keys, then their first place
  uint32_t groupTotal[kGroups][kBins];
  uint32_t shift[kBins];  // a key's place in the output less its place in the tile
  uint32_t warpSums[kGroups * kWarps];
};

// Predecessors whose status words a look-back step reads at once. With one at a time the 245 tiles of a
// million keys, all resident together, walked back over one another's counts for 9 us of a 20 us pass.
constexpr uint32_t kLookbackWindow = 4;

// Keys of digit d in the tiles before `tile`, by decoupled look-back.
__device__ __forceinline__ uint32_t digitLookback(const uint64_t* status, uint32_t tile, uint32_t epoch,
                                                  uint32_t d, uint32_t* error) {
  uint32_t exclusive = 0;
  for (int j = static_cast<int>(tile) - 1; j >= 0; j -= static_cast<int>(kLookbackWindow)) {
    uint64_t w[kLookbackWindow];
#pragma unroll
    for (int k = 0; k < static_cast<int>(kLookbackWindow); ++k)
      w[k] = j >= k ? loadStatus(status + static_cast<size_t>(j - k) * kBins + d) : 0u;
#pragma unroll
    for (int k = 0; k < static_cast<int>(kLookbackWindow); ++k) {
      if (j < k) return exclusive;
      const bool ready = static_cast<uint32_t>(w[k] >> 34) == (epoch & 0x3fffffffu) && ((w[k] >> 32) & 3u) != 0u;
      if (!ready) w[k] = waitStatus(status + static_cast<size_t>(j - k) * kBins + d, epoch, error);
      exclusive += static_cast<uint32_t>(w[k]);
      if (((w[k] >> 32) & 3u) == kFlagPrefix) return exclusive;
    }
  }
  return exclusive;
}

struct ScatterArgs {
  const uint32_t* keysIn;
  const uint32_t* valuesIn;
  uint32_t* keysOut;
  uint32_t* valuesOut;
  const uint32_t* count;
  uint32_t capacity, shift;
  const uint32_t* digitBase;
  uint64_t* status;
  uint32_t* counters;
  uint32_t epoch;
  uint32_t* error;
  uint32_t withheldPlusOne;
};

// One tile of 256 * kGroups * kPer keys. The keys a last tile lacks are taken as all ones: they rank behind every
// key that is there (digit 255, last in source order), so only the loads and the writes test bounds.
template <bool kImplicitValues, bool kWriteKeys, uint32_t kGroups, uint32_t kPer>
__device__ __forceinline__ void scatterTile(const ScatterArgs& a, ScatterSmem<kGroups>& s, uint32_t* stageKey,
                                            uint32_t* stageValue, uint32_t tile, uint32_t n) {
  constexpr uint32_t kBlock = kThreads * kGroups, kTile = kBlock * kPer;
  const uint32_t warp = threadIdx.x >> 5, lane = laneId();
  const uint32_t d = threadIdx.x % kBins, group = threadIdx.x / kBins;  // the digit this thread sums
  const uint32_t first = tile * kTile + warp * (32 * kPer) + lane;
  uint32_t key[kPer];
#pragma unroll
  for (uint32_t r = 0; r < kPer; ++r) {
    const uint32_t e = first + r * 32;
    key[r] = e < n ? a.keysIn[e] : 0xffffffffu;
  }
  const uint32_t base = __ldg(a.digitBase + d);
  // Rank each key among the equal digits of its warp, row by row (source order).
  uint32_t rank[kPer];
  const uint32_t below = lanemaskLt();
#pragma unroll
  for (uint32_t r = 0; r < kPer; ++r) {
    const uint32_t digit = (key[r] >> a.shift) & 0xffu;
    const uint32_t peers = matchDigit(digit);
    const uint32_t before = s.warpCount[warp][digit];
    __syncwarp();
    if ((peers & below) == 0u) s.warpCount[warp][digit] = before + __popc(peers);
    __syncwarp();
    rank[r] = before + __popc(peers & below);
  }
  __syncthreads();
  // Per digit: the tile's total, published for the tiles after it. A tile named by the test hook
  // (withheldPlusOne = tile + 1; 0 names none) publishes nothing, so its successors' bounded
  // waits run out.
  uint32_t counts[kWarps], total = 0, lower = 0;
#pragma unroll
  for (uint32_t w = 0; w < kWarps; ++w) {
    counts[w] = s.warpCount[group * kWarps + w][d];
    total += counts[w];
  }
  if constexpr (kGroups > 1) {
    s.groupTotal[group][d] = total;
    __syncthreads();
    total = 0;
#pragma unroll
    for (uint32_t g = 0; g < kGroups; ++g) {
      const uint32_t t = s.groupTotal[g][d];
      if (g < group) lower += t;
      total += t;
    }
  }
  uint64_t* mine = a.status + static_cast<size_t>(tile) * kBins + d;
  const bool publish = group == 0 && tile + 1u != a.withheldPlusOne;
  if (publish) storeStatus(mine, makeStatus(a.epoch, tile == 0 ? kFlagPrefix : kFlagAggregate, total));
  // Exclusive scan of the totals: where each digit's run starts in the tile, and each warp's part of
  // it (every group scans for itself).
  uint32_t inc = total;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t up = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= static_cast<uint32_t>(o)) inc += up;
  }
  if (lane == 31) s.warpSums[warp] = inc;
  __syncthreads();
  uint32_t localOffset = inc - total;
#pragma unroll
  for (uint32_t w = 0; w < kWarps; ++w) localOffset += w < warp % kWarps ? s.warpSums[group * kWarps + w] : 0u;
  uint32_t run = localOffset + lower;
#pragma unroll
  for (uint32_t w = 0; w < kWarps; ++w) {
    s.warpCount[group * kWarps + w][d] = run;
    run += counts[w];
  }
  __syncthreads();
  // keys, then values, staged in digit order (a value's loads start when the key's register is free)
#pragma unroll
  for (uint32_t r = 0; r < kPer; ++r) {
    rank[r] += s.warpCount[warp][(key[r] >> a.shift) & 0xffu];
    stageKey[rank[r]] = key[r];
  }
#pragma unroll
  for (uint32_t r = 0; r < kPer; ++r) {
    const uint32_t e = first + r * 32;
    key[r] = kImplicitValues ? e : (e < n ? a.valuesIn[e] : 0u);
  }
#pragma unroll
  for (uint32_t r = 0; r < kPer; ++r) stageValue[rank[r]] = key[r];
  if (group == 0) {
    uint32_t exclusive = 0;
    if (tile != 0) {
      exclusive = digitLookback(a.status, tile, a.epoch, d, a.error);
      if (publish) storeStatus(mine, makeStatus(a.epoch, kFlagPrefix, exclusive + total));
    }
    s.shift[d] = base + exclusive - localOffset;
  }
  __syncthreads();
  const uint32_t inTile = min(kTile, n - tile * kTile);
#pragma unroll
  for (uint32_t r = 0; r < kPer; ++r) {
    const uint32_t i = threadIdx.x + r * kBlock;
    if (i < inTile) {
      const uint32_t k = stageKey[i];
      const uint32_t at = i + s.shift[(k >> a.shift) & 0xffu];
      // Only a look-back that gave up can put `at` past the end; never write there.
      if (at < n) {
        if (kWriteKeys) a.keysOut[at] = k;
        a.valuesOut[at] = stageValue[i];
      } else {
        atomicOr(a.error, SK_DEVERR_BOUNDS);
      }
    }
  }
}

template <bool kImplicitValues, bool kWriteKeys, uint32_t kGroups, uint32_t kPer>
__global__ void __launch_bounds__(kThreads* kGroups, kGroups * kPer > 16 ? 2 : 4 / kGroups)
    scatterKernel(const __grid_constant__ ScatterArgs a) {
  constexpr uint32_t kBlock = kThreads * kGroups, kTile = kBlock * kPer;
  __shared__ ScatterSmem<kGroups> s;
  extern __shared__ uint32_t stage[];
  // The tile and the cleared counts come before the wait for the kernel before this one: the tile
  // counter is this launch's alone (its last block left it at zero in an earlier, finished launch).
  for (uint32_t i = threadIdx.x; i < kGroups * kWarps * kBins; i += kBlock) (&s.warpCount[0][0])[i] = 0;
  const uint32_t tile = takeTile(a.counters);
  chainedKernelStart();
  const uint32_t n = clampCount(a.count, a.capacity);
  const uint32_t tiles = (n + kTile - 1) / kTile;
  if (tile < tiles) scatterTile<kImplicitValues, kWriteKeys, kGroups, kPer>(a, s, stage, stage + kTile, tile, n);
  finishTile(a.counters);
}

template <bool kImplicitValues, bool kWriteKeys, uint32_t kGroups, uint32_t kPer>
cudaError_t launchScatter(const ScatterArgs& a, uint32_t tiles, cudaStream_t stream) {
  constexpr size_t kBytes = size_t{2} * kThreads * kGroups * kPer * 4;  // staged keys and values
  constexpr auto kernel = scatterKernel<kImplicitValues, kWriteKeys, kGroups, kPer>;
  if constexpr (kBytes + sizeof(ScatterSmem<kGroups>) > 48 * 1024) {
    static std::atomic<uint64_t> done{0};
    const cudaError_t e = oncePerDevice(done, [&] {
      return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kBytes));
    });
    if (e != cudaSuccess) return e;
  }
  return launchChainedShared(kernel, tiles, kThreads * kGroups, kBytes, stream, a);
}

inline size_t alignUp(size_t v, size_t a) { return (v + a - 1) / a * a; }

}  // namespace

uint32_t sortTileKeys() { return kTileKeys; }

uint32_t* sortDigitAccumulators(const SortArgs& a) { return a.histogram; }
uint32_t* sortDigitBases(const SortArgs& a) { return a.histogram + kMaxPasses * kBins; }

static uint32_t sortTiles(uint32_t capacity, uint32_t tileKeys = kTileKeys) {
  return max(1u, (capacity + tileKeys - 1) / tileKeys);
}

static uint32_t tileKeysOf(const SortArgs& a) { return a.tileKeys ? a.tileKeys : kTileKeys; }

constexpr size_t kCounterBytes = 256;
static_assert((kMaxPasses + 1) * 2 * 4 <= kCounterBytes, "two words per pass and for the histogram");

size_t sortWorkspaceBytesFor(uint32_t capacity, uint32_t minTileKeys) {
  const size_t n = alignUp(static_cast<size_t>(max(capacity, 1u)) * 4, 256);
  return 3 * n                                             // keysA, keysB, valuesTmp
         + alignUp(2 * kMaxPasses * kBins * 4, 256)        // histogram accumulators + bases
         + kCounterBytes
         + alignUp(static_cast<size_t>(sortTiles(capacity, minTileKeys)) * kBins * 8, 256);  // status
}

size_t sortWorkspaceBytes(uint32_t capacity) { return sortWorkspaceBytesFor(capacity, kTileKeys); }

void sortBindWorkspaceFor(SortArgs& a, void* workspace, uint32_t capacity, uint32_t minTileKeys) {
  char* p = static_cast<char*>(workspace);
  const size_t n = alignUp(static_cast<size_t>(max(capacity, 1u)) * 4, 256);
  a.keysA = reinterpret_cast<uint32_t*>(p), p += n;
  a.keysB = reinterpret_cast<uint32_t*>(p), p += n;
  a.valuesTmp = reinterpret_cast<uint32_t*>(p), p += n;
  a.histogram = reinterpret_cast<uint32_t*>(p), p += alignUp(2 * kMaxPasses * kBins * 4, 256);
  a.counters = reinterpret_cast<uint32_t*>(p), p += kCounterBytes;
  a.status = reinterpret_cast<uint64_t*>(p);
  a.statusTiles = sortTiles(capacity, minTileKeys);
}

void sortBindWorkspace(SortArgs& a, void* workspace, uint32_t capacity) {
  sortBindWorkspaceFor(a, workspace, capacity, kTileKeys);
}

cudaError_t sortResetWorkspace(const SortArgs& a, cudaStream_t stream) {
  // the counters follow the histogram: one clear (1M 16-bit keys, whole call: 36.9 us, 39.1 with two)
  char* first = reinterpret_cast<char*>(a.histogram);
  return cudaMemsetAsync(first, 0, reinterpret_cast<char*>(a.counters) + kCounterBytes - first, stream);
}

cudaError_t launchSort(const SortArgs& a, cudaStream_t stream) {
  const uint32_t passes = static_cast<uint32_t>(min(max(a.bits, 8), 32) + 7) / 8u;
  if (sortInOneLaunch(a.capacity) && a.withheldTilePlusOne == 0) return launchClusterSort(a, passes, stream);
  const uint32_t tileKeys = tileKeysOf(a);
  if (tileKeys != 2048 && tileKeys != 4096 && tileKeys != 6144) return cudaErrorInvalidValue;
  const uint32_t tiles = sortTiles(a.capacity, tileKeys);
  if (tiles > a.statusTiles) return cudaErrorInvalidValue;  // the workspace was bound for larger tiles
  // 4096-key tiles: while all of them fit the chip at once (two 512-thread blocks per SM) a pass lasts as
  // long as one tile, which twice the threads finish sooner (1M 16-bit keys: 26 us for two passes against
  // 31); beyond that a pass is bound by instructions, and 16 keys per thread take fewer of them per key
  // (40M 32-bit keys: 957 us for four passes against 1294).
  const bool oneWave = tiles <= 2 * 148;
  uint32_t* accum = a.histogram;
  uint32_t* bases = a.histogram + kMaxPasses * kBins;
  cudaError_t e = cudaSuccess;
  if (!a.basesReady) {
    const uint32_t histBlocks = min(sortTiles(a.capacity), 148u * 4u);
    e = launchChained(histogramKernel, histBlocks, kThreads, stream, a.keysIn, a.count, a.capacity,
                      passes, accum, bases, a.counters);
    if (e != cudaSuccess) return e;
  }
  const uint32_t* kin = a.keysIn;
  const uint32_t* vin = a.valuesIn;
  for (uint32_t p = 0; p < passes; ++p) {
    const bool last = p + 1 == passes;
    uint32_t* kout = last ? a.keysOut : (p % 2 == 0 ? a.keysA : a.keysB);
    uint32_t* vout = ((passes - 1 - p) % 2 == 0) ? a.valuesOut : a.valuesTmp;
    uint32_t* counters = a.counters + 2 * (p + 1);
    const uint32_t epoch = (a.epoch + p) & 0x3fffffffu;
    const bool implicit = p == 0 && vin == nullptr;
    const bool writeKeys = kout != nullptr;
    const ScatterArgs sa{kin, vin, kout, vout, a.count, a.capacity, 8 * p, bases + p * kBins, a.status,
                         counters, epoch, a.error, p == 0 ? a.withheldTilePlusOne : 0u};
#define SK_SCATTER(IMPLICIT, WRITE)                                                        \
  e = tileKeys == 2048   ? launchScatter<IMPLICIT, WRITE, 1u, 8u>(sa, tiles, stream)       \
      : tileKeys == 6144 ? launchScatter<IMPLICIT, WRITE, 1u, 24u>(sa, tiles, stream)      \
      : oneWave          ? launchScatter<IMPLICIT, WRITE, 2u, 8u>(sa, tiles, stream)       \
                         : launchScatter<IMPLICIT, WRITE, 1u, 16u>(sa, tiles, stream)
    if (implicit) {
      if (writeKeys) SK_SCATTER(true, true); else SK_SCATTER(true, false);
    } else {
      if (writeKeys) SK_SCATTER(false, true); else SK_SCATTER(false, false);
    }
#undef SK_SCATTER
    if (e != cudaSuccess) return e;
    kin = kout;
    vin = vout;
  }
  return cudaGetLastError();
}

}  // namespace sk
