// Direct lists: each patch's front-to-back list of survivors, written in place.
//
// A patch is a square of 1, 2 or 4 binning cells a side (patchGrid). Its list holds, in depth order,
// one entry per survivor whose box of cells touches it: the survivor's projected index and a bit
// for each of the patch's cells it touches. A composite tile reads its patch's list and keeps the
// entries with its cell's bit, which are the cell's front-to-back list that binning + a stable
// sort of (cell, projected index) pairs by cell give (binning.cu, radix_sort.cu). On a target of at
// most kDirectMaxPatches patches this file builds the lists without a sort:
//   1. count: every block of depth ranks histograms its (survivor, patch) pairs by patch;
//   2. scan: per patch, the running sum of the block histograms gives each block's first slot in
//      the patch's list; the lists' starts come from a decoupled look-back across groups of 8
//      patches, in patch order; the ranges and the entry count follow;
//   3. emit: every block histograms its 8 warps' ranks by patch again, so that warp w starts each
//      patch after warps 0..w-1, then each warp walks its output 32 entries at a time in depth order
//      and writes each entry at its patch's next slot (lanes of one round that share a patch take
//      consecutive slots).
// A batch of views runs each pass once for all of them (launchPatchListsBatch): every block finds
// its view in a table (its first count/emit block and first patch group), works on that view's
// ranks, patches and workspace rows, and the look-back of pass 2 runs over the groups of all views
// in order, so each view's entries start where the previous view's end.
//
// Why patches and not cells on larger targets: a splat of 3 cells touches about 1.4 patches, and a grid of
// 4 x 4 patches is 16 times coarser than the cell grid, so the block histograms of the three passes
// (block x patch words) no longer dominate them, and a splat near the camera, whose box holds hundreds of
// cells, is 16 times fewer entries for the one warp that writes them. The price is the composite's
// filter. 1M splats at 1080p (2040 cells, 135 patches): the passes 105 -> 52 us against lists per cell,
// the composite 193 -> 203. 3M at 3840 x 2160 (8160 cells, 510 patches): 164 us against 668 for the
// stable sort of (cell, splat) pairs that lists per cell needed there. Small targets keep patches of one
// cell: their cell grid is small, and many entries of a patch would miss a tile's cell (24 views of up
// to 640 x 480: composite 1342 us, 1620 with 4 x 4 patches). Where the lines lie stands at PatchGoals.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "sk_device.cuh"
#include "sk_kernels.h"
#include "sk_launch.cuh"
#include "sk_tiles.cuh"

namespace sk {
namespace {

constexpr uint32_t kThreads = 256;
constexpr uint32_t kWarps = kThreads / 32;
// Depth ranks per lane. A frame's count and emission blocks take 512 depth ranks (1024: emission 32 -> 50
// us at 1M). Up to 151,552 ranks, where all blocks of 256 ranks are on the chip at once and a pass lasts as
// long as one block, they take 256: 100k splats at 720p emit in 11 us against 16, the frame 213.6 against
// 217.1; a thumbnail's frame 62.7 against 65.0. Above, 512 ranks halve the rows to scan. A batch whose
// patches are all single cells takes 1024, whose spans then stay in registers (24 views of up to 640 x
// 480: count, scan and emission 84, 23 and 205 us; at 512 ranks 88, 25 and 211); with larger patches 512.
constexpr uint32_t kMostItems = 2;
constexpr uint32_t kCellItems = 4;
constexpr uint32_t kFewRanks = 148 * 4 * kThreads;

constexpr uint32_t kScanThreads = 512;
constexpr uint32_t kGroup = 8;                              // patches per scan block
constexpr uint32_t kScanLanes = kScanThreads / kGroup;      // row lanes per patch
constexpr uint32_t kRowsInRegisters = 16;                   // block rows one row lane keeps
// Boxes of more patches than this are walked by the whole warp, smaller ones by their own lane.
constexpr uint32_t kLanePatches = 8;

struct Work {
  uint32_t* blockRows;  // blocks x patches: each block's count per patch, then (after pass 2) its
                        // first slot in each patch's list
  uint64_t* status;     // one look-back word per group of patches
  // a whole batch in one launch (views non-null): the view table, each view's ranks
  // [viewFirst[v], viewFirst[v + 1]) of args.order, and the workspace its rows are in
  const PatchListView* views;
  uint32_t viewCount;
  const uint32_t* viewFirst;
  uint8_t* base;
  PatchGrid grid;  // a frame's patches
};

// What one block of a pass works on: its block (or patch group) within its view, the view's ranks
// [first, first + n) of the depth order, patches, workspace rows and patch ranges.
struct Job {
  uint32_t block, first, n, patches, patchesX, shift;
  uint32_t* blockRows;
  uint2* ranges;
};

__host__ __device__ inline uint32_t counterWords(uint32_t patches) { return (patches + 1) / 2; }
__host__ __device__ inline size_t align16(size_t n) { return (n + 15) & ~size_t{15}; }
__host__ __device__ inline uint32_t groupsOf(uint32_t patches) { return (patches + kGroup - 1) / kGroup; }
__host__ __device__ inline uint32_t blocksOf(uint32_t capacity, uint32_t items) {
  return (capacity + kThreads * items - 1) / (kThreads * items);
}
// A frame's ranks per lane.
inline uint32_t itemsFor(uint32_t capacity) { return capacity <= kFewRanks ? 1u : kMostItems; }

// The job of block (or patch group, byGroup) `index` of a pass.
__device__ __forceinline__ Job jobOf(const BinArgs& a, const Work& w, uint32_t patches,
                                     uint32_t index, bool byGroup, uint2* ranges) {
  Job j;
  if (!w.views) {  // a frame: the ranks [0, count) of the depth order
    j.block = index;
    j.first = 0;
    j.n = min(*a.count, a.capacity);
    j.patches = patches;
    j.patchesX = w.grid.x;
    j.shift = w.grid.shift;
    j.blockRows = w.blockRows;
    j.ranges = ranges;
    return j;
  }
  const uint32_t lo = lastAtOrBelow(w.viewCount, index, [&](uint32_t v) {
    return byGroup ? __ldg(&w.views[v].groupBase) : __ldg(&w.views[v].blockBase);
  });
  const PatchListView v = w.views[lo];
  j.block = index - (byGroup ? v.groupBase : v.blockBase);
  j.first = w.viewFirst[lo];
  j.n = min(w.viewFirst[lo + 1] - j.first, v.capacity);
  j.patches = v.patches;
  j.patchesX = v.patchesX;
  j.shift = v.shift;
  j.blockRows = reinterpret_cast<uint32_t*>(w.base + v.work);
  j.ranges = ranges + v.patchBase;
  return j;
}

// A frame's workspace: the look-back words at a fixed place (whatever the target, so that they hold
// nothing but look-back words), then the block rows.
constexpr size_t kStatusBytes = size_t{kDirectMaxPatches / kGroup} * 8;

Work workOf(void* workspace, PatchGrid grid) {
  Work w{};
  w.grid = grid;
  w.status = static_cast<uint64_t*>(workspace);
  w.blockRows = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(workspace) + kStatusBytes);
  return w;
}

// Entries of a span: its listed cells where a patch is one cell, else the patches of its box.
__device__ __forceinline__ uint32_t entryCount(const uint4 s, uint32_t shift) {
  if (shift == 0) return spanCount(s);
  const PatchBox b = patchBox(s, shift);
  return b.w * b.h;
}

// visit(cell) for every listed cell of a masked box whose first cell is `first` (flat over the mask's
// bits: rows walked one by one diverge more than the division per cell costs).
template <typename Visit>
__device__ __forceinline__ void visitListed(const uint4 s, uint32_t first, uint32_t tilesX, Visit visit) {
  const uint32_t w = s.y & 0xffffu;
  for (uint32_t m = s.z; m != 0u; m &= m - 1) visit(boxCell(first, __ffs(m) - 1, w, tilesX));
  for (uint32_t m = s.w; m != 0u; m &= m - 1) visit(boxCell(first, 31 + __ffs(m), w, tilesX));
}

// visit(patch) for every entry of the warp's spans: a masked box of single-cell patches is walked bit
// by bit and a box of at most kLanePatches patches patch by patch, by its own lane; a larger one by
// the whole warp. Every lane of the warp calls this.
template <typename Visit>
__device__ __forceinline__ void visitPatches(const uint4 s, uint32_t shift, uint32_t patchesX, Visit visit) {
  const PatchBox b = patchBox(s, shift);
  const uint32_t lane = laneId(), first = b.y0 * patchesX + b.x0;
  uint32_t area = b.w * b.h;
  if (shift == 0 && area <= 64) {
    visitListed(s, first, patchesX, visit);
    area = 0;
  }
  if (area <= kLanePatches && area != 0) {
    for (uint32_t y = 0; y < b.h; ++y)
      for (uint32_t x = 0; x < b.w; ++x) visit(first + y * patchesX + x);
  }
  uint32_t big = __ballot_sync(0xffffffffu, area > kLanePatches);
  while (big != 0u) {
    const uint32_t src = __ffs(big) - 1;
    big &= big - 1;
    const uint32_t w = __shfl_sync(0xffffffffu, b.w, src), n = __shfl_sync(0xffffffffu, area, src);
    const uint32_t at = __shfl_sync(0xffffffffu, first, src);
    for (uint32_t k = lane; k < n; k += 32) visit(boxCell(at, k, w, patchesX));
  }
}

// Pass 1: each block's entries per patch; the (survivor, cell) pairs are added up beside them.
template <uint32_t kItems>
__global__ void __launch_bounds__(kThreads)
    patchCountKernel(const __grid_constant__ BinArgs a, Work work, uint32_t patches) {
  constexpr uint32_t kBlockRanks = kThreads * kItems;
  chainedKernelStart();
  extern __shared__ uint32_t hist[];
  __shared__ uint32_t warpPairs[kWarps];
  const Job job = jobOf(a, work, patches, blockIdx.x, false, nullptr);
  const uint32_t n = job.n;
  patches = job.patches;
  const uint32_t* order = a.order + job.first;
  const uint32_t begin = job.block * kBlockRanks;
  if (begin >= n) return;  // rows of idle blocks are never read
  uint32_t value[kItems];
#pragma unroll
  for (uint32_t r = 0; r < kItems; ++r) {
    const uint32_t i = begin + r * kThreads + threadIdx.x;
    value[r] = i < n ? order[i] : 0xffffffffu;
  }
  for (uint32_t c = threadIdx.x; c < patches; c += kThreads) hist[c] = 0;
  __syncthreads();
  uint4 span[kItems];
#pragma unroll
  for (uint32_t r = 0; r < kItems; ++r)
    span[r] = value[r] != 0xffffffffu ? __ldg(a.spans + value[r]) : make_uint4(0, 0, 0, 0);
  uint32_t pairs = 0;
#pragma unroll
  for (uint32_t r = 0; r < kItems; ++r) {
    pairs += spanCount(span[r]);
    visitPatches(span[r], job.shift, job.patchesX, [](uint32_t p) { atomicAdd(&hist[p], 1u); });
  }
  pairs = __reduce_add_sync(0xffffffffu, pairs);
  if (laneId() == 0) warpPairs[threadIdx.x >> 5] = pairs;
  __syncthreads();
  uint32_t* row = job.blockRows + size_t{job.block} * patches;
  for (uint32_t c = threadIdx.x; c < patches; c += kThreads) row[c] = hist[c];
  if (threadIdx.x == 0) {
    uint32_t sum = 0;
    for (uint32_t w = 0; w < kWarps; ++w) sum += warpPairs[w];
    atomicAdd(a.instanceCount, sum);
  }
}

// Pass 2: one block per group of 8 patches (groups handed out in start order, so a group only
// waits on groups already running). Thread t is row lane t / 8 of the group's patch t % 8: it sums
// a contiguous share of the block rows, the first 16 of them kept in registers between the two
// sweeps (a warp reads four rows' 32-byte sectors at a time).
template <uint32_t kItems>
__global__ void __launch_bounds__(kScanThreads)
    patchScanKernel(const __grid_constant__ BinArgs a, Work work, uint32_t patches, uint2* ranges,
                    uint32_t* entryCount, uint32_t* counters, uint32_t epoch, uint32_t* error) {
  chainedKernelStart();
  __shared__ uint32_t part[kScanLanes * kGroup];
  __shared__ uint32_t totals[kGroup], starts[kGroup];
  const uint32_t group = takeTile(counters);  // over all views of a batch
  const Job job = jobOf(a, work, patches, group, true, ranges);
  patches = job.patches;
  const uint32_t active = blocksOf(job.n, kItems);
  const uint32_t warp = threadIdx.x >> 5, lane = laneId();
  const uint32_t c = threadIdx.x % kGroup, rowLane = threadIdx.x / kGroup;
  const uint32_t patch = job.block * kGroup + c;
  const bool valid = patch < patches;
  const uint32_t share = (active + kScanLanes - 1) / kScanLanes;
  const uint32_t r0 = min(rowLane * share, active), r1 = min(r0 + share, active);
  uint32_t* rows = job.blockRows + patch;
  uint32_t v[kRowsInRegisters];
  uint32_t sum = 0;
#pragma unroll
  for (uint32_t k = 0; k < kRowsInRegisters; ++k) {
    const uint32_t row = r0 + k;
    v[k] = valid && row < r1 ? __ldcg(rows + size_t{row} * patches) : 0u;
    sum += v[k];
  }
  for (uint32_t at = r0 + kRowsInRegisters; at < r1; at += kRowsInRegisters) {
#pragma unroll
    for (uint32_t k = 0; k < kRowsInRegisters; ++k)
      if (valid && at + k < r1) sum += __ldcg(rows + size_t{at + k} * patches);
  }
  part[threadIdx.x] = sum;
  __syncthreads();
  if (warp < kGroup) {  // warp w: the running sum of patch w's 64 row lanes, two per lane
    uint32_t own[kScanLanes / 32], total = 0;
#pragma unroll
    for (uint32_t k = 0; k < kScanLanes / 32; ++k) {
      own[k] = part[(lane * (kScanLanes / 32) + k) * kGroup + warp];
      total += own[k];
    }
    uint32_t inc = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= static_cast<uint32_t>(o)) inc += up;
    }
    uint32_t run = inc - total;
#pragma unroll
    for (uint32_t k = 0; k < kScanLanes / 32; ++k) {
      part[(lane * (kScanLanes / 32) + k) * kGroup + warp] = run;
      run += own[k];
    }
    if (lane == 31) totals[warp] = inc;
  }
  __syncthreads();
  if (warp == 0) {
    const uint32_t total = lane < kGroup ? totals[lane] : 0u;
    uint32_t inc = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= static_cast<uint32_t>(o)) inc += up;
    }
    const uint32_t aggregate = __shfl_sync(0xffffffffu, inc, 31);
    uint32_t before = 0;
    if (group == 0) {
      if (lane == 0) storeStatus(work.status, makeStatus(epoch, kFlagPrefix, aggregate));
    } else {
      if (lane == 0) storeStatus(work.status + group, makeStatus(epoch, kFlagAggregate, aggregate));
      before = warpLookback(work.status, group, epoch, error);
      if (lane == 0)
        storeStatus(work.status + group, makeStatus(epoch, kFlagPrefix, before + aggregate));
    }
    const uint32_t start = before + inc - total;
    if (lane < kGroup) {
      starts[lane] = start;
      if (job.block * kGroup + lane < patches)
        job.ranges[job.block * kGroup + lane] = make_uint2(min(start, a.instanceCapacity),
                                                           min(start + total, a.instanceCapacity));
    }
    if (group == gridDim.x - 1 && lane == 31) {
      const uint32_t entries = before + aggregate;
      *entryCount = entries;
      *a.overflow = entries > a.instanceCapacity ? 1u : 0u;
    }
  }
  __syncthreads();
  if (valid) {  // each count becomes the block's first slot in the patch's list, in place
    uint32_t run = part[threadIdx.x] + starts[c];
#pragma unroll
    for (uint32_t k = 0; k < kRowsInRegisters; ++k) {
      const uint32_t row = r0 + k;
      if (row < r1) rows[size_t{row} * patches] = run;
      run += v[k];
    }
    // the rows past the registers, read again: a batch of loads, then their stores
    for (uint32_t at = r0 + kRowsInRegisters; at < r1; at += kRowsInRegisters) {
#pragma unroll
      for (uint32_t k = 0; k < kRowsInRegisters; ++k)
        v[k] = at + k < r1 ? __ldcg(rows + size_t{at + k} * patches) : 0u;
#pragma unroll
      for (uint32_t k = 0; k < kRowsInRegisters; ++k) {
        if (at + k < r1) rows[size_t{at + k} * patches] = run;
        run += v[k];
      }
    }
  }
  finishTile(counters);
}

// One round of a warp's output: lanes with an entry (valid) write it at their patch's next slots in lane
// order. Lanes with the same patch take consecutive slots (a match instruction finds them: one ballot per bit
// of a patch index took 216 us of the 24-view batch's emission against 205, 33.7 of a 1M frame's against 32.5).
__device__ __forceinline__ void writeRound(const BinArgs& a, const uint32_t* where, uint32_t* mine, bool valid,
                                           uint32_t patch, uint32_t value, uint32_t mask) {
  const uint32_t peers = __match_any_sync(0xffffffffu, valid ? patch : 0xffffffffu);
  const uint32_t half = (patch & 1u) * 16;
  uint32_t slot = 0;
  if (valid) slot = where[patch] + ((mine[patch >> 1] >> half) & 0xffffu) + __popc(peers & lanemaskLt());
  __syncwarp();
  if (valid && laneId() == 31 - __clz(peers)) atomicAdd(mine + (patch >> 1), __popc(peers) << half);
  __syncwarp();
  if (valid && slot < a.instanceCapacity) {
    a.instanceValues[slot] = value;
    if (a.instanceMasks) a.instanceMasks[slot] = static_cast<uint16_t>(mask);
  }
}

// Zeroes the block's slot counters and fetches its first slots.
__device__ __forceinline__ void emitSetup(const Job& job, uint32_t* slots, uint32_t* where, uint32_t words) {
  for (uint32_t i = threadIdx.x; i < kWarps * words; i += kThreads) slots[i] = 0;
  const uint32_t* starts = job.blockRows + size_t{job.block} * job.patches;
  for (uint32_t c = threadIdx.x; c < job.patches; c += kThreads) where[c] = __ldcg(starts + c);
}

// Warp w's first slot per patch: the counts of warps 0..w-1 (both halves of a word at once).
__device__ __forceinline__ void slotsFromCounts(uint32_t* slots, uint32_t words) {
  for (uint32_t q = threadIdx.x; q < words; q += kThreads) {
    uint32_t run = 0;
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w) {
      const uint32_t v = slots[w * words + q];
      slots[w * words + q] = run;
      run += v;
    }
  }
}

// Pass 3 where every patch is one cell. The warp's spans stay in registers, and a masked span's cells are
// staged by the lane that has it (a box of more than 64 cells by the whole warp): most splats of such
// targets list one or two cells, so that the walk costs less than finding each position's span does, and a
// box of many cells is walked twice, where patchEmitKernel's windows each walk it again. Whole frames of single
// cells against patchEmitKernel's single-cell branch: 200k splats at 640 x 480 from 4 m 120 us and 177, 20k from
// 6 m 53 and 67, 30k at 517 x 389 from 15 m 52.6 and 54.5, 1M at 400 x 300 210 and 201. 24 views of up to 640 x
// 480: count, scan and emission 84, 23 and 205 us, there (at 512 ranks) 97, 25 and 192.
template <uint32_t kItems>
__global__ void __launch_bounds__(kThreads)
    cellEmitKernel(const __grid_constant__ BinArgs a, Work work, uint32_t patches) {
  constexpr uint32_t kBlockRanks = kThreads * kItems;
  constexpr uint32_t kChunk = 32 * kItems;  // ranks per warp
  constexpr uint32_t kWindow = 8 * kChunk;  // positions staged at a time
  static_assert(kChunk <= 256, "an item is a byte");
  chainedKernelStart();
  extern __shared__ uint32_t patchSmem[];
  __shared__ uint32_t itemValue[kWarps][kChunk];
  __shared__ uint16_t stageCell[kWarps][kWindow];
  __shared__ uint8_t stageItem[kWarps][kWindow];
  const Job job = jobOf(a, work, patches, blockIdx.x, false, nullptr);
  const uint32_t n = job.n, cellsX = job.patchesX;
  const uint32_t* order = a.order + job.first;
  const uint32_t begin = job.block * kBlockRanks;
  if (begin >= n) return;
  const uint32_t warp = threadIdx.x >> 5, lane = laneId();
  uint32_t value[kItems], offset[kItems];
  uint4 span[kItems];
#pragma unroll
  for (uint32_t r = 0; r < kItems; ++r) {
    const uint32_t i = begin + warp * kChunk + r * 32 + lane;
    value[r] = i < n ? order[i] : 0xffffffffu;
  }
  const uint32_t words = counterWords(job.patches);
  uint32_t* slots = patchSmem;
  uint32_t* where = patchSmem + kWarps * words;
  emitSetup(job, slots, where, words);
  uint32_t* mine = slots + warp * words;
  uint16_t* sCell = stageCell[warp];
  uint8_t* sItem = stageItem[warp];
  // the warp's items in (row, lane) order = depth order, with their first output position
  uint32_t total = 0;
#pragma unroll
  for (uint32_t r = 0; r < kItems; ++r) {
    span[r] = value[r] != 0xffffffffu ? __ldg(a.spans + value[r]) : make_uint4(0, 0, 0, 0);
    itemValue[warp][r * 32 + lane] = value[r];
  }
#pragma unroll
  for (uint32_t r = 0; r < kItems; ++r) {
    const uint32_t cnt = spanCount(span[r]);
    uint32_t inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= static_cast<uint32_t>(o)) inc += up;
    }
    offset[r] = total + inc - cnt;
    total += __shfl_sync(0xffffffffu, inc, 31);
  }
  __syncthreads();  // the counters are zero, the starts there

  // put(cell, position, item) for every entry at a position of [lo, hi)
  auto walk = [&](uint32_t lo, uint32_t hi, auto put) {
#pragma unroll
    for (uint32_t r = 0; r < kItems; ++r) {
      const uint32_t w = span[r].y & 0xffffu, area = spanArea(span[r]), item = r * 32 + lane;
      const uint32_t first = (span[r].x >> 16) * cellsX + (span[r].x & 0xffffu);
      uint32_t pos = offset[r];
      if (area <= 64 && pos < hi)
        visitListed(span[r], first, cellsX, [&](uint32_t cell) {
          if (pos >= lo && pos < hi) put(cell, pos, item);
          ++pos;
        });
      uint32_t big = __ballot_sync(0xffffffffu, area > 64 && offset[r] < hi && offset[r] + area > lo);
      while (big != 0u) {
        const uint32_t src = __ffs(big) - 1;
        big &= big - 1;
        const uint32_t bw = __shfl_sync(0xffffffffu, w, src), cells = __shfl_sync(0xffffffffu, area, src);
        const uint32_t at = __shfl_sync(0xffffffffu, first, src), from = __shfl_sync(0xffffffffu, offset[r], src);
        const uint32_t k0 = lo > from ? lo - from : 0u, k1 = min(cells, hi - from);
        for (uint32_t k = k0 + lane; k < k1; k += 32) put(boxCell(at, k, bw, cellsX), from + k, r * 32 + src);
      }
    }
  };
  // every entry counted by cell, the first window staged
  walk(0u, 0xffffffffu, [&](uint32_t cell, uint32_t pos, uint32_t item) {
    atomicAdd(mine + (cell >> 1), 1u << ((cell & 1u) * 16));
    if (pos < kWindow) {
      sCell[pos] = static_cast<uint16_t>(cell);
      sItem[pos] = static_cast<uint8_t>(item);
    }
  });
  __syncthreads();
  slotsFromCounts(slots, words);
  __syncthreads();
  for (uint32_t w0 = 0; w0 < total; w0 += kWindow) {
    const uint32_t w1 = min(total, w0 + kWindow);
    if (w0 > 0) {
      __syncwarp();
      walk(w0, w1, [&](uint32_t cell, uint32_t pos, uint32_t item) {
        sCell[pos - w0] = static_cast<uint16_t>(cell);
        sItem[pos - w0] = static_cast<uint8_t>(item);
      });
    }
    __syncwarp();
    for (uint32_t p0 = w0; p0 < w1; p0 += 32) {
      const uint32_t p = p0 + lane;
      const bool valid = p < w1;
      uint32_t cell = 0, val = 0;
      if (valid) {
        cell = sCell[p - w0];
        val = itemValue[warp][sItem[p - w0]];
      }
      writeRound(a, where, mine, valid, cell, val, 1u);
    }
  }
}

// Pass 3. Dynamic shared memory: kWarps x words per-warp slot counters (16-bit halves: a warp's
// slots count from the block's first slot in the patch, at most the block's ranks on), then each patch's
// first slot for the block. A warp's entries, in depth order, are worked out kWindow positions at a
// time, one position per lane and step (however many patches the items have), and staged as
// (patch, item, cell mask); a warp of more entries works each further window out when it writes it.
template <uint32_t kItems>
__global__ void __launch_bounds__(kThreads)
    patchEmitKernel(const __grid_constant__ BinArgs a, Work work, uint32_t patches) {
  constexpr uint32_t kBlockRanks = kThreads * kItems;
  constexpr uint32_t kChunk = 32 * kItems;  // ranks per warp
  constexpr uint32_t kWindow = 4 * kChunk;  // positions staged at a time
  static_assert(kChunk < 256, "an item and a marker are bytes");
  chainedKernelStart();
  extern __shared__ uint32_t patchSmem[];
  __shared__ uint4 itemSpan[kWarps][kChunk];
  __shared__ uint32_t itemValue[kWarps][kChunk], itemOffset[kWarps][kChunk];
  __shared__ uint16_t stagePatch[kWarps][kWindow], stageMask[kWarps][kWindow];
  __shared__ alignas(4) uint8_t stageItem[kWarps][kWindow];
  const Job job = jobOf(a, work, patches, blockIdx.x, false, nullptr);
  const uint32_t n = job.n;
  patches = job.patches;
  const uint32_t* order = a.order + job.first;
  const uint32_t begin = job.block * kBlockRanks;
  if (begin >= n) return;
  const uint32_t warp = threadIdx.x >> 5, lane = laneId();
  uint32_t value[kItems];
#pragma unroll
  for (uint32_t r = 0; r < kItems; ++r) {
    const uint32_t i = begin + warp * kChunk + r * 32 + lane;
    value[r] = i < n ? order[i] : 0xffffffffu;
  }
  const uint32_t words = counterWords(patches);
  uint32_t* slots = patchSmem;
  uint32_t* where = patchSmem + kWarps * words;
  emitSetup(job, slots, where, words);
  uint32_t* mine = slots + warp * words;
  uint16_t* sPatch = stagePatch[warp];
  uint16_t* sMask = stageMask[warp];
  uint8_t* sItem = stageItem[warp];
  uint32_t* sOffset = itemOffset[warp];
  // the warp's items in (row, lane) order = depth order, with their first output position
  uint32_t total = 0, listed = 0;  // listed: bit r when item r * 32 + lane has a patch
#pragma unroll
  for (uint32_t r = 0; r < kItems; ++r) {
    const uint4 span = value[r] != 0xffffffffu ? __ldg(a.spans + value[r]) : make_uint4(0, 0, 0, 0);
    const uint32_t cnt = entryCount(span, job.shift);
    uint32_t inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= static_cast<uint32_t>(o)) inc += up;
    }
    itemSpan[warp][r * 32 + lane] = span;
    itemValue[warp][r * 32 + lane] = value[r];
    sOffset[r * 32 + lane] = total + inc - cnt;
    if (cnt) listed |= 1u << r;
    total += __shfl_sync(0xffffffffu, inc, 31);
  }
  __syncthreads();  // the counters are zero, the starts there

  // Stages the entries at positions [w0, w1). Single-cell patches (a batch's small targets beside larger
  // ones, at kMostItems): every lane walks its items' listed cells (most items have one or two; a box of
  // more than 64 cells is walked by the whole warp).
  // Larger patches: one position per lane and step; every item marks its first position, and an
  // entry's item is the last mark at or before its position (a running maximum).
  auto stageWindow = [&](uint32_t w0, uint32_t w1, uint32_t& carry, bool count) {
    if (kItems == kMostItems && job.shift == 0) {
      auto put = [&](uint32_t patch, uint32_t pos, uint32_t item) {
        if (pos < w0 || pos >= w1) return;
        if (count) atomicAdd(mine + (patch >> 1), 1u << ((patch & 1u) * 16));
        sPatch[pos - w0] = static_cast<uint16_t>(patch);
        sMask[pos - w0] = 1u;
        sItem[pos - w0] = static_cast<uint8_t>(item);
      };
#pragma unroll 1
      for (uint32_t r = 0; r < kItems; ++r) {
        const uint32_t item = r * 32 + lane;
        const uint4 span = itemSpan[warp][item];
        const uint32_t w = span.y & 0xffffu, area = spanArea(span);
        const uint32_t first = (span.x >> 16) * job.patchesX + (span.x & 0xffffu);
        uint32_t pos = sOffset[item];
        if (area <= 64 && pos < w1) {
          visitListed(span, first, job.patchesX, [&](uint32_t cell) { put(cell, pos++, item); });
        }
        uint32_t big = __ballot_sync(0xffffffffu, area > 64);
        while (big != 0u) {
          const uint32_t src = __ffs(big) - 1;
          big &= big - 1;
          const uint32_t bw = __shfl_sync(0xffffffffu, w, src), n = __shfl_sync(0xffffffffu, area, src);
          const uint32_t at = __shfl_sync(0xffffffffu, first, src), from = __shfl_sync(0xffffffffu, pos, src);
          for (uint32_t k = lane; k < n; k += 32) put(boxCell(at, k, bw, job.patchesX), from + k, r * 32 + src);
        }
      }
      return;
    }
    for (uint32_t i = lane; i < kWindow / 4; i += 32) reinterpret_cast<uint32_t*>(sItem)[i] = 0u;
    __syncwarp();
#pragma unroll
    for (uint32_t r = 0; r < kItems; ++r) {
      const uint32_t at = sOffset[r * 32 + lane];
      if (((listed >> r) & 1u) && at >= w0 && at < w1) sItem[at - w0] = static_cast<uint8_t>(r * 32 + lane + 1);
    }
    __syncwarp();
    for (uint32_t p0 = w0; p0 < w1; p0 += 32) {
      const uint32_t p = p0 + lane;
      uint32_t mark = p < w1 ? sItem[p - w0] : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, mark, o);
        if (lane >= static_cast<uint32_t>(o)) mark = max(mark, up);
      }
      mark = max(mark, carry);
      carry = __shfl_sync(0xffffffffu, mark, 31);
      if (p < w1) {
        const uint32_t item = mark - 1;
        const uint4 span = itemSpan[warp][item];
        const PatchBox box = patchBox(span, job.shift);
        const uint32_t k = p - sOffset[item];
        const uint32_t y = static_cast<uint32_t>(__fdividef(static_cast<float>(k) + 0.5f, static_cast<float>(box.w)));
        const uint32_t px = box.x0 + (k - y * box.w), py = box.y0 + y;
        const uint32_t patch = py * job.patchesX + px;
        if (count) atomicAdd(mine + (patch >> 1), 1u << ((patch & 1u) * 16));
        sPatch[p - w0] = static_cast<uint16_t>(patch);
        sMask[p - w0] = static_cast<uint16_t>(patchMask(span, px, py, job.shift));
        sItem[p - w0] = static_cast<uint8_t>(item);
      }
      __syncwarp();
    }
  };
  // every entry counted by patch; a single window stays staged
  for (uint32_t w0 = 0, carry = 0; w0 < total; w0 += kWindow)
    stageWindow(w0, min(total, w0 + kWindow), carry, true);
  __syncthreads();
  slotsFromCounts(slots, words);
  __syncthreads();

  for (uint32_t w0 = 0, carry = 0; w0 < total; w0 += kWindow) {
    const uint32_t w1 = min(total, w0 + kWindow);
    if (total > kWindow) {
      __syncwarp();
      stageWindow(w0, w1, carry, false);
    }
    __syncwarp();
    for (uint32_t p0 = w0; p0 < w1; p0 += 32) {
      const uint32_t p = p0 + lane;
      const bool valid = p < w1;
      uint32_t patch = 0, val = 0, mask = 0;
      if (valid) {
        patch = sPatch[p - w0];
        mask = sMask[p - w0];
        val = itemValue[warp][sItem[p - w0]];
      }
      writeRound(a, where, mine, valid, patch, val, mask);
    }
  }
}

size_t emitDynamicBytes(uint32_t patches) {
  return (size_t{kWarps} * counterWords(patches) + patches) * sizeof(uint32_t);
}

size_t countDynamicBytes(uint32_t patches) { return size_t{patches} * sizeof(uint32_t); }

}  // namespace

PatchGoals patchGoalsFor(uint32_t capacity) { return capacity <= kFewRanks ? kSmallPatches : kFramePatches; }

bool patchListsFit(uint32_t patches) { return patches > 0 && patches <= kDirectMaxPatches; }

uint32_t patchListBlocks(uint32_t capacity, bool cells) {
  return blocksOf(std::max(capacity, 1u), cells ? kCellItems : kMostItems);
}

uint32_t patchListGroups(uint32_t patches) { return groupsOf(patches); }

size_t patchListRowBytes(uint32_t capacity, uint32_t patches, bool cells) {
  return align16(size_t{patchListBlocks(capacity, cells)} * patches * 4);
}

size_t patchListBytes(uint32_t capacity, uint32_t patches) {
  return kStatusBytes + align16(size_t{blocksOf(std::max(capacity, 1u), itemsFor(capacity))} * std::max(patches, 1u) * 4);
}

size_t patchListStatusBytes() { return kStatusBytes; }

namespace {

cudaError_t launchPasses(uint32_t items, bool cells, const BinArgs& a, const Work& work, uint32_t patches,
                         uint32_t blocks, uint32_t groups, uint2* ranges, uint32_t* entryCount, uint32_t* counters,
                         uint32_t epoch, uint32_t* error, cudaStream_t stream) {
  const auto count = items == 1 ? patchCountKernel<1> : items == 2 ? patchCountKernel<2> : patchCountKernel<4>;
  const auto scan = items == 1 ? patchScanKernel<1> : items == 2 ? patchScanKernel<2> : patchScanKernel<4>;
  const auto emit = !cells       ? items == 1 ? patchEmitKernel<1> : patchEmitKernel<2>
                    : items == 1 ? cellEmitKernel<1>
                    : items == 2 ? cellEmitKernel<2>
                                 : cellEmitKernel<4>;
  cudaError_t e = patchListsConfigure();
  if (e == cudaSuccess)
    e = launchChainedShared(count, blocks, kThreads, countDynamicBytes(patches), stream, a, work, patches);
  if (e == cudaSuccess)
    e = launchChained(scan, groups, kScanThreads, stream, a, work, patches, ranges, entryCount, counters, epoch,
                      error);
  if (e == cudaSuccess)
    e = launchChainedShared(emit, blocks, kThreads, emitDynamicBytes(patches), stream, a, work, patches);
  return e;
}

}  // namespace

cudaError_t patchListsConfigure() {
  static std::atomic<uint64_t> done{0};
  return oncePerDevice(done, [] {
    // targets of single-cell patches have at most 320 of them: within the default limit
    const int most = static_cast<int>(emitDynamicBytes(kDirectMaxPatches));
    const cudaError_t e =
        cudaFuncSetAttribute(patchEmitKernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    return e != cudaSuccess
               ? e
               : cudaFuncSetAttribute(patchEmitKernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  });
}

cudaError_t launchPatchLists(const BinArgs& a, const PatchLists& lists, cudaStream_t stream) {
  const PatchGrid g = lists.grid;
  const uint32_t patches = g.x * g.y, items = itemsFor(a.capacity);
  if (!patchListsFit(patches) || a.capacity == 0) return cudaErrorInvalidValue;
  return launchPasses(items, g.shift == 0, a, workOf(lists.workspace, g), patches, blocksOf(a.capacity, items),
                      groupsOf(patches), lists.ranges, lists.entryCount, lists.counters, lists.epoch, lists.error,
                      stream);
}

cudaError_t launchPatchListsBatch(const BinArgs& a, const PatchListBatch& lists, cudaStream_t stream) {
  if (lists.viewCount == 0 || lists.blocks == 0 || lists.groups == 0 || !patchListsFit(lists.mostPatches))
    return cudaErrorInvalidValue;
  Work work{};
  work.status = lists.status;
  work.views = lists.views;
  work.viewCount = lists.viewCount;
  work.viewFirst = lists.viewFirst;
  work.base = static_cast<uint8_t*>(lists.workspace);
  // each block reads its own view's patches from the table
  return launchPasses(lists.cells ? kCellItems : kMostItems, lists.cells, a, work, lists.mostPatches, lists.blocks,
                      lists.groups, lists.ranges, lists.entryCount, lists.counters, lists.epoch, lists.error, stream);
}

}  // namespace sk
