// The argsort of up to 32,768 keys in one launch: one cluster of up to 16 blocks runs every digit pass.
//
// A small sort by onesweep passes (radix_sort.cu) is a histogram kernel and one scatter kernel per
// digit, each a chain of launch, tile hand-out, loads, look-back and completion count that lasts about 7
// us whatever the keys, with two cleared workspaces before it. Here a block keeps its 512 * kRows
// positions of the sequence in shared memory for all passes. A pass ranks the keys by ballot matching (as
// radix_sort.cu does: per warp, row by row, in source order), writes the block's digit counts into every
// block of the cluster, and writes the digit runs, staged in order, to the blocks that hold their
// positions (the last pass: to the output); two cluster barriers (hardware barriers of co-scheduled
// blocks, nothing polls) stand in for the kernel boundaries and the look-back, and one more, under the
// loads and the first ranking, makes sure that every block has started. The order is the same.
//
// Bound by the chain of barriers and shared-memory round trips, about 4.5 us a pass: 20,011 32-bit keys
// 37 -> 19.5 us (8 blocks of 1024 threads 29.5, 16 of 1024 21.4, 16 of 256 19.7; counts read from the other
// blocks instead of written to them 29.4); the 16-bit sort of a 4,000-splat frame 15 -> 6.3 us. Beyond 32,768 keys
// 16 SMs are too few: at 100k keys a pass would take as long as a scatter kernel.
#include <cuda_runtime.h>

#include "sk_cluster.cuh"
#include "sk_device.cuh"
#include "sk_kernels.h"
#include "sk_launch.cuh"

namespace sk {
namespace {

constexpr uint32_t kThreads = 512;
constexpr uint32_t kWarps = kThreads / 32;
constexpr uint32_t kBins = 256;
constexpr uint32_t kGroups = kThreads / kBins;       // threads per digit
constexpr uint32_t kGroupWarps = kWarps / kGroups;
constexpr uint32_t kMostBlocks = 16;
constexpr uint32_t kMostRows = 4;

struct ClusterSortArgs {
  const uint32_t* keysIn;
  const uint32_t* valuesIn;  // null: the key positions
  uint32_t* keysOut;         // null: not written
  uint32_t* valuesOut;
  const uint32_t* count;
  uint32_t capacity, passes;
};

struct Smem {
  uint32_t warpCount[kWarps][kBins];  // per warp and digit: its keys, then their first place in the block
  uint32_t groupTotal[kGroups][kBins];
  uint32_t blockTotal[kMostBlocks][kBins];  // every block's keys per digit, written by that block
  uint32_t groupAll[kGroups][kBins], groupBefore[kGroups][kBins];
  uint32_t shift[kBins];       // a key's place in the output less its place in the block
  uint32_t warpSums[kWarps];
};

// Exclusive sum over the 256 values of each group of threads (every group holds the same ones).
__device__ __forceinline__ uint32_t digitScan(uint32_t v, uint32_t* warpSums) {
  const uint32_t warp = threadIdx.x >> 5, lane = laneId();
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t up = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= static_cast<uint32_t>(o)) inc += up;
  }
  if (lane == 31) warpSums[warp] = inc;
  __syncthreads();
  uint32_t before = inc - v;
  const uint32_t first = warp / kGroupWarps * kGroupWarps;
#pragma unroll
  for (uint32_t w = 0; w < kGroupWarps; ++w) before += first + w < warp ? warpSums[first + w] : 0u;
  return before;
}

template <uint32_t kRows>
__global__ void __launch_bounds__(kThreads, 1) clusterSortKernel(const __grid_constant__ ClusterSortArgs a) {
  constexpr uint32_t kShare = kThreads * kRows;
  clusterArrive();
  extern __shared__ uint32_t dynamic[];
  Smem& s = *reinterpret_cast<Smem*>(dynamic);
  uint32_t* stageKey = dynamic + sizeof(Smem) / 4;
  uint32_t* stageValue = stageKey + kShare;
  uint32_t* heldKey = stageValue + kShare;  // the block's positions of the sequence between the passes
  uint32_t* heldValue = heldKey + kShare;
  const uint32_t warp = threadIdx.x >> 5, lane = laneId();
  const uint32_t d = threadIdx.x % kBins, group = threadIdx.x / kBins;
  const uint32_t rank = clusterRank(), blocks = gridDim.x;  // one cluster: the whole grid
  chainedKernelStart();
  const uint32_t n = min(*a.count, a.capacity);
  const uint32_t mine = warp * (32 * kRows) + lane;  // this thread's first place in the block
  const uint32_t held = rank * kShare < n ? min(kShare, n - rank * kShare) : 0u;
  const uint32_t below = lanemaskLt();
  uint32_t key[kRows], value[kRows], at[kRows];
#pragma unroll
  for (uint32_t r = 0; r < kRows; ++r) {
    const uint32_t e = rank * kShare + mine + r * 32;
    key[r] = e < n ? __ldg(a.keysIn + e) : 0xffffffffu;  // missing keys rank behind all others
    value[r] = e < n && a.valuesIn ? __ldg(a.valuesIn + e) : e;
  }
  for (uint32_t p = 0; p < a.passes; ++p) {
    const bool last = p + 1 == a.passes;
    const uint32_t shift = 8 * p;
    for (uint32_t i = threadIdx.x; i < kWarps * kBins; i += kThreads) (&s.warpCount[0][0])[i] = 0;
    __syncthreads();
#pragma unroll
    for (uint32_t r = 0; r < kRows; ++r) {
      const uint32_t digit = (key[r] >> shift) & 0xffu;
      uint32_t peers = 0xffffffffu;
#pragma unroll
      for (uint32_t b = 0; b < 8; ++b) {
        const bool bit = (digit >> b) & 1u;
        const uint32_t vote = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? vote : ~vote;
      }
      const uint32_t before = s.warpCount[warp][digit];
      __syncwarp();
      if ((peers & below) == 0u) s.warpCount[warp][digit] = before + __popc(peers);
      __syncwarp();
      at[r] = before + __popc(peers & below);
    }
    __syncthreads();
    uint32_t counts[kGroupWarps], total = 0, lower = 0;
#pragma unroll
    for (uint32_t w = 0; w < kGroupWarps; ++w) {
      counts[w] = s.warpCount[group * kGroupWarps + w][d];
      total += counts[w];
    }
    s.groupTotal[group][d] = total;
    __syncthreads();
    total = 0;
#pragma unroll
    for (uint32_t g = 0; g < kGroups; ++g) {
      const uint32_t t = s.groupTotal[g][d];
      if (g < group) lower += t;
      total += t;
    }
    if (p == 0) clusterWait();  // every block of the cluster has started
    // The padding of a last block counts as digit 255 here, but no block after it has keys.
    for (uint32_t b = group; b < blocks; b += kGroups) storeRemote(&s.blockTotal[rank][d], b, total);
    const uint32_t local = digitScan(total, s.warpSums);
    uint32_t run = local + lower;
#pragma unroll
    for (uint32_t w = 0; w < kGroupWarps; ++w) {
      s.warpCount[group * kGroupWarps + w][d] = run;
      run += counts[w];
    }
    __syncthreads();
    clusterArrive();  // the block's totals are there
#pragma unroll
    for (uint32_t r = 0; r < kRows; ++r) {
      at[r] += s.warpCount[warp][(key[r] >> shift) & 0xffu];
      stageKey[at[r]] = key[r];
      stageValue[at[r]] = value[r];
    }
    clusterWait();
    uint32_t all = 0, before = 0;
    for (uint32_t b = group; b < blocks; b += kGroups) {
      const uint32_t t = s.blockTotal[b][d];
      if (b < rank) before += t;
      all += t;
    }
    s.groupAll[group][d] = all;
    s.groupBefore[group][d] = before;
    __syncthreads();
    all = before = 0;
#pragma unroll
    for (uint32_t g = 0; g < kGroups; ++g) {
      all += s.groupAll[g][d];
      before += s.groupBefore[g][d];
    }
    const uint32_t base = digitScan(all, s.warpSums);
    if (group == 0) s.shift[d] = base + before - local;
    __syncthreads();
#pragma unroll
    for (uint32_t r = 0; r < kRows; ++r) {
      const uint32_t i = threadIdx.x + r * kThreads;
      if (i < held) {
        const uint32_t k = stageKey[i];
        const uint32_t to = i + s.shift[(k >> shift) & 0xffu];
        if (last) {
          if (a.keysOut) a.keysOut[to] = k;
          a.valuesOut[to] = stageValue[i];
        } else {  // to the block that holds the position
          storeRemote(heldKey + to % kShare, to / kShare, k);
          storeRemote(heldValue + to % kShare, to / kShare, stageValue[i]);
        }
      }
    }
    // every block is through with the totals and the stores of this pass
    clusterArrive();
    clusterWait();
    if (!last) {
#pragma unroll
      for (uint32_t r = 0; r < kRows; ++r) {
        const uint32_t e = mine + r * 32;
        key[r] = e < held ? heldKey[e] : 0xffffffffu;
        value[r] = heldValue[e];
      }
    }
  }
}

template <uint32_t kRows>
constexpr size_t kSharedBytes = sizeof(Smem) + size_t{4} * kThreads * kRows * 4;

template <uint32_t kRows>
void configOf(cudaLaunchConfig_t& config, cudaLaunchAttribute* attribute, uint32_t blocks, cudaStream_t stream) {
  config = cudaLaunchConfig_t{};
  config.gridDim = blocks;
  config.blockDim = kThreads;
  config.dynamicSmemBytes = kSharedBytes<kRows>;
  config.stream = stream;
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = blocks;
  attribute[0].val.clusterDim.y = 1;
  attribute[0].val.clusterDim.z = 1;
  attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute;
  config.numAttrs = 2;
}

template <uint32_t kRows>
cudaError_t configureRows() {
  cudaError_t e = cudaFuncSetAttribute(clusterSortKernel<kRows>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(kSharedBytes<kRows>));
  if (e == cudaSuccess)  // clusters of more than the portable 8 blocks
    e = cudaFuncSetAttribute(clusterSortKernel<kRows>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

template <uint32_t kRows>
cudaError_t launchRows(const ClusterSortArgs& a, uint32_t blocks, cudaStream_t stream) {
  cudaLaunchConfig_t config;
  cudaLaunchAttribute attribute[2];
  configOf<kRows>(config, attribute, blocks, stream);
  return cudaLaunchKernelEx(&config, clusterSortKernel<kRows>, a);
}

// Whether the current device can hold the largest cluster; the kernels are configured on the way.
bool clusterFits() {
  static std::atomic<uint64_t> fits{0};
  return oncePerDevice(fits, [] {
           cudaError_t e = configureRows<1>();
           if (e == cudaSuccess) e = configureRows<2>();
           if (e == cudaSuccess) e = configureRows<4>();
           cudaLaunchConfig_t config;
           cudaLaunchAttribute attribute[2];
           configOf<kMostRows>(config, attribute, kMostBlocks, nullptr);
           config.numAttrs = 1;
           int clusters = 0;
           if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, clusterSortKernel<kMostRows>, &config);
           if (e != cudaSuccess) cudaGetLastError();
           return e != cudaSuccess ? e : (clusters > 0 ? cudaSuccess : cudaErrorNotSupported);
         }) == cudaSuccess;
}

}  // namespace

bool sortInOneLaunch(uint32_t capacity) {
  return capacity <= kMostBlocks * kThreads * kMostRows && clusterFits();
}

cudaError_t launchClusterSort(const SortArgs& s, uint32_t passes, cudaStream_t stream) {
  const ClusterSortArgs a{s.keysIn, s.valuesIn, s.keysOut, s.valuesOut, s.count, s.capacity, passes};
  // few rows first: a pass lasts as long as a block's rows take
  uint32_t rows = 1;
  while (rows < kMostRows && kMostBlocks * kThreads * rows < s.capacity) rows *= 2;
  uint32_t blocks = 1;
  while (blocks * kThreads * rows < s.capacity) blocks *= 2;
  return rows == 1   ? launchRows<1>(a, blocks, stream)
         : rows == 2 ? launchRows<2>(a, blocks, stream)
                     : launchRows<4>(a, blocks, stream);
}

}  // namespace sk
