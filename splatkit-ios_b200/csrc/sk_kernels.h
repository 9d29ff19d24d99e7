// Kernel launch interfaces (host side). Each launcher enqueues on `stream` and returns the
// launch status; none synchronises. Sizes that only the GPU knows (survivor count, instance
// count, LOD cut size) are passed as device pointers and every grid is sized by a host-known
// capacity, so a whole frame enqueues without a host round trip.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <memory>
#include <utility>
#include <vector>

#include "sk_layout.h"

namespace sk {

// ---- visibility (visibility.cu) --------------------------------------------------------
// Ranges of a frame that travel in the cull's parameters, where each thread scans them; more are copied to
// device memory first (two copies ahead of the cull) and searched there. 30k splats at 517 x 389, whole frame,
// scanned against copied: 3 ranges 175 us and 185, 16 ranges 180 and 186, 32 ranges 189 and 194, 64 ranges 202
// and 208; at 1M splats the scan of 64 costs what the copies do. The line stays where the scan is short.
constexpr uint32_t kInlineRanges = 16;
struct VisibilityArgs {
  const GpuSplat* splats;
  const uint32_t* sh;  // shStride words per splat
  uint32_t shStride;   // shDeviceStride(world degree); the frame may use fewer bands
  uint32_t worldCount;
  // ranges mode: record t of the frame is splat t + shift of the last range that starts at or below t
  uint32_t rangeCount;
  uint32_t inlineStart[kInlineRanges], inlineShift[kInlineRanges];  // up to kInlineRanges of them
  const Range* ranges;  // more (device)
  const uint32_t* rangeStarts;
  const uint32_t* indices;     // indexed (LOD) mode
  const uint32_t* indexCount;  // indexed mode: entries in indices (device)
  uint32_t total;              // ranges mode: sum of counts; indexed mode: capacity bound
  uint32_t* keys;
  Projected* projected;
  uint4* spans;  // per survivor: the binning cells its quad touches (sk_tiles.cuh)
  uint32_t tilesX, tilesY;  // binning cells (kBinSize pixels) per row and column
  uint32_t* visibleCount;
  uint64_t* status;    // one word per tile of visibilityTileSplats() records
  uint32_t* counters;  // two words
  uint32_t epoch;
  uint32_t* error;
  PartLabels parts;  // labels.labels null: no part styling
  // the depth sort's digit histogram, summed over the survivors' keys as they are written (the
  // last block turns it into digit bases); sortPasses 0: not summed
  uint32_t* sortAccum;
  uint32_t* sortBases;
  uint32_t sortPasses;
  const Camera* cameraInMemory;  // device; null: `camera`, passed with the launch
  Camera camera;
};
uint32_t visibilityTileSplats();  // records of a tile, and of a batch's work item
cudaError_t launchVisibility(const VisibilityArgs& args, int shDegree, bool key16, bool indexed,
                             cudaStream_t stream);

// A batch of views (visibility.cu): one launch over every view's records, 16-bit depth keys with
// the view id above them, survivors of all views contiguous in (view, source) order.
struct BatchVisibilityArgs {
  const BatchView* views;   // viewCount entries
  const Camera* cameras;    // one per view (device)
  uint32_t viewCount;
  uint32_t items;           // work items: per view max(1, ceil(count / visibilityTileSplats()))
  uint32_t* keys;
  Projected* projected;
  uint4* spans;
  uint32_t* viewFirst;      // viewCount + 1 words: each view's first survivor, then the total
  uint32_t* visibleCount;
  uint64_t* status;         // one word per item
  uint32_t* counters;       // two words
  uint32_t epoch;
  uint32_t* error;
};
cudaError_t launchVisibilityBatch(const BatchVisibilityArgs& args, int shDegree,
                                  cudaStream_t stream);

// ---- radix sort (radix_sort.cu) --------------------------------------------------------
// Stable ascending sort of `count` (key, value) pairs with 8-bit digits: one histogram pass,
// then one onesweep scatter pass per digit. valuesIn null: values are the key positions.
// keysIn is left untouched; keysOut (optional) receives the sorted keys.
struct SortArgs {
  const uint32_t* keysIn;
  const uint32_t* valuesIn;
  uint32_t* keysOut;
  uint32_t* valuesOut;
  const uint32_t* count;  // device
  uint32_t capacity;      // count is clamped to this
  int bits;               // key bits: 8, 16, 24 or 32 (one 8-bit digit pass each)
  // workspace (sortWorkspaceBytes)
  uint32_t* keysA;
  uint32_t* keysB;
  uint32_t* valuesTmp;
  uint32_t* histogram;  // 2 * 4 * 256 words
  uint64_t* status;     // sortTiles(capacity) * 256 words
  uint32_t* counters;   // 2 * 5 words
  uint32_t epoch;       // uses epoch .. epoch + 3
  uint32_t* error;
  uint32_t tileKeys;    // keys per scatter tile: 2048, 4096 (0: the default) or 6144
  uint32_t statusTiles; // tiles the bound status region holds (set by the bind)
  // 1: the kernel that wrote the keys already summed their digits and left the bases in the
  // workspace (VisibilityArgs.sortPasses); the histogram pass is skipped
  uint32_t basesReady;
  // test hook (sk_testing_withhold_sort_status): tile + 1 of the first pass whose look-back
  // status words are not published; 0: none
  uint32_t withheldTilePlusOne;
};
// Where a bound workspace keeps the digit accumulators (zero between sorts) and the bases.
uint32_t* sortDigitAccumulators(const SortArgs& args);
uint32_t* sortDigitBases(const SortArgs& args);
uint32_t sortTileKeys();
size_t sortWorkspaceBytes(uint32_t capacity);
// Carves the workspace into the SortArgs fields.
void sortBindWorkspace(SortArgs& args, void* workspace, uint32_t capacity);
// The same for sorts that may use tiles as small as minTileKeys keys.
size_t sortWorkspaceBytesFor(uint32_t capacity, uint32_t minTileKeys);
void sortBindWorkspaceFor(SortArgs& args, void* workspace, uint32_t capacity, uint32_t minTileKeys);
cudaError_t launchSort(const SortArgs& args, cudaStream_t stream);
// Whether launchSort sorts up to `capacity` keys in one launch (cluster_sort.cu, unless the test hook asks
// for the look-back): it then uses neither the histogram, the counters nor the status words.
bool sortInOneLaunch(uint32_t capacity);
cudaError_t launchClusterSort(const SortArgs& args, uint32_t passes, cudaStream_t stream);
// Clears the counters and histogram accumulators of a bound workspace.
cudaError_t sortResetWorkspace(const SortArgs& args, cudaStream_t stream);

// ---- tile binning (binning.cu) ---------------------------------------------------------
struct BinArgs {
  const uint4* spans;     // per survivor tile spans, indexed like the projected records
  const uint32_t* order;  // depth order (indices into projected)
  const uint32_t* count;  // survivors (device)
  uint32_t capacity;      // bound on count
  uint32_t width, height, tilesX, tilesY;  // tilesX/Y: binning cells per row and column
  uint32_t* instanceKeys;    // binning cell per instance
  uint32_t* instanceValues;  // projected index per instance
  uint16_t* instanceMasks;   // direct lists: the cells of its patch each entry touches (null: not
                             // written, where every patch is one cell)
  uint32_t instanceCapacity;
  uint32_t* instanceCount;  // FrameCounters.instances (the direct lists add to it: zero beforehand)
  uint32_t* overflow;       // FrameCounters.overflow
  uint32_t* blockSums;      // binBlocks(capacity) words of scratch
  // a batch (viewCount > 0): tile ids are batch-wide, each view's from its table entry
  const BatchView* views;
  const uint32_t* viewFirst;  // viewCount + 1 words (BatchVisibilityArgs)
  uint32_t viewCount;
  // emission: 0 walks each warp's items one by one (best near one wave of blocks), 1 balances
  // each warp's output over its lanes (fewer instructions per instance; best for large grids)
  uint32_t balanced;
};
uint32_t binBlocks(uint32_t capacity);
cudaError_t launchBinning(const BinArgs& args, cudaStream_t stream);

// Per binning cell, the [start, end) range of its entries in the cell-sorted instance keys.
// ranges: one uint2 per cell, cleared beforehand by clearTileRanges (cells with no entry keep
// (0, 0)); the clear is issued early so the chained kernels of a frame run back to back.
cudaError_t clearTileRanges(uint2* ranges, uint32_t tiles, cudaStream_t stream);
cudaError_t launchTileRanges(const uint32_t* sortedKeys, const uint32_t* instanceCount,
                             uint32_t instanceCapacity, uint2* ranges, uint32_t tiles,
                             cudaStream_t stream);

// Direct lists (cell_lists.cu) on targets of at most kDirectMaxPatches patches (patchGrid): per patch, the
// front-to-back projected indices of the survivors whose cell box touches it, each with the bits of the cells it touches there. A cell's entries are those of its patch with its
// bit, the same list that binning + stable tile sort + ranges produce. args.instanceValues and
// args.instanceMasks receive the entries, args.instanceCount the number of (survivor, cell) pairs;
// instanceKeys and blockSums are unused.
constexpr uint32_t kDirectMaxPatches = 4096;
struct PatchLists {
  PatchGrid grid;        // the target's patches, by patchGoalsFor(args.capacity)
  void* workspace;       // patchListBytes(capacity, patches), the first patchListStatusBytes() zero
                         // before the first launch
  uint2* ranges;         // per patch [start, end), clamped to the instance capacity
  uint32_t* entryCount;  // FrameCounters.entries
  uint32_t* counters;    // two words, zero before the first launch (each launch restores them)
  uint32_t epoch;        // look-back epoch, fresh per launch
  uint32_t* error;       // SK_DEVERR_* bits
};
// How many patches the target of a frame of up to `capacity` ranks gets.
PatchGoals patchGoalsFor(uint32_t capacity);
// Whether a target of `patches` patches takes the direct path.
bool patchListsFit(uint32_t patches);
size_t patchListBytes(uint32_t capacity, uint32_t patches);
size_t patchListStatusBytes();
cudaError_t launchPatchLists(const BinArgs& args, const PatchLists& lists, cudaStream_t stream);

// Every view of a batch in one launch per pass. View v's ranks are [viewFirst[v], viewFirst[v+1])
// of args.order (at most `capacity` of them), its patches patchBase .. patchBase + patches of the
// batch's ranges; its count/emit blocks are blockBase .. blockBase + patchListBlocks(capacity,
// cells), its patch groups groupBase .. groupBase + patchListGroups(patches), and its block rows the
// patchListRowBytes(capacity, patches, cells) bytes at workspace + work. The look-back runs over the
// groups of all views in view order, so view v's entries follow those of views 0..v-1;
// *entryCount receives the total and args.overflow whether it exceeds args.instanceCapacity.
struct PatchListView {
  uint32_t blockBase, groupBase, patches, patchesX;
  uint32_t patchBase, capacity, shift, pad;
  uint64_t work;
};
struct PatchListBatch {
  const PatchListView* views;  // device table, views in order
  uint32_t viewCount;
  const uint32_t* viewFirst;  // viewCount + 1 rank offsets (device)
  void* workspace;            // the views' block rows, no clearing needed
  uint64_t* status;           // one look-back word per patch group of the batch, zero beforehand
  uint2* ranges;              // the batch's patches
  uint32_t* entryCount;
  uint32_t* counters;         // two words, zero before the first launch (each launch restores them)
  uint32_t epoch;
  uint32_t* error;
  uint32_t blocks, groups, mostPatches;  // totals over the views; the largest view's patches
  bool cells;                            // every view's patches are single cells
};
uint32_t patchListBlocks(uint32_t capacity, bool cells);
uint32_t patchListGroups(uint32_t patches);
size_t patchListRowBytes(uint32_t capacity, uint32_t patches, bool cells);
cudaError_t launchPatchListsBatch(const BinArgs& args, const PatchListBatch& lists, cudaStream_t stream);
// Sets the emission kernel's shared-memory limit (once; before any stream capture).
cudaError_t patchListsConfigure();

// ---- composite (composite.cu) ----------------------------------------------------------
enum PixelFormat : int { kRgba8 = 0, kRgba32f = 1 };
struct CompositeArgs {
  const Projected* projected;
  const uint32_t* values;  // list entries' projected indices, front to back
  const uint16_t* masks;   // direct lists: each entry's cells of its patch; null: lists per cell
  PatchGrid grid;          // direct lists of a frame: the target's patches
  uint32_t patches;        // a batch: 1 when the views' lists start at their patchBase (else binBase)
  const uint2* ranges;     // per patch (direct lists) or per binning cell
  uint32_t width, height, tilesX, tilesY;  // composite tiles (kTileSize pixels)
  uint32_t binsX;                          // binning cells per row
  float background[3];
  int opaque;
  float cutoff;  // transmittance below which a pixel stops
  void* image;   // row 0 on top
  int format;
  uint32_t* fragments;  // FrameCounters.fragments_lo/hi (64-bit add), when countFragments
  uint32_t countFragments;
  uint32_t* loaded;     // FrameCounters.loaded
  // one block per tile firstTile .. firstTile + tiles of the target, or (viewCount > 0) of a batch's tiles,
  // view after view, with image = the batch image
  uint32_t firstTile, tiles;
  const BatchView* views;
  uint32_t viewCount;
  uint32_t records;  // about how many records the lists before this launch were made of (0: few, or no
                     // lists right before it)
};
cudaError_t launchComposite(const CompositeArgs& args, cudaStream_t stream);

// ---- LOD selection (lod.cu) ------------------------------------------------------------
struct LodArgs {
  const LodCluster* clusters;
  const uint32_t* leaves;
  uint32_t clusterCount;
  uint32_t capacity;  // indices buffer size and the guard's bound
  uint32_t limit;     // splats one selection may emit (<= capacity)
  float pixelLimit;
  float colorWeight;
  uint32_t cull;
  uint32_t rounds;
  uint32_t fanout;    // most child clusters of any cluster: round r's frontier holds at most
                      // fanout^r clusters (0: unknown)
  uint32_t frontierCapacity;
  uint32_t* frontier[2];
  uint2* costs;     // (extra | flags, exclusive prefix of extra)
  uint4* offsets;   // (kids, splats, packets exclusive, flags)
  uint4* packets;   // (leafStart, count, destination, 1)
  uint32_t* indices;
  LodState* state;
  uint64_t* status;  // 3 arrays of lodTiles(frontierCapacity) words
  uint32_t* counters;
  uint32_t epoch;  // uses epoch .. epoch + 2 * rounds
  uint32_t* error;
  uint32_t* report;  // six words copied from the state at the end (FrameCounters.lod)
};
uint32_t lodTileClusters();
cudaError_t launchLodSelect(const Camera* cam, const LodArgs& args, cudaStream_t stream);

// ---- LOD tree build (tree_build.cu) -----------------------------------------------------
// The octree of sk_build_lod_tree built on the device from host arrays; the nodes come back in
// the breadth-first layout (node 0 the root), childStart/childCount per node (0/0 for a leaf).
struct LodBuildInput {
  const float* positions;    // host, 3 per splat
  const float* covariances;  // 6
  const float* colors;       // 3
  const float* alphas;
  const float* sh;           // shStride per splat (nullptr when shStride is 0)
  uint32_t count;
  uint32_t shStride;
  float boundsMin[3];
  float extent;  // the largest side of the bounds (at least 1e-6)
  uint32_t depth;          // 1 .. 21
  uint32_t clusterLeaves;  // >= 2
};
// Host arrays that a resize leaves uninitialised (a default-initialising allocator): the arrays
// of a built tree are filled by a bulk copy or a parallel loop right after they are sized, so
// zeroing hundreds of MB on one thread first would only add time.
template <typename T>
struct UninitAllocator : std::allocator<T> {
  template <typename U>
  struct rebind {
    using other = UninitAllocator<U>;
  };
  UninitAllocator() = default;
  template <typename U>
  UninitAllocator(const UninitAllocator<U>&) noexcept {}
  template <typename U>
  void construct(U* p) noexcept {
    ::new (static_cast<void*>(p)) U;
  }
  template <typename U, typename... Args>
  void construct(U* p, Args&&... args) {
    ::new (static_cast<void*>(p)) U(std::forward<Args>(args)...);
  }
};
template <typename T>
using HostArray = std::vector<T, UninitAllocator<T>>;

struct LodBuildOutput {
  uint32_t count = 0;
  HostArray<float> positions, covariances, colors, alphas, sh;
  HostArray<LodNode> layout;
};
constexpr uint32_t kMaxLodBuildLeaves = 0x7fffffffu;
cudaError_t buildLodTreeGpu(const LodBuildInput& in, LodBuildOutput& out);

}  // namespace sk
