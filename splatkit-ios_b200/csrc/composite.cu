// Front-to-back compositing of 16x16 pixel tiles.
//
// The equations are the reference's raster stage (splatkit-ios/.../metal/raster/
// SplatRaster.metal:27-44, .../metal/layout/SplatProjection.metalh:155-175, blend state
// .../metal/raster/MetalSplatPipeline.mm:116-140): a pixel offset d = s a1 + t a2 inside the quad
// |s|, |t| <= radius gets alpha = min(1, peak * exp(-(s^2 + t^2) / 2)), dropped below 1/255;
// colour and coverage blend "under": C += (1 - A) alpha c, A += (1 - A) alpha; the background
// goes under what is left. The reference's fp16 target, unorm10 vertex colour and saturation
// mask between four draw batches are replaced by FP32 accumulation and per-pixel early
// termination when the remaining transmittance drops below `cutoff`.
//
// A block of 128 threads owns a 16x16 tile; each thread owns two horizontally adjacent pixels and
// each warp an 8x8-pixel quadrant. The tile reads the list of the 32x32 binning cell it lies in
// (the splats touching the cell, front to back) in batches of 128 records; with the direct lists it
// picks them out of its patch's list (several cells) by their cell bit, 1024 entries at a time.
// Thread i fetches record i (two 128-bit loads), turns it into the coverage form (pixel centre, inverse
// axes, radius, log cutoff, colour) in shared memory and marks which of the four quadrants its
// quad overlaps (separating-axis test). Each warp compacts, by ballot, the batch entries that
// reach it and sweeps only those, both of its pixels per entry. The coverage decision (quad bound
// and 1/255 cutoff) is a fixed sequence of correctly rounded operations, bit-identical to the host
// oracle's FP32 formula.
//
// Bound by instruction issue (73% of the issue slots, half of the ALU's): 1M splats at 1080p take 179M
// warp instructions and 203 us, 26M of them the filter and the staging of records that miss the tile.
// The exponential predicated on the coverage, no minimum where no peak is above 1, a quarter of a load
// per entry for its place and packed row terms took the sweep's entry from 35 instructions to 31
// (193M -> 179M with the filter, 212 -> 203 us).
#include <cuda_runtime.h>

#include <type_traits>

#include "sk_device.cuh"
#include "sk_kernels.h"
#include "sk_launch.cuh"

namespace sk {
namespace {

constexpr uint32_t kThreads = kTileSize * kTileSize / 2;  // 128: two pixels per thread
constexpr uint32_t kWarps = kThreads / 32;
constexpr uint32_t kEntries = kThreads;  // list entries staged per batch (one per thread)
constexpr uint32_t kQuadrant = kTileSize / 2;  // each warp owns an 8x8 quadrant

struct alignas(16) Splat2D {
  float cx, cy, m00, m10;
  float m01, m11, radius, lcut;
  float lpeak, r, g, b;  // lpeak = log2 of the peak alpha
};
static_assert(sizeof(Splat2D) == 48, "Splat2D is three 16-byte words");

struct CompositeSmem {
  Splat2D splat[kEntries];
  // per warp: where in `splat` (bytes) the batch entries are whose quad reaches its quadrant
  alignas(16) uint32_t list[kWarps][kEntries];
  uint8_t reach[kEntries];         // per entry: bit w set when it reaches quadrant w
};

// The direct lists' filter: kPick entries of the patch's list per step, eight per thread (one
// 16-byte load of their masks), the tile's own compacted into `queue` in list order.
constexpr uint32_t kPickPerThread = 8;
constexpr uint32_t kPick = kThreads * kPickPerThread;
struct FilterSmem {
  uint32_t queue[kEntries + kPick];  // positions in the list of entries of the tile's cell
  uint32_t warpTotal[kWarps];
};

// Fills the coverage form; returns the bitmask of the warp quadrants its quad overlaps.
__device__ __forceinline__ uint32_t coverageForm(const uint4 lo, const uint4 hi, float halfW,
                                                 float halfH, float tileX, float tileTop,
                                                 Splat2D& s) {
  s.cx = __fmul_rn(__fadd_rn(asF(lo.x), 1.0f), halfW);
  s.cy = __fmul_rn(__fadd_rn(asF(lo.y), 1.0f), halfH);
  const float a1x = lowHalf(lo.z), a1y = highHalf(lo.z);
  const float a2x = lowHalf(lo.w), a2y = highHalf(lo.w);
  const float det = __fsub_rn(__fmul_rn(a1x, a2y), __fmul_rn(a2x, a1y));
  const float inv = __fdiv_rn(1.0f, det);
  s.m00 = __fmul_rn(a2y, inv);
  s.m01 = -__fmul_rn(a2x, inv);
  s.m10 = -__fmul_rn(a1y, inv);
  s.m11 = __fmul_rn(a1x, inv);
  const float peak = highHalf(hi.y);
  s.lcut = __fmul_rn(2.0f, lnF32(__fmul_rn(255.0f, peak)));  // 2 ln(255 peak), exact doubling
  s.lpeak = __log2f(peak);
  s.radius = asF(hi.z);
  s.r = lowHalf(hi.x);
  s.g = highHalf(hi.x);
  s.b = lowHalf(hi.y);
  const bool any = det != 0.0f && isfinite(inv) && isfinite(s.cx) && isfinite(s.cy);
  if (!any) {
    s.radius = -1.0f;
    return 0u;
  }
  // Separating axes of the quad c + s a1 + t a2 (|s|, |t| <= radius) against each quadrant's
  // square, taken half a pixel beyond its pixel centres (4 px from the quadrant centre): the
  // screen x and y axes and the normals of a1 and a2. The slack keeps the test conservative
  // against the rounding of the inverse used by the coverage decision.
  constexpr float kHalf = 0.5f * kQuadrant;
  const float ex = s.radius * (fabsf(a1x) + fabsf(a2x)) + kHalf;
  const float ey = s.radius * (fabsf(a1y) + fabsf(a2y)) + kHalf;
  const float n1x = -a1y, n1y = a1x, n2x = -a2y, n2y = a2x;
  const float e1 = s.radius * fabsf(a2x * n1x + a2y * n1y) + kHalf * (fabsf(n1x) + fabsf(n1y));
  const float e2 = s.radius * fabsf(a1x * n2x + a1y * n2y) + kHalf * (fabsf(n2x) + fabsf(n2y));
  // the distances of quadrant 0's centre (y up) along the four axes; a quadrant to the right or
  // below is kQuadrant pixels on along x or y
  constexpr float kStep = kQuadrant;
  const float dx = tileX + kHalf - s.cx, dy = tileTop - kHalf - s.cy;
  const float d1 = dx * n1x + dy * n1y, d2 = dx * n2x + dy * n2y;
  const float s1x = kStep * n1x, s1y = kStep * n1y, s2x = kStep * n2x, s2y = kStep * n2y;
  const bool x0 = fabsf(dx) <= ex, x1 = fabsf(dx + kStep) <= ex;
  const bool y0 = fabsf(dy) <= ey, y1 = fabsf(dy - kStep) <= ey;
  uint32_t reach = 0;
  if (x0 && y0 && fabsf(d1) <= e1 && fabsf(d2) <= e2) reach |= 1u;
  if (x1 && y0 && fabsf(d1 + s1x) <= e1 && fabsf(d2 + s2x) <= e2) reach |= 2u;
  if (x0 && y1 && fabsf(d1 - s1y) <= e1 && fabsf(d2 - s2y) <= e2) reach |= 4u;
  if (x1 && y1 && fabsf(d1 + (s1x - s1y)) <= e1 && fabsf(d2 + (s2x - s2y)) <= e2) reach |= 8u;
  return reach;
}

// A thread's two pixels, packed so that Blackwell's paired FP32 instructions (FADD2, FMUL2,
// FFMA2: two independent IEEE operations, each rounded like its scalar form) work on both at once.
// A pixel is finished once its transmittance T is below the cutoff (T never grows); a pixel
// outside the target starts at T = -1.
struct PixelPair {
  float2 T = make_float2(1.0f, 1.0f), r = make_float2(0.0f, 0.0f), g = make_float2(0.0f, 0.0f),
         b = make_float2(0.0f, 0.0f);
};

__device__ __forceinline__ float2 pair(float v) { return make_float2(v, v); }

// A pixel's alpha: min(1, 2^e) by the hardware approximation (relative error about 2^-22) where
// the splat covers it (reach <= radius, q <= lcut) and it is not finished, else 0. kClamp false: e is
// never above 0, where the approximation is never above 1, and the minimum falls away. The exponential
// itself is predicated on the coverage, so that no select follows it. kCount: covered pixels are
// counted in `blended`.
template <bool kCount, bool kClamp>
__device__ __forceinline__ float pixelAlpha(float T, float cutoff, float reach, float radius, float q,
                                            float lcut, float e, uint32_t& blended) {
  float alpha;
  if constexpr (kCount) {
    asm("{\n\t.reg .pred p;\n\t"
        "setp.ge.f32 p, %2, %3;\n\t"
        "setp.le.and.f32 p, %4, %5, p;\n\t"
        "setp.le.and.f32 p, %6, %7, p;\n\t"
        "mov.f32 %0, 0f00000000;\n\t"
        "@p ex2.approx.ftz.f32 %0, %8;\n\t"
        "@p add.u32 %1, %1, 1;\n\t}"
        : "=&f"(alpha), "+r"(blended)
        : "f"(T), "f"(cutoff), "f"(reach), "f"(radius), "f"(q), "f"(lcut), "f"(e));
  } else {
    asm("{\n\t.reg .pred p;\n\t"
        "setp.ge.f32 p, %1, %2;\n\t"
        "setp.le.and.f32 p, %3, %4, p;\n\t"
        "setp.le.and.f32 p, %5, %6, p;\n\t"
        "mov.f32 %0, 0f00000000;\n\t"
        "@p ex2.approx.ftz.f32 %0, %7;\n\t}"
        : "=&f"(alpha)
        : "f"(T), "f"(cutoff), "f"(reach), "f"(radius), "f"(q), "f"(lcut), "f"(e));
  }
  return kClamp ? fminf(alpha, 1.0f) : alpha;
}

// Both pixels against one splat. px = the two pixel centres' x. The coverage terms u, v, q are the
// oracle's FP32 sequence per pixel (px - cx is px + (-cx) exactly); an uncovered or finished pixel
// takes alpha 0, which leaves its colour and transmittance bit for bit as they were, so a warp none
// of whose pixels the splat covers runs the blend all the same (no vote: the unrolled sweep keeps no
// branch between entries). alpha = min(1, 2^(log2 peak - q log2(e) / 2)) and T -= T alpha.
template <bool kCount, bool kClamp>
__device__ __forceinline__ void blendPair(PixelPair& p, const Splat2D* __restrict__ splat, float2 px, float py,
                                          float cutoff, uint32_t& blended) {
  const float4 w0 = reinterpret_cast<const float4*>(splat)[0];  // cx, cy, m00, m10
  const float4 w1 = reinterpret_cast<const float4*>(splat)[1];  // m01, m11, radius, lcut
  const float4 c = reinterpret_cast<const float4*>(splat)[2];   // lpeak, r, g, b
  const float2 mdy = __fmul2_rn(make_float2(w1.x, w1.y), pair(__fsub_rn(py, w0.y)));  // m01 dy, m11 dy
  const float2 dx = __fadd2_rn(px, pair(-w0.x));
  const float2 u = __ffma2_rn(pair(w0.z), dx, pair(mdy.x));
  const float2 v = __ffma2_rn(pair(w0.w), dx, pair(mdy.y));
  // q = u^2 + v^2 against 2 ln(255 peak): the oracle's (u^2 + v^2) / 2 <= ln(255 peak) with both
  // sides doubled, which is exact, so every decision is the same
  const float2 q = __ffma2_rn(u, u, __fmul2_rn(v, v));
  const float2 e = __ffma2_rn(q, pair(-0.7213475204444817f), pair(c.x));  // -q log2(e) / 2
  // |u|, |v| <= radius as one bound on the larger (a NaN u or v makes q NaN, so the q test
  // still fails as the separate bounds would)
  const float2 alpha = make_float2(
      pixelAlpha<kCount, kClamp>(p.T.x, cutoff, fmaxf(fabsf(u.x), fabsf(v.x)), w1.z, q.x, w1.w, e.x, blended),
      pixelAlpha<kCount, kClamp>(p.T.y, cutoff, fmaxf(fabsf(u.y), fabsf(v.y)), w1.z, q.y, w1.w, e.y, blended));
  const float2 weight = __fmul2_rn(p.T, alpha);
  p.r = __ffma2_rn(weight, pair(c.y), p.r);
  p.g = __ffma2_rn(weight, pair(c.z), p.g);
  p.b = __ffma2_rn(weight, pair(c.w), p.b);
  p.T = __ffma2_rn(pair(-1.0f), weight, p.T);
}

// The warp's `count` listed splats, front to back, onto its pixels; stops once every pixel of the
// warp is finished (looked at every 16 entries).
template <bool kCount, bool kClamp>
__device__ __forceinline__ void sweep(const CompositeSmem& sm, const uint32_t* list, uint32_t count,
                                      PixelPair& p, float2 px, float py, float cutoff, uint32_t& blended) {
  auto splatAt = [&](uint32_t offset) {
    return reinterpret_cast<const Splat2D*>(reinterpret_cast<const char*>(sm.splat) + offset);
  };
  for (uint32_t k0 = 0; k0 < count; k0 += 16) {
    if (__all_sync(0xffffffffu, p.T.x < cutoff && p.T.y < cutoff)) break;
    const uint32_t k1 = min(count, k0 + 16);
    uint32_t k = k0;
    for (; k + 4 <= k1; k += 4) {  // four entries' places in one load
      const uint4 at = *reinterpret_cast<const uint4*>(list + k);
      blendPair<kCount, kClamp>(p, splatAt(at.x), px, py, cutoff, blended);
      blendPair<kCount, kClamp>(p, splatAt(at.y), px, py, cutoff, blended);
      blendPair<kCount, kClamp>(p, splatAt(at.z), px, py, cutoff, blended);
      blendPair<kCount, kClamp>(p, splatAt(at.w), px, py, cutoff, blended);
    }
    for (; k < k1; ++k) blendPair<kCount, kClamp>(p, splatAt(list[k]), px, py, cutoff, blended);
  }
}

// The target one tile block draws into: the context's image, or its view's part of a batch image.
struct Target {
  uint32_t width, height, tilesX, tile, binsX, listBase, patchesX, patchShift;
  void* image;
};

template <int kFormat>
__device__ __forceinline__ void writePixel(const CompositeArgs& a, const Target& t, float T,
                                           float r, float g, float b, uint32_t col, uint32_t row) {
  if (col >= t.width || row >= t.height) return;
  float outR, outG, outB, outA;
  if (a.opaque) {
    outR = r + T * a.background[0];
    outG = g + T * a.background[1];
    outB = b + T * a.background[2];
    outA = 1.0f;
  } else {
    outR = r, outG = g, outB = b, outA = 1.0f - T;
  }
  outR = fminf(fmaxf(outR, 0.0f), 1.0f);
  outG = fminf(fmaxf(outG, 0.0f), 1.0f);
  outB = fminf(fmaxf(outB, 0.0f), 1.0f);
  outA = fminf(fmaxf(outA, 0.0f), 1.0f);
  const size_t at = static_cast<size_t>(row) * t.width + col;
  if constexpr (kFormat == kRgba32f) {
    reinterpret_cast<float4*>(t.image)[at] = make_float4(outR, outG, outB, outA);
  } else {
    const uint32_t r8 = __float2uint_rn(outR * 255.0f), g8 = __float2uint_rn(outG * 255.0f);
    const uint32_t b8 = __float2uint_rn(outB * 255.0f), a8 = __float2uint_rn(outA * 255.0f);
    reinterpret_cast<uint32_t*>(t.image)[at] = r8 | (g8 << 8) | (b8 << 16) | (a8 << 24);
  }
}

// Block b is tile firstTile + b: of the target, or with kBatch of the batch, where its view is the last one
// whose first tile is at or below that.
// kCount: count blended fragments (a statistic; without it the loop saves an add per splat).
// kPatches: the lists are per patch, each entry with its cells (else per cell).
template <int kFormat, bool kBatch, bool kCount, bool kPatches>
__global__ void __launch_bounds__(kThreads) compositeKernel(const __grid_constant__ CompositeArgs a) {
  chainedKernelStart();
  __shared__ CompositeSmem sm;
  __shared__ std::conditional_t<kPatches, FilterSmem, uint32_t> filter;
  Target t{a.width, a.height, a.tilesX, a.firstTile + blockIdx.x, a.binsX, 0u, 0u, 0u, a.image};
  if constexpr (kPatches && !kBatch) {
    t.patchesX = a.grid.x, t.patchShift = a.grid.shift;
  }
  if constexpr (kBatch) {
    const uint32_t tile = a.firstTile + blockIdx.x;
    const uint32_t lo = lastAtOrBelow(a.viewCount, tile, [&](uint32_t v) { return __ldg(&a.views[v].tileBase); });
    const BatchView* v = a.views + lo;
    t.width = __ldg(&v->width);
    t.height = __ldg(&v->height);
    t.tilesX = __ldg(&v->tilesX);
    t.tile = tile - __ldg(&v->tileBase);
    t.binsX = __ldg(&v->binsX);
    t.listBase = a.patches ? __ldg(&v->patchBase) : __ldg(&v->binBase);
    if constexpr (kPatches) {
      const PatchGrid g = patchGrid(t.binsX, __ldg(&v->binsY), kSmallPatches);
      t.patchesX = g.x, t.patchShift = g.shift;
    }
    t.image = static_cast<char*>(a.image) +
              __ldg(reinterpret_cast<const unsigned long long*>(&v->pixelOffset)) *
                  (kFormat == kRgba32f ? 16u : 4u);
  }
  const uint32_t tx = t.tile % t.tilesX, ty = t.tile / t.tilesX;
  // the binning cell holding this tile (cells are 2x2 tiles), its patch and its bit there
  const uint32_t binX = tx / 2, binY = ty / 2;
  const uint32_t list =
      t.listBase + (kPatches ? (binY >> t.patchShift) * t.patchesX + (binX >> t.patchShift) : binY * t.binsX + binX);
  const uint32_t inPatch = (1u << t.patchShift) - 1u;
  const uint32_t cellBit = ((binY & inPatch) << t.patchShift) + (binX & inPatch);
  const uint32_t warp = threadIdx.x >> 5, lane = laneId();
  const uint32_t col = tx * kTileSize + (warp & 1u) * kQuadrant + (lane % 4u) * 2u;  // and col + 1
  const uint32_t row = ty * kTileSize + (warp >> 1) * kQuadrant + lane / 4u;
  const float height = static_cast<float>(t.height);
  const float px0 = static_cast<float>(col) + 0.5f, px1 = px0 + 1.0f;
  const float py = static_cast<float>(t.height - row) - 0.5f;  // y up, as NDC
  const float tileX = static_cast<float>(tx * kTileSize);
  const float tileTop = height - static_cast<float>(ty * kTileSize);
  const float halfW = 0.5f * static_cast<float>(t.width);
  const float halfH = 0.5f * height;
  const uint2 range = a.ranges[list];
  const uint32_t below = lanemaskLt();
  const float2 px = make_float2(px0, px1);
  PixelPair p;
  if (!(col < t.width && row < t.height)) p.T.x = -1.0f;
  if (!(col + 1 < t.width && row < t.height)) p.T.y = -1.0f;
  const float cutoff = a.cutoff;
  auto finished = [&] { return p.T.x < cutoff && p.T.y < cutoff; };
  uint32_t blended = 0, loaded = 0;
  // direct lists: the next kPick entries start at `next`, a multiple of eight (so that their masks
  // load as whole 16-byte words); `queued` entries of the tile's cell wait at queue[head ..]
  uint32_t next = range.x & ~(kPickPerThread - 1u), queued = 0, head = 0;
  for (uint32_t start = range.x;; start += kEntries) {
    uint32_t inBatch;
    if constexpr (kPatches) {
      if (queued < kEntries && next < range.y) {
        // the waiting entries move to the front (below the ones added here)
        uint32_t keep = 0;
        if (threadIdx.x < queued) keep = filter.queue[head + threadIdx.x];
        __syncthreads();
        if (threadIdx.x < queued) filter.queue[threadIdx.x] = keep;
        head = 0;
        while (queued < kEntries && next < range.y) {
          const uint32_t first = next + threadIdx.x * kPickPerThread;
          uint32_t mine = 0;  // bit k: entry first + k is in the list and touches the cell
          if (first < range.y) {
            const uint4 m = __ldg(reinterpret_cast<const uint4*>(a.masks + first));
            // the cell's bit of every half, then the eight bits together in list order
            const uint32_t two = 0x00010001u;
            const uint32_t spread = ((m.x >> cellBit) & two) + (((m.y >> cellBit) & two) << 2) +
                                    (((m.z >> cellBit) & two) << 4) + (((m.w >> cellBit) & two) << 6);
            mine = (spread | (spread >> 15)) & 0xffu;
            if (first < range.x) mine &= 0xffu << (range.x - first);
            if (first + kPickPerThread > range.y) mine &= (1u << (range.y - first)) - 1u;
          }
          const uint32_t own = __popc(mine);
          uint32_t inc = own;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= static_cast<uint32_t>(o)) inc += up;
          }
          if (lane == 31) filter.warpTotal[warp] = inc;
          __syncthreads();
          uint32_t at = queued + inc - own;
#pragma unroll
          for (uint32_t w = 0; w < kWarps; ++w) {
            const uint32_t total = filter.warpTotal[w];
            if (w < warp) at += total;
            queued += total;
          }
          for (; mine != 0u; mine &= mine - 1u) filter.queue[at++] = first + __ffs(mine) - 1;
          next += kPick;
          __syncthreads();
        }
      }
      inBatch = min(kEntries, queued);
    } else {
      inBatch = start < range.y ? min(kEntries, range.y - start) : 0u;
    }
    if (inBatch == 0) break;
    loaded += inBatch;
    bool above = false;
#pragma unroll
    for (uint32_t e = threadIdx.x; e < kEntries; e += kThreads) {
      if (e < inBatch) {
        uint32_t entry = start + e;
        if constexpr (kPatches) entry = filter.queue[head + e];
        const uint32_t v = a.values[entry];
        const uint4* p = reinterpret_cast<const uint4*>(a.projected + v);
        Splat2D s;
        sm.reach[e] =
            static_cast<uint8_t>(coverageForm(__ldg(p), __ldg(p + 1), halfW, halfH, tileX, tileTop, s));
        sm.splat[e] = s;
        above = s.lpeak > 0.0f;
      }
    }
    // a peak alpha above 1 (a merged LOD splat) anywhere in the batch: alphas need the clamp
    const bool clamp = __syncthreads_or(above) != 0;
    if (!__all_sync(0xffffffffu, finished())) {
      // this warp's entries, in batch (= depth) order
      uint32_t count = 0;
      for (uint32_t c = 0; c < inBatch; c += 32) {
        const uint32_t j = c + lane;
        const bool mine = j < inBatch && ((sm.reach[j] >> warp) & 1u);
        const uint32_t m = __ballot_sync(0xffffffffu, mine);
        if (mine) sm.list[warp][count + __popc(m & below)] = j * static_cast<uint32_t>(sizeof(Splat2D));
        count += __popc(m);
      }
      __syncwarp();
      if (clamp) {
        sweep<kCount, true>(sm, sm.list[warp], count, p, px, py, cutoff, blended);
      } else {
        sweep<kCount, false>(sm, sm.list[warp], count, p, px, py, cutoff, blended);
      }
    }
    if (__syncthreads_count(finished() ? 0 : 1) == 0) break;
    if constexpr (kPatches) {
      head += inBatch;
      queued -= inBatch;
    }
  }
  // blended fragments: one 64-bit add per block
  __shared__ unsigned long long blockFragments;
  if (threadIdx.x == 0) blockFragments = 0;
  __syncthreads();
  uint32_t warpSum = blended;
  for (int o = 16; o > 0; o >>= 1) warpSum += __shfl_xor_sync(0xffffffffu, warpSum, o);
  if (lane == 0 && warpSum) atomicAdd(&blockFragments, static_cast<unsigned long long>(warpSum));
  __syncthreads();
  if (kCount && threadIdx.x == 0 && blockFragments)
    atomicAdd(reinterpret_cast<unsigned long long*>(a.fragments), blockFragments);
  if (threadIdx.x == 0 && loaded) atomicAdd(a.loaded, loaded);
  writePixel<kFormat>(a, t, p.T.x, p.r.x, p.g.x, p.b.x, col, row);
  writePixel<kFormat>(a, t, p.T.y, p.r.y, p.g.y, p.b.y, col + 1, row);
}

// Where all of a target's blocks are on the chip at once (eight on each of 148 multiprocessors), it is drawn
// as fast as its busiest multiprocessor. Dispatched early, while two or more of the emission's blocks (of 256
// ranks) still hold every multiprocessor, its blocks pile up on those that first have room; launched after
// the emission they spread evenly, for 2 to 3 us. Whole frames, chained and after it: 350k splats at 380 x
// 240 281 us and 223, 500k at 200 x 130 336 and 263, 100k at 520 x 330 97 and 93; 50k there 68.7 and 69.9, 4k
// 36.1 and 38.1. Larger targets level out as their blocks follow one another: 200k at 700 x 450 (1276 tiles)
// 139 and 148, at 900 x 620 144 and 146.
constexpr uint32_t kSpreadTiles = 148 * 8;
constexpr uint32_t kSpreadRecords = 148 * 2 * 256;

template <int kFormat, bool kBatch>
cudaError_t launchKind(const CompositeArgs& a, cudaStream_t stream) {
  const bool count = a.countFragments != 0;
  void (*kernel)(CompositeArgs);
  if (a.masks) {
    kernel = count ? compositeKernel<kFormat, kBatch, true, true> : compositeKernel<kFormat, kBatch, false, true>;
  } else {
    kernel = count ? compositeKernel<kFormat, kBatch, true, false> : compositeKernel<kFormat, kBatch, false, false>;
  }
  if (a.tiles <= kSpreadTiles && a.records > kSpreadRecords) {
    kernel<<<a.tiles, kThreads, 0, stream>>>(a);
    return cudaGetLastError();
  }
  return launchChained(kernel, a.tiles, kThreads, stream, a);
}

template <int kFormat>
cudaError_t launchFormat(const CompositeArgs& a, cudaStream_t stream) {
  return a.viewCount > 0 ? launchKind<kFormat, true>(a, stream) : launchKind<kFormat, false>(a, stream);
}

}  // namespace

cudaError_t launchComposite(const CompositeArgs& a, cudaStream_t stream) {
  if (a.tiles == 0) return cudaSuccess;
  return a.format == kRgba32f ? launchFormat<kRgba32f>(a, stream) : launchFormat<kRgba8>(a, stream);
}

}  // namespace sk
