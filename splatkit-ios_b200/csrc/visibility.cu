// The visibility pass: per splat, reveal clip, opacity cut, view transform, near/far test,
// 2D covariance, ellipse axes, quad radius, edge margin, sub-pixel cut, SH colour and depth
// key; survivors compacted in SOURCE order.
//
// Follows splatkit-ios/Sources/SplatKitCore/rendering/metal/layout/SplatProjection.metalh:6-141
// and .../metal/cull/SplatVisibility.metal:16-106. The reference compacts with one atomic per
// SIMD group, so its survivor order depends on scheduling; here each 256-splat tile counts
// its survivors, takes its offset by decoupled look-back and writes them in source order, so
// the sorted order downstream is deterministic and equal to a stable sort of (key, source
// position).
//
// Bound by instruction issue and latency (1M SH3 splats, 128 MB: 65 us, 2 TB/s, 22 us at the measured peak,
// 68% of the issue slots; 3M: 201 us, 75%, 60 us of it the span masks at 3840 x 2160), a batch of many waves by instructions (12M splats in 560 us, 476 without the harmonics' arithmetic).
// One splat per thread, four blocks per SM that take tiles in turn and look a tile's place up one tile
// later: 80 -> 65 us (1M), 222 -> 201 (3M), 30 -> 18 (a 0.4M-splat LOD cut), 15.5 -> 8.0 (4k) against 1024-splat
// tiles that waited at once. With two splats per thread 78 us (1M), with three blocks per SM 71, with five 74.
// The quad radius by 8-bit opacity from a table, saturating half conversions and 32 views searched at once
// are the batch's share (604 -> 560 us).
//
// Built with -fmad=false: every product and sum rounds on its own, in the order written.
#include <cuda_runtime.h>

#include "sk_device.cuh"
#include "sk_kernels.h"
#include "sk_launch.cuh"
#include "sk_tiles.cuh"

namespace sk {
namespace {

constexpr float kQuadMinAlpha = 2.0f / 255.0f;
constexpr float kBoundsRadius = 2.5f;
constexpr float kLodBoundsRadius = 5.0f;
constexpr float kMaxPixelRadius = 512.0f;
constexpr float kLowPassVariance = 0.3f;
constexpr float kProjectionFovClamp = 1.3f;
constexpr uint32_t kDepthKeyShift = 11;
constexpr uint32_t kDepthKeyMax = 65535;

constexpr uint32_t kThreads = 256;
constexpr uint32_t kWarps = kThreads / 32;
constexpr uint32_t kTileSplats = kThreads;     // a splat per thread
constexpr uint32_t kResidentBlocks = 148 * 4;  // of either kernel

// Per block, by 8-bit opacity: i / 255 (also the 8-bit colour channels: the same IEEE quotients the
// division gives, computed once per block instead of four times per splat) and the quad radius that
// opacity allows; and the camera's near distance proj[14] / proj[10].
__shared__ float blockUnorm8[256];
__shared__ float blockReach[256];
__shared__ float blockZNear;

__device__ __forceinline__ float quadReach(float alpha, float bound) {
  return fminf(bound, sqrtf(2.0f * lnF32(fmaxf(alpha / kQuadMinAlpha, 1.0f))));
}

// The block's tables (the caller syncs). They depend on nothing that a kernel before wrote.
__device__ __forceinline__ void fillBlockTables() {
  const float unorm = static_cast<float>(threadIdx.x) / 255.0f;
  blockUnorm8[threadIdx.x] = unorm;
  blockReach[threadIdx.x] = quadReach(unorm, kBoundsRadius);
}

// Copies the view's camera and its near distance into shared memory (the caller syncs); the camera is
// in device memory, or (a plain load) in the kernel's parameters.
__device__ __forceinline__ void loadView(const Camera* __restrict__ camera, Camera* cam) {
  loadCamera(camera, cam);
  if (threadIdx.x == kThreads - 1) blockZNear = __ldg(&camera->proj[14]) / __ldg(&camera->proj[10]);
}
__device__ __forceinline__ void copyView(const Camera& camera, Camera* cam) {
  if (threadIdx.x < sizeof(Camera) / 4)
    reinterpret_cast<uint32_t*>(cam)[threadIdx.x] = reinterpret_cast<const uint32_t*>(&camera)[threadIdx.x];
  if (threadIdx.x == kThreads - 1) blockZNear = camera.proj[14] / camera.proj[10];
}

__device__ __forceinline__ void mulPoint(const float* m, float x, float y, float z, float w,
                                         float* o) {
#pragma unroll
  for (int r = 0; r < 4; ++r) o[r] = ((m[r] * x + m[4 + r] * y) + m[8 + r] * z) + m[12 + r] * w;
}

template <int D>
struct ShWords {
  static constexpr uint32_t kWords = shDeviceStride(D);
  uint32_t w[kWords > 0 ? kWords : 1];
  __device__ __forceinline__ void load(const uint32_t* sh, uint32_t index, uint32_t stride) {
    if constexpr (kWords > 0) {
      const uint4* p = reinterpret_cast<const uint4*>(sh + static_cast<size_t>(index) * stride);
#pragma unroll
      for (uint32_t i = 0; i < kWords / 4; ++i) {
        const uint4 v = __ldg(p + i);
        w[i * 4 + 0] = v.x, w[i * 4 + 1] = v.y, w[i * 4 + 2] = v.z, w[i * 4 + 3] = v.w;
      }
    }
  }
  __device__ __forceinline__ float at(uint32_t k, uint32_t ch) const {
    const uint32_t h = k * 3u + ch;
    return (h & 1u) ? highHalf(w[h >> 1]) : lowHalf(w[h >> 1]);
  }
};

// SplatProjection.metalh:50-76, summed in the order the oracle writes.
template <int D>
__device__ __forceinline__ void shColor(const ShWords<D>& s, float x, float y, float z,
                                        float* rgb) {
  const float C1 = 0.4886025119f;
  const float b0 = (-C1) * y, b1 = C1 * z, b2 = C1 * x;
  float q3 = 0, q4 = 0, q5 = 0, q6 = 0, q7 = 0;
  float q8 = 0, q9 = 0, q10 = 0, q11 = 0, q12 = 0, q13 = 0, q14 = 0;
  if constexpr (D >= 2) {
    const float xx = x * x, yy = y * y, zz = z * z, xy = x * y, yz = y * z, xz = x * z;
    q3 = 1.0925484306f * xy;
    q4 = -1.0925484306f * yz;
    q5 = 0.3153915653f * (((2.0f * zz) - xx) - yy);
    q6 = -1.0925484306f * xz;
    q7 = 0.5462742153f * (xx - yy);
    if constexpr (D >= 3) {
      q8 = (-0.5900435899f * y) * ((3.0f * xx) - yy);
      q9 = (2.8906114426f * xy) * z;
      q10 = (-0.4570457995f * y) * (((4.0f * zz) - xx) - yy);
      q11 = (0.3731763326f * z) * (((2.0f * zz) - (3.0f * xx)) - (3.0f * yy));
      q12 = (-0.4570457995f * x) * (((4.0f * zz) - xx) - yy);
      q13 = (1.4453057213f * z) * (xx - yy);
      q14 = (-0.5900435899f * x) * (xx - (3.0f * yy));
    }
  }
#pragma unroll
  for (uint32_t ch = 0; ch < 3; ++ch) {
    float c = (b0 * s.at(0, ch) + b1 * s.at(1, ch)) - b2 * s.at(2, ch);
    if constexpr (D >= 2) {
      const float s2 =
          (((q3 * s.at(3, ch) + q4 * s.at(4, ch)) + q5 * s.at(5, ch)) + q6 * s.at(6, ch)) +
          q7 * s.at(7, ch);
      c = c + s2;
      if constexpr (D >= 3) {
        const float s3 = (((((q8 * s.at(8, ch) + q9 * s.at(9, ch)) + q10 * s.at(10, ch)) +
                            q11 * s.at(11, ch)) +
                           q12 * s.at(12, ch)) +
                          q13 * s.at(13, ch)) +
                         q14 * s.at(14, ch);
        c = c + s3;
      }
    }
    rgb[ch] = c;
  }
}

// SplatProjection.metalh:78-141 and SplatVisibility.metal:86-92. Writes the 8 words of a
// Projected record and the depth key; returns whether the splat survives.
template <int D, bool kKey16>
__device__ __forceinline__ bool projectSplat(const Camera& cam, const uint4 lo, const uint4 hi,
                                             uint32_t index, const uint32_t* sh, uint32_t shStride,
                                             uint32_t& key, uint32_t* out) {
  const float px = asF(lo.x), py = asF(lo.y), pz = asF(lo.z);
  const uint32_t rgba8 = lo.w;
  const uint32_t cov0 = hi.x, cov1 = hi.y, cov2 = hi.z, lodAlpha = hi.w;
  if (!(cam.reveal[0] - py >= 0.0f)) return false;
  const float ca = blockUnorm8[rgba8 >> 24];
  const float alpha = lodAlpha != 0u ? asF(lodAlpha) : ca;
  if (alpha < kQuadMinAlpha) return false;

  float v[4];
  mulPoint(cam.view, px, py, pz, 1.0f, v);
  if (v[2] >= 0.0f) return false;
  float clip[4];
  mulPoint(cam.proj, v[0], v[1], v[2], v[3], clip);
  if (clip[2] < 0.0f || clip[2] > clip[3]) return false;
  if (clip[3] <= blockZNear) return false;

  // projectCovariance (SplatProjection.metalh:6-24)
  const float vz = v[2];
  const float invZ = 1.0f / vz;
  const float invZ2 = invZ * invZ;
  const float limX = kProjectionFovClamp * cam.tanHalfFov[0];
  const float limY = kProjectionFovClamp * cam.tanHalfFov[1];
  const float vx = fminf(fmaxf(v[0] * invZ, -limX), limX) * vz;
  const float vy = fminf(fmaxf(v[1] * invZ, -limY), limY) * vz;
  const float fx = cam.focal[0], fy = cam.focal[1];
  const float j00 = fx * invZ;
  const float j11 = fy * invZ;
  const float j02 = ((-fx) * vx) * invZ2;
  const float j12 = ((-fy) * vy) * invZ2;
  float t0[3], t1[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    t0[c] = j00 * cam.view[c * 4 + 0] + j02 * cam.view[c * 4 + 2];
    t1[c] = j11 * cam.view[c * 4 + 1] + j12 * cam.view[c * 4 + 2];
  }
  const float xx = lowHalf(cov0), xy = highHalf(cov0), xz = lowHalf(cov1);
  const float yy = highHalf(cov1), yz = lowHalf(cov2), zz = highHalf(cov2);
  const float V[3][3] = {{xx, xy, xz}, {xy, yy, yz}, {xz, yz, zz}};
  float m0[3], m1[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    m0[c] = (t0[0] * V[0][c] + t0[1] * V[1][c]) + t0[2] * V[2][c];
    m1[c] = (t1[0] * V[0][c] + t1[1] * V[1][c]) + t1[2] * V[2][c];
  }
  const float ca2 = ((m0[0] * t0[0] + m0[1] * t0[1]) + m0[2] * t0[2]) + kLowPassVariance;
  const float cb2 = (m1[0] * t0[0] + m1[1] * t0[1]) + m1[2] * t0[2];
  const float cd2 = ((m1[0] * t1[0] + m1[1] * t1[1]) + m1[2] * t1[2]) + kLowPassVariance;

  // ellipseAxes (SplatProjection.metalh:26-37)
  const float det = ca2 * cd2 - cb2 * cb2;
  const float mean = 0.5f * (ca2 + cd2);
  const float dist = fmaxf(0.1f, sqrtf(fmaxf(mean * mean - det, 0.0f)));
  const float lambda1 = mean + dist;
  const float lambda2 = mean - dist;
  float e1x, e1y;
  if (cb2 == 0.0f) {
    e1x = (ca2 > cd2) ? 1.0f : 0.0f;
    e1y = (ca2 > cd2) ? 0.0f : 1.0f;
  } else {
    const float nx = cb2, ny = cd2 - lambda2;
    const float len = sqrtf(nx * nx + ny * ny);
    e1x = nx / len;
    e1y = ny / len;
  }
  const float s1 = sqrtf(lambda1);
  const float s2 = sqrtf(fmaxf(lambda2, 0.0f));
  const float a1x = e1x * s1, a1y = e1y * s1;
  const float a2x = e1y * s2, a2y = (-e1x) * s2;

  float radius = lodAlpha != 0u ? quadReach(alpha, kLodBoundsRadius) : blockReach[rgba8 >> 24];
  const float sigmaPixels = sqrtf(fmaxf(a1x * a1x + a1y * a1y, a2x * a2x + a2y * a2y));
  radius = fminf(radius, kMaxPixelRadius / fmaxf(sigmaPixels, 1e-6f));

  const uint32_t axis1 = packHalf2(a1x, a1y);
  const uint32_t axis2 = packHalf2(a2x, a2y);
  const float extX = radius * (fabsf(lowHalf(axis1)) + fabsf(lowHalf(axis2)));
  const float extY = radius * (fabsf(highHalf(axis1)) + fabsf(highHalf(axis2)));
  const float marginX = (((extX + 0.5f) * 2.0f) * clip[3]) / cam.screenSize[0];
  const float marginY = (((extY + 0.5f) * 2.0f) * clip[3]) / cam.screenSize[1];
  if (fabsf(clip[0]) > clip[3] + marginX || fabsf(clip[1]) > clip[3] + marginY) return false;

  const float halfDifference = 0.5f * (ca2 - cd2);
  const float sourceVariance =
      (0.5f * (ca2 + cd2) + sqrtf(fmaxf(halfDifference * halfDifference + cb2 * cb2, 0.0f))) -
      kLowPassVariance;
  if (!(sqrtf(fmaxf(sourceVariance, 0.0f)) * radius >= cam.minPixelRadius)) return false;

  const float depth = -v[2];
  if (!isfinite(depth)) return false;

  float rgb[3] = {blockUnorm8[rgba8 & 0xffu], blockUnorm8[(rgba8 >> 8) & 0xffu],
                  blockUnorm8[(rgba8 >> 16) & 0xffu]};
  if constexpr (D >= 1) {
    ShWords<D> words;
    words.load(sh, index, shStride);
    const float dx = px - cam.cameraPosition[0];
    const float dy = py - cam.cameraPosition[1];
    const float dz = pz - cam.cameraPosition[2];
    const float len = sqrtf((dx * dx + dy * dy) + dz * dz);
    float c[3];
    shColor<D>(words, dx / len, dy / len, dz / len, c);
#pragma unroll
    for (int j = 0; j < 3; ++j) rgb[j] = fmaxf(rgb[j] + c[j], 0.0f);
  }

  if constexpr (kKey16) {
    const float zNear = blockZNear;
    const uint32_t steps = asU(fmaxf(depth, zNear)) - asU(zNear);
    key = min(steps >> kDepthKeyShift, kDepthKeyMax);
  } else {
    key = asU(depth);
  }
  out[0] = asU(clip[0] / clip[3]);
  out[1] = asU(clip[1] / clip[3]);
  out[2] = axis1;
  out[3] = axis2;
  out[4] = packHalf2(rgb[0], rgb[1]);
  out[5] = packHalf2(rgb[2], alpha);
  out[6] = asU(radius);
  out[7] = index;
  return true;
}

// SplatVisibility.metal:69-84: a labelled part's tint, brightness and opacity applied to the
// packed colours, in the same rounded steps as the host; false when the opacity drops the splat.
// A label without a state, or a state without a palette entry, draws unstyled.
__device__ __forceinline__ bool styleRecord(const PartLabels& parts, uint32_t index, uint32_t* rec) {
  const uint32_t label = parts.labels[index];
  if (label >= parts.stateCount) return true;
  const uint32_t state = __ldg(parts.states + label);
  if (state >= kPartStyles) return true;
  const PartStyle st = parts.palette[state];
  if (!(st.tintAmount != 0.0f || st.brightness != 1.0f || st.opacity != 1.0f)) return true;
  const float r = lowHalf(rec[4]), g = highHalf(rec[4]), b = lowHalf(rec[5]), a = highHalf(rec[5]);
  const float r2 = (r + (st.tint[0] - r) * st.tintAmount) * st.brightness;
  const float g2 = (g + (st.tint[1] - g) * st.tintAmount) * st.brightness;
  const float b2 = (b + (st.tint[2] - b) * st.tintAmount) * st.brightness;
  const float alpha = a * st.opacity;
  rec[4] = packHalf2(r2, g2);
  rec[5] = packHalf2(b2, alpha);
  return alpha >= kQuadMinAlpha;
}

// SplatProjection.metalh:177-189 for an encoded-space target: splats below the reveal level
// within `band` of it glow toward the reveal tint and brighten.
__device__ __forceinline__ void revealGlow(const Camera& cam, float height, uint32_t* rec) {
  if (!(cam.reveal[1] > 0.0f)) return;
  float glow = fminf(fmaxf(1.0f - (cam.reveal[0] - height) / cam.reveal[1], 0.0f), 1.0f);
  glow = glow * glow;
  if (!(glow > 0.0f)) return;
  const float r = lowHalf(rec[4]), g = highHalf(rec[4]), b = lowHalf(rec[5]), a = highHalf(rec[5]);
  const float t = cam.reveal[2] * glow, boost = 1.0f + cam.reveal[3] * glow;
  const float r2 = (r + (cam.revealTint[0] - r) * t) * boost;
  const float g2 = (g + (cam.revealTint[1] - g) * t) * boost;
  const float b2 = (b + (cam.revealTint[2] - b) * t) * boost;
  rec[4] = packHalf2(r2, g2);
  rec[5] = packHalf2(b2, a);
}

__device__ __forceinline__ uint32_t sourceIndex(const VisibilityArgs& a, uint32_t t) {
  // SplatVisibility.metal:30-37: the range whose start is the last one <= t.
  if (a.rangeCount <= kInlineRanges) {
    uint32_t shift = a.inlineShift[0];
    for (uint32_t i = 1; i < a.rangeCount; ++i)
      if (a.inlineStart[i] <= t) shift = a.inlineShift[i];
    return t + shift;
  }
  uint32_t lo = 0, hi = a.rangeCount;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) / 2;
    if (a.rangeStarts[mid] <= t) lo = mid; else hi = mid;
  }
  return a.ranges[lo].offset + (t - a.rangeStarts[lo]);
}

// One tile in shared memory: survivors staged at their source slot, then compacted.
struct TileSmem {
  uint4 rec[kTileSplats * 2];    // projected records by source slot
  uint32_t key[kTileSplats];     // depth keys by source slot
  uint16_t slotOf[kTileSplats];  // survivor k of the tile -> its source slot
  uint32_t survivors[kWarps];    // per warp: a bit per lane
};

// A block works on two tiles: one whose survivors wait for their place in the output, and the next one,
// projected meanwhile.
struct VisibilitySmem {
  TileSmem tile[2];
  uint32_t next;      // the tile after the one being projected
  uint32_t tileBase;  // survivors before the waiting tile
};

// Projects one tile into shared memory, a record per thread: survivors' keys and records at their source
// slot, and per warp the mask of survivors. Part styles (when labels are given) and the reveal glow are
// applied to each survivor's record after its projection. index is this thread's record, 0xffffffff past
// the end. keyHigh is or-ed into every key (the view id of a batch, above a 16-bit key).
template <int D, bool kKey16>
__device__ __forceinline__ void projectTile(TileSmem& s, const Camera& cam, const GpuSplat* __restrict__ splats,
                                            const uint32_t* __restrict__ sh, uint32_t shStride,
                                            const PartLabels& parts, uint32_t index, uint32_t keyHigh) {
  bool visible = false;
  if (index != 0xffffffffu) {
    const uint4* p = reinterpret_cast<const uint4*>(splats + index);
    const uint4 lo = __ldg(p), hi = __ldg(p + 1);
    uint32_t key, rec[8];
    visible = projectSplat<D, kKey16>(cam, lo, hi, index, sh, shStride, key, rec);
    if (visible && parts.labels) visible = styleRecord(parts, index, rec);
    if (visible) revealGlow(cam, asF(lo.y), rec);
    if (visible) {
      const uint32_t slot = threadIdx.x;
      s.key[slot] = key | keyHigh;
      s.rec[2 * slot] = make_uint4(rec[0], rec[1], rec[2], rec[3]);
      s.rec[2 * slot + 1] = make_uint4(rec[4], rec[5], rec[6], rec[7]);
    }
  }
  const uint32_t mask = __ballot_sync(0xffffffffu, visible);
  if (laneId() == 0) s.survivors[threadIdx.x >> 5] = mask;
}

// A block's tiles, taken in start order until none is left. Survivors are compacted in source order: a
// tile's place follows from the counts of the tiles before it by decoupled look-back over
// out.status[0 .. tile]. A tile's count is published as soon as it is projected, but its place is looked up
// only after the block has projected its next tile, when the tiles before it have long published theirs
// (looked up at once, a third of the warps' time went by at the barriers behind it: tiles that start
// together end together). The source names the tiles: enter (all threads, no barrier) loads tile's view for
// buffer b, project projects it, width/height/binsX/binsY are b's target, finish takes its place and count.
// With digitPasses > 0 each survivor key's 8-bit digits are counted into digits[pass][digit].
struct VisibilityOut {
  uint32_t* keys;
  Projected* projected;
  uint4* spans;
  uint64_t* status;
  uint32_t* counters;
  uint32_t epoch;
  uint32_t* error;
};

template <typename Source>
__device__ __forceinline__ void runTiles(VisibilitySmem& s, Source& source, const VisibilityOut& out,
                                         uint32_t tile, uint32_t tiles, uint32_t (*digits)[256],
                                         uint32_t digitPasses) {
  const uint32_t warp = threadIdx.x >> 5, lane = laneId();
  constexpr uint32_t kNone = 0xffffffffu;
  uint32_t waiting = kNone, waitingCount = 0;
  for (uint32_t b = 0; tile < tiles || waiting != kNone; b ^= 1u) {
    const bool have = tile < tiles;
    TileSmem& t = s.tile[b];
    const TileSmem& w = s.tile[b ^ 1u];
    if (have) source.project(t, tile, b);
    if (threadIdx.x == 0) s.next = have ? atomicAdd(&out.counters[0], 1u) : kNone;
    __syncthreads();
    uint32_t count = 0;
    if (have) {
      uint32_t pos = 0;
#pragma unroll
      for (uint32_t v = 0; v < kWarps; ++v) {
        if (v == warp) pos = count;
        count += __popc(t.survivors[v]);
      }
      if (threadIdx.x == 0)
        storeStatus(out.status + tile, makeStatus(out.epoch, tile == 0 ? kFlagPrefix : kFlagAggregate, count));
      const uint32_t mask = t.survivors[warp];
      if (mask & (1u << lane)) t.slotOf[pos + __popc(mask & lanemaskLt())] = static_cast<uint16_t>(threadIdx.x);
    }
    uint4 span = make_uint4(0, 0, 0, 0);
    const uint32_t k = threadIdx.x;
    if (waiting != kNone) {
      if (warp == 0) {
        uint32_t before = 0;
        if (waiting != 0) {
          before = warpLookback(out.status, waiting, out.epoch, out.error);
          if (lane == 0) storeStatus(out.status + waiting, makeStatus(out.epoch, kFlagPrefix, before + waitingCount));
        }
        if (lane == 0) s.tileBase = before;
      }
      if (k < waitingCount) {
        const uint32_t slot = w.slotOf[k];
        span = tileSpan(w.rec[2 * slot], w.rec[2 * slot + 1], source.width(b ^ 1u), source.height(b ^ 1u),
                        source.binsX(b ^ 1u), source.binsY(b ^ 1u));
        const uint32_t key = w.key[slot];
        for (uint32_t p = 0; p < digitPasses; ++p) atomicAdd(&digits[p][(key >> (8 * p)) & 0xffu], 1u);
      }
    }
    __syncthreads();
    if (waiting != kNone) {
      const uint32_t base = s.tileBase;
      if (k < waitingCount) {
        const uint32_t slot = w.slotOf[k];
        out.keys[base + k] = w.key[slot];
        uint4* o = reinterpret_cast<uint4*>(out.projected + base + k);
        o[0] = w.rec[2 * slot];
        o[1] = w.rec[2 * slot + 1];
        out.spans[base + k] = span;
      }
      if (threadIdx.x == 0) source.finish(waiting, b ^ 1u, base, waitingCount);
    }
    waiting = have ? tile : kNone;
    waitingCount = count;
    tile = s.next;
    __syncthreads();  // the waiting tile's buffer, s.next and s.tileBase are free
    if (tile < tiles) {
      source.enter(tile, b ^ 1u);
      if constexpr (Source::kEnters) __syncthreads();
    }
  }
}

// A frame's tiles: the records of its ranges, or of a LOD cut, on one target.
template <int D, bool kKey16, bool kIndexed>
struct FrameSource {
  static constexpr bool kEnters = false;
  const VisibilityArgs& a;
  const Camera& cam;
  uint32_t total, tiles;

  // Asks for this thread's record of the tile (and its harmonics) ahead of their loads.
  __device__ __forceinline__ void enter(uint32_t tile, uint32_t) {
    const uint32_t at = tile * kTileSplats + threadIdx.x;
    if (at >= total || (!kIndexed && a.rangeCount > kInlineRanges)) return;
    const uint32_t index = kIndexed ? a.indices[at] : sourceIndex(a, at);
    if (index >= a.worldCount) return;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(a.splats + index));
    if (D > 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.sh + size_t{index} * a.shStride));
  }
  __device__ __forceinline__ void project(TileSmem& t, uint32_t tile, uint32_t) {
    const uint32_t at = tile * kTileSplats + threadIdx.x;
    uint32_t index = 0xffffffffu;
    if (at < total) {
      index = kIndexed ? a.indices[at] : sourceIndex(a, at);
      if (index >= a.worldCount) {
        atomicOr(a.error, SK_DEVERR_BOUNDS);
        index = 0xffffffffu;
      }
    }
    projectTile<D, kKey16>(t, cam, a.splats, a.sh, a.shStride, a.parts, index, 0u);
  }
  __device__ __forceinline__ float width(uint32_t) const { return cam.screenSize[0]; }
  __device__ __forceinline__ float height(uint32_t) const { return cam.screenSize[1]; }
  __device__ __forceinline__ uint32_t binsX(uint32_t) const { return a.tilesX; }
  __device__ __forceinline__ uint32_t binsY(uint32_t) const { return a.tilesY; }
  __device__ __forceinline__ void finish(uint32_t tile, uint32_t, uint32_t before, uint32_t count) {
    if (tile == tiles - 1) *a.visibleCount = before + count;
  }
};

template <int D, bool kKey16, bool kIndexed>
__global__ void __launch_bounds__(kThreads, 4)
    visibilityKernel(const __grid_constant__ VisibilityArgs a) {
  __shared__ VisibilitySmem s;
  __shared__ Camera cam;
  __shared__ uint32_t digits[4][256];
  // Before the wait for the kernel before this one: what depends on nothing it writes (the tile counter
  // is this launch's alone; its last block left it at zero in an earlier, finished launch).
  fillBlockTables();
  for (uint32_t p = 0; p < a.sortPasses; ++p) digits[p][threadIdx.x] = 0;
  const uint32_t tile = takeTile(a.counters);
  if (!kIndexed) copyView(a.camera, &cam);
  chainedKernelStart();
  if (kIndexed) loadView(a.cameraInMemory, &cam);
  __syncthreads();
  const uint32_t total = kIndexed ? min(*a.indexCount, a.total) : a.total;
  const uint32_t tiles = (total + kTileSplats - 1) / kTileSplats;
  FrameSource<D, kKey16, kIndexed> source{a, cam, total, tiles};
  runTiles(s, source, VisibilityOut{a.keys, a.projected, a.spans, a.status, a.counters, a.epoch, a.error}, tile, tiles,
           digits, a.sortPasses);
  if (tiles == 0 && tile == 0 && threadIdx.x == 0) *a.visibleCount = 0;
  if (a.sortPasses) {
    __syncthreads();
    for (uint32_t p = 0; p < a.sortPasses; ++p) {
      const uint32_t v = digits[p][threadIdx.x];
      if (v) atomicAdd(&a.sortAccum[p * 256 + threadIdx.x], v);
    }
    if (finishTile(a.counters)) finishDigitHistograms(a.sortAccum, a.sortBases, a.sortPasses);
    return;
  }
  finishTile(a.counters);
}

// A batch of views in one launch. Work item i is a 256-record chunk of one view's range (or of
// a LOD view's cut, in emission order: the chunks past the cut's length hold nothing); items
// are numbered view by view, so one look-back chain over all items places every view's
// survivors contiguously, in (view, source) order, and the first item of each view records
// where that view starts. Keys carry the view id above the 16-bit depth key, so one stable
// sort orders all views at once.
template <int D>
struct BatchSource {
  static constexpr bool kEnters = true;
  const BatchVisibilityArgs& a;
  Camera& cam;
  BatchView* view;     // per buffer
  uint32_t* viewIndex; // per buffer

  __device__ __forceinline__ void enter(uint32_t item, uint32_t b) {
    // the last view whose first item is <= item
    const uint32_t v = lastAtOrBelow(a.viewCount, item, [&](uint32_t i) { return __ldg(&a.views[i].itemStart); });
    loadView(a.cameras + v, &cam);
    if (threadIdx.x < sizeof(BatchView) / 4)
      reinterpret_cast<uint32_t*>(view + b)[threadIdx.x] =
          __ldg(reinterpret_cast<const uint32_t*>(a.views + v) + threadIdx.x);
    if (threadIdx.x == 0) viewIndex[b] = v;
  }
  __device__ __forceinline__ void project(TileSmem& t, uint32_t item, uint32_t b) {
    const BatchView& w = view[b];
    const uint32_t at = (item - w.itemStart) * kTileSplats + threadIdx.x;
    // a LOD view draws its cut (written by this stream's selection before this kernel)
    const uint32_t drawn = w.indices ? min(w.count, *w.indexCount) : w.count;
    uint32_t index = 0xffffffffu;
    if (at < drawn) {
      index = w.indices ? w.indices[at] : w.offset + at;
      if (w.indices && index >= w.worldCount) {
        atomicOr(a.error, SK_DEVERR_BOUNDS);
        index = 0xffffffffu;
      }
    }
    projectTile<D, true>(t, cam, w.splats, w.sh, w.shStride, PartLabels{}, index, viewIndex[b] << 16);
  }
  __device__ __forceinline__ float width(uint32_t b) const { return static_cast<float>(view[b].width); }
  __device__ __forceinline__ float height(uint32_t b) const { return static_cast<float>(view[b].height); }
  __device__ __forceinline__ uint32_t binsX(uint32_t b) const { return view[b].binsX; }
  __device__ __forceinline__ uint32_t binsY(uint32_t b) const { return view[b].binsY; }
  __device__ __forceinline__ void finish(uint32_t item, uint32_t b, uint32_t before, uint32_t count) {
    if (item == view[b].itemStart) a.viewFirst[viewIndex[b]] = before;
    if (item == a.items - 1) {
      a.viewFirst[a.viewCount] = before + count;
      *a.visibleCount = before + count;
    }
  }
};

template <int D>
__global__ void __launch_bounds__(kThreads, 4)
    visibilityBatchKernel(const __grid_constant__ BatchVisibilityArgs a) {
  __shared__ VisibilitySmem s;
  __shared__ Camera cam;
  __shared__ BatchView view[2];
  __shared__ uint32_t viewIndex[2];
  fillBlockTables();
  const uint32_t item = takeTile(a.counters);
  chainedKernelStart();
  BatchSource<D> source{a, cam, view, viewIndex};
  if (item < a.items) source.enter(item, 0);
  __syncthreads();
  runTiles(s, source, VisibilityOut{a.keys, a.projected, a.spans, a.status, a.counters, a.epoch, a.error}, item, a.items,
           nullptr, 0u);
  finishTile(a.counters);
}

template <int D, bool kKey16, bool kIndexed>
void launchOne(const VisibilityArgs& a, cudaStream_t stream) {
  const uint32_t tiles = max(1u, (a.total + kTileSplats - 1) / kTileSplats);
  launchChained(visibilityKernel<D, kKey16, kIndexed>, min(tiles, kResidentBlocks), kThreads, stream, a);
}

template <int D>
void launchDegree(const VisibilityArgs& a, bool key16, bool indexed, cudaStream_t stream) {
  if (key16) {
    if (indexed) launchOne<D, true, true>(a, stream);
    else launchOne<D, true, false>(a, stream);
  } else {
    if (indexed) launchOne<D, false, true>(a, stream);
    else launchOne<D, false, false>(a, stream);
  }
}

}  // namespace

uint32_t visibilityTileSplats() { return kTileSplats; }

cudaError_t launchVisibilityBatch(const BatchVisibilityArgs& args, int shDegree,
                                  cudaStream_t stream) {
  if (args.items == 0 || args.viewCount == 0) return cudaSuccess;
  const uint32_t blocks = min(args.items, kResidentBlocks);
  switch (shDegree) {
    case 0: launchChained(visibilityBatchKernel<0>, blocks, kThreads, stream, args); break;
    case 1: launchChained(visibilityBatchKernel<1>, blocks, kThreads, stream, args); break;
    case 2: launchChained(visibilityBatchKernel<2>, blocks, kThreads, stream, args); break;
    default: launchChained(visibilityBatchKernel<3>, blocks, kThreads, stream, args); break;
  }
  return cudaGetLastError();
}

cudaError_t launchVisibility(const VisibilityArgs& args, int shDegree,
                             bool key16, bool indexed, cudaStream_t stream) {
  switch (shDegree) {
    case 0: launchDegree<0>(args, key16, indexed, stream); break;
    case 1: launchDegree<1>(args, key16, indexed, stream); break;
    case 2: launchDegree<2>(args, key16, indexed, stream); break;
    default: launchDegree<3>(args, key16, indexed, stream); break;
  }
  return cudaGetLastError();
}

}  // namespace sk
