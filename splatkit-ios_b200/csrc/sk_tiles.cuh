// Which binning cells (kBinSize pixels square) a projected splat's quad touches.
//
// The quad is the parallelogram c + s a1 + t a2, |s|, |t| <= radius, in pixel units (y up), with
// the half-rounded axes the compositor inverts. Its tiles are those of its pixel box whose
// square it overlaps by the separating-axis test (x, y and the normals of a1 and a2). The cell
// square is the pixel area, half a pixel beyond every pixel centre, so the test can only keep
// too many cells, never drop one the compositor would cover. ("Tile" below means a cell.)
//
// A span packs the result in 16 bytes: (x0 | y0 << 16, width | height << 16, mask lo, mask hi),
// bit k of the mask standing for box tile (x0 + k % width, y0 + k / width). A box of more than
// 64 tiles keeps all of them (its mask is unused); a width of 0 means no tile.
#pragma once
#include "sk_device.cuh"

namespace sk {

struct Quad {
  float cx, cy, a1x, a1y, a2x, a2y, r;
};

__device__ __forceinline__ Quad quadOf(const uint4 lo, const uint4 hi, float halfW, float halfH) {
  Quad q;
  q.cx = (asF(lo.x) + 1.0f) * halfW;
  q.cy = (asF(lo.y) + 1.0f) * halfH;
  q.a1x = lowHalf(lo.z), q.a1y = highHalf(lo.z);
  q.a2x = lowHalf(lo.w), q.a2y = highHalf(lo.w);
  q.r = asF(hi.z);
  return q;
}

// The span of one projected record (two uint4 words) on a width x height target.
__device__ __forceinline__ uint4 tileSpan(const uint4 lo, const uint4 hi, float width, float height,
                                          uint32_t tilesX, uint32_t tilesY) {
  const Quad q = quadOf(lo, hi, 0.5f * width, 0.5f * height);
  const float ex = q.r * (fabsf(q.a1x) + fabsf(q.a2x)) + 1.0f;
  const float ey = q.r * (fabsf(q.a1y) + fabsf(q.a2y)) + 1.0f;
  if (!(isfinite(q.cx) && isfinite(q.cy) && isfinite(ex) && isfinite(ey) && q.r >= 0.0f))
    return make_uint4(0, 0, 0, 0);
  const float xa = floorf(q.cx - ex), xb = ceilf(q.cx + ex);
  const float ya = floorf(q.cy - ey), yb = ceilf(q.cy + ey);
  if (xb < 0.0f || xa >= width || yb < 0.0f || ya >= height) return make_uint4(0, 0, 0, 0);
  // columns [c0, c1]; rows from the y-up box: row = H - y_up - 0.5
  const uint32_t c0 = static_cast<uint32_t>(fmaxf(xa, 0.0f));
  const uint32_t c1 = static_cast<uint32_t>(fminf(xb, width - 1.0f));
  const uint32_t r0 = static_cast<uint32_t>(fmaxf(height - yb - 1.0f, 0.0f));
  const uint32_t r1 = static_cast<uint32_t>(fminf(fmaxf(height - ya, 0.0f), height - 1.0f));
  const uint32_t x0 = c0 / kBinSize, x1 = min(c1 / kBinSize, tilesX - 1);
  const uint32_t y0 = r0 / kBinSize, y1 = min(r1 / kBinSize, tilesY - 1);
  if (x0 > x1 || y0 > y1) return make_uint4(0, 0, 0, 0);
  const uint32_t w = x1 - x0 + 1, area = w * (y1 - y0 + 1);
  uint64_t mask = 0;
  if (area <= 64) {
    // Separating-axis test of the quad against each cell's pixel square (y up), the box's cells
    // row by row (bit k = cell (x0 + k % w, y0 + k / w)); the quad's extents along x, y and the
    // normals of a1 and a2 (along a normal of a1 the extent comes from t a2 only) are taken once.
    const float half = 0.5f * static_cast<float>(kBinSize);
    const float exq = q.r * (fabsf(q.a1x) + fabsf(q.a2x)) + half;
    const float eyq = q.r * (fabsf(q.a1y) + fabsf(q.a2y)) + half;
    const float n1x = -q.a1y, n1y = q.a1x, n2x = -q.a2y, n2y = q.a2x;
    const float e1 = q.r * fabsf(q.a2x * n1x + q.a2y * n1y) + half * (fabsf(n1x) + fabsf(n1y));
    const float e2 = q.r * fabsf(q.a1x * n2x + q.a1y * n2y) + half * (fabsf(n2x) + fabsf(n2y));
    uint32_t k = 0;
    for (uint32_t ty = y0; ty <= y1; ++ty) {
      const float ry = height - (static_cast<float>(ty * kBinSize) + half);
      const float dy = ry - q.cy;
      const bool rowIn = !(fabsf(dy) > eyq);
      for (uint32_t tx = x0; tx <= x1; ++tx, ++k) {
        const float rx = static_cast<float>(tx * kBinSize) + half;
        const float dx = rx - q.cx;
        const bool hit = rowIn && !(fabsf(dx) > exq) && !(fabsf(dx * n1x + dy * n1y) > e1) &&
                         !(fabsf(dx * n2x + dy * n2y) > e2);
        if (hit) mask |= 1ull << k;
      }
    }
    if (mask == 0) return make_uint4(0, 0, 0, 0);
  }
  return make_uint4(x0 | (y0 << 16), w | ((y1 - y0 + 1) << 16), static_cast<uint32_t>(mask),
                    static_cast<uint32_t>(mask >> 32));
}

// Tiles of a span's box.
__device__ __forceinline__ uint32_t spanArea(const uint4 s) { return (s.y & 0xffffu) * (s.y >> 16); }

// Tiles a span lists.
__device__ __forceinline__ uint32_t spanCount(const uint4 s) {
  const uint32_t area = spanArea(s);
  if (area > 64) return area;
  return static_cast<uint32_t>(__popc(s.z) + __popc(s.w));
}

// Position of the k-th (from 0) set bit of x; x holds more than k set bits. Bisection on halves.
__device__ __forceinline__ uint32_t kthSetBit(uint32_t x, uint32_t k) {
  uint32_t pos = 0;
#pragma unroll
  for (uint32_t width = 16; width > 0; width >>= 1) {
    const uint32_t low = __popc(x & ((1u << width) - 1u));
    if (k >= low) {
      k -= low;
      x >>= width;
      pos += width;
    }
  }
  return pos;
}

// Cell of box position b of a box w cells wide whose first cell is `first`, on a grid tilesX
// cells wide. b / w in float: (b + 1/2) / w lies at least 1/(2w) from an integer, and the fast
// divide errs by at most 2 ulp of the quotient, less than that for b < 2^19 (a box holds at most
// 512 x 512 cells), so truncation gives the quotient.
__device__ __forceinline__ uint32_t boxCell(uint32_t first, uint32_t b, uint32_t w,
                                            uint32_t tilesX) {
  const uint32_t q = static_cast<uint32_t>(
      __fdividef(static_cast<float>(b) + 0.5f, static_cast<float>(w)));
  return first + q * tilesX + (b - q * w);
}

// ---- patches (sk_layout.h) --------------------------------------------------------------
struct PatchBox {
  uint32_t x0, y0, w, h;  // first patch, patches per row and column; w 0: none
};

// The patches of 2^shift cells a side that a span's box touches.
__device__ __forceinline__ PatchBox patchBox(const uint4 s, uint32_t shift) {
  const uint32_t x0 = s.x & 0xffffu, y0 = s.x >> 16, w = s.y & 0xffffu, h = s.y >> 16;
  PatchBox b;
  b.x0 = x0 >> shift;
  b.y0 = y0 >> shift;
  b.w = w ? ((x0 + w - 1) >> shift) - b.x0 + 1 : 0u;
  b.h = w ? ((y0 + h - 1) >> shift) - b.y0 + 1 : 0u;
  return b;
}

// The cells of patch (px, py) a span lists (0 when its box only touches the patch).
__device__ __forceinline__ uint32_t patchMask(const uint4 s, uint32_t px, uint32_t py, uint32_t shift) {
  const uint32_t x0 = s.x & 0xffffu, y0 = s.x >> 16, w = s.y & 0xffffu, h = s.y >> 16;
  const uint32_t cx = px << shift, cy = py << shift, edge = 1u << shift;
  const uint32_t xa = max(x0, cx), xb = min(x0 + w, cx + edge);
  const uint32_t ya = max(y0, cy), yb = min(y0 + h, cy + edge);
  const uint32_t row = (1u << (xb - xa)) - 1u;
  const bool masked = w * h <= 64;
  uint32_t out = 0;
  uint32_t at = (ya - y0) * w + (xa - x0);  // the row's first bit of the box mask
  uint32_t to = ((ya - cy) << shift) + (xa - cx);
  for (uint32_t y = ya; y < yb; ++y, at += w, to += edge) {
    uint32_t bits = row;
    if (masked) bits &= at < 32 ? __funnelshift_r(s.z, s.w, at) : s.w >> (at - 32);
    out |= bits << to;
  }
  return out;
}

}  // namespace sk
