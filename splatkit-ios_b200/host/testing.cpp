// The test hooks of include/splatkit_b200_testing.h: one-shot states the library's own
// paths read (DeviceBuffer::allocate, Context::check, the depth sort's launch arguments), and the raw lists.
#include "../../include/splatkit_b200_testing.h"

#include <algorithm>

#include "context.h"

extern "C" {

void sk_testing_fail_device_allocations(uint32_t count) {
  sk::gTestFailedAllocations.store(count);
  sk::gTestPassedAllocations.store(0);
}

void sk_testing_pass_device_allocations(uint32_t count) { sk::gTestPassedAllocations.store(count); }

sk_status sk_testing_fail_next_check(sk_context* handle, int32_t cuda_error) {
  auto* ctx = reinterpret_cast<sk::Context*>(handle);
  if (!ctx || cuda_error == 0) return SK_E_INVALID;
  ctx->testInjectedError = static_cast<cudaError_t>(cuda_error);
  return SK_OK;
}

sk_status sk_testing_withhold_sort_status(sk_context* handle, uint32_t tile) {
  auto* ctx = reinterpret_cast<sk::Context*>(handle);
  if (!ctx || tile == 0xffffffffu) return SK_E_INVALID;
  ctx->testWithheldTile = tile + 1;
  return SK_OK;
}

void sk_testing_fail_image_step(uint32_t after) { sk::gTestFailedImageStep.store(after + 1); }

sk_status sk_testing_read_patch_lists(sk_context* handle, uint32_t* grid, uint32_t* ranges, uint32_t* values,
                                      uint16_t* masks, uint32_t capacity, uint32_t* count) {
  auto* ctx = reinterpret_cast<sk::Context*>(handle);
  if (!ctx || !grid || !count) return SK_E_INVALID;
  const sk_status st = ctx->finishFrame(true);
  if (st != SK_OK) return st;
  const sk::Context::Slot& slot = ctx->slots[ctx->lastSlot];
  const sk::FrameScratch& f = ctx->scratchOf(ctx->lastSlot);
  if (!slot.direct || ctx->listsPerCell || !f.spansKept) return SK_E_INVALID;
  const sk::PatchGrid g = slot.patches;
  grid[0] = g.shift, grid[1] = g.x, grid[2] = g.y;
  *count = ctx->lastCounters.entries;
  const size_t copy = std::min({*count, capacity, f.instanceCapacity});
  cudaError_t e = cudaSuccess;
  if (ranges) e = cudaMemcpy(ranges, f.ranges.ptr, size_t{g.x} * g.y * 8, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && values && copy)
    e = cudaMemcpy(values, f.instValuesSorted.ptr, copy * 4, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && masks && copy && g.shift)
    e = cudaMemcpy(masks, f.instKeysSorted.ptr, copy * 2, cudaMemcpyDeviceToHost);
  else if (masks)
    std::fill_n(masks, copy, uint16_t{1});
  return ctx->check(e, "patch lists");
}

}  // extern "C"
