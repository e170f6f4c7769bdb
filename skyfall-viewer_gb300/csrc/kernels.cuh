// Launch interface of the hot-path kernels (kernels.cu).
#pragma once

#include "sky_types.cuh"
#include "sort.cuh"

namespace sky {

void launch_preprocess(const DevBuffers& b, uint32_t n, uint32_t views, cudaStream_t s);
// step: the scan of a step's items, which also writes the sort groups' bounds
// and checks the capacity.  Returns the number of kernels launched.
int launch_scan(const DevBuffers& b, uint32_t n_items, bool step, cudaStream_t s);
uint32_t scan_block_count(uint32_t n_items);
void launch_group_bounds(const DevBuffers& b, cudaStream_t s);
void launch_emit(const DevBuffers& b, uint32_t n, uint32_t views, cudaStream_t s);
void launch_ranges(const DevBuffers& b, uint32_t icap, cudaStream_t s);
// Zeroes the partials the last exact backward left unwritten, for a read-back.
void launch_partials_fill(const DevBuffers& b, uint32_t total, cudaStream_t s);
// Completes flatten (the item of every sorted intersection) for a read-back.
void launch_flatten_fill(const DevBuffers& b, uint32_t total, cudaStream_t s);
// Splat-batch depths of the rasterizers: the forward stages fb splats per
// batch (64, 128 or 256), the 16x16-tile exact backward bb (32, 64 or 128);
// other values select the defaults.  Results do not depend on them.
// Default backward depth for 16x16 tiles (few tiles: 128, k_backward_exact2).
constexpr uint32_t kBwdBatch16 = 64;
// The 16x16 backward's variant for few tiles: where all of them are resident at
// once, at this many blocks per multiprocessor of the device.
constexpr int kFewTileBlocks = 5;
inline bool few_tiles(uint32_t tiles, int multiprocessors) {
  return tiles <= (uint32_t)kFewTileBlocks * (uint32_t)multiprocessors;
}
// count: the pair-counting variants (16x16 tiles at the default depths only;
// other shapes launch the plain kernels and count nothing).  Counting steps of
// few tiles run the 64-deep backward too.
// launch_forward_tiles: tiles [first, first + tiles) alone (no SSIM term).
void launch_forward_tiles(const DevBuffers& b, uint32_t first, uint32_t tiles, uint32_t ts, uint32_t fb,
                          bool count, cudaStream_t s);
void launch_forward(const DevBuffers& b, uint32_t max_tiles, uint32_t ts, uint32_t fb, bool ssim,
                    uint32_t views, uint32_t max_view_pixels, bool count, cudaStream_t s);
// Doubles of b.loss_partials for a step of `tiles` tiles.
size_t loss_partial_count(uint64_t tiles);
void launch_loss_final(const DevBuffers& b, uint32_t max_tiles, cudaStream_t s);
void launch_backward(const DevBuffers& b, uint32_t max_tiles, uint32_t ts, uint32_t bb, bool ref,
                     bool count, cudaStream_t s);
// Training steps of at most kFewViews views in the exact backward mode hand the
// SH part of Adam to a kernel of its own (b.sh_items, 24 bytes per item).  Both
// parts then fit more warps, but that kernel reads every item once more: 1M
// Gaussians, one kernel -> two: 1 view 542 -> 394 us, 4 views 688 -> 568, 6:
// 788 -> 686, 16: 1323 -> 1213; 250k Gaussians: 16 views 340 -> 333, 32: 561 ->
// 576, 64: 996 -> 1060.
constexpr int kFewViews = 16;
// train_exact: a training step (no gradients out) in the exact backward mode.
// Returns the number of kernels launched.
int launch_geom_adam(const DevBuffers& b, uint32_t n, uint32_t views, bool train_exact, cudaStream_t s);
// Exact mode, before launch_geom_adam: per-item sums of the partials.
void launch_item_sums(const DevBuffers& b, uint64_t items, cudaStream_t s);

// Prune / densify / opacity reset (compact.cu).
void launch_prune_flags(const float* params, uint32_t stride, uint32_t n, float min_opacity,
                        float max_scale, const uint8_t* mask, uint32_t* flags, cudaStream_t s);
void launch_compact(const float* src, float* dst, uint32_t src_stride, uint32_t dst_stride,
                    uint32_t planes, uint32_t n, const uint32_t* keep_scan, cudaStream_t s);
void launch_reset_opacity(float* params, uint32_t stride, uint32_t n, float max_logit,
                          cudaStream_t s);

}  // namespace sky
