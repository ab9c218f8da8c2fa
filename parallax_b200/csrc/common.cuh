// common.cuh -- shared device definitions of the splat training core (sm_100a).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "pxs.h"

namespace pxs {

constexpr int kTile = PXS_TILE;           // logical binning tile, pixels
constexpr int kTilePixels = kTile * kTile;
constexpr float kMaxAlpha = 0.99f;        // SplatRaster.cpp:22
constexpr float kFrustumSlack = 1.3f;     // SplatRaster.cpp:26
constexpr float kShC0 = 0.28209479177387814f;  // GaussianCloud.h:54

// Items per radix-sort block tile; the per-view slot stride is padded to it so
// a sort block never straddles two views.
constexpr int kSortThreads = 256;
constexpr int kSortItemsPerThread = 16;
constexpr int kSortTile = kSortThreads * kSortItemsPerThread;

constexpr uint32_t kCulledKey = 0xFFFFFFFFu;

// Widest image, in tiles, the row-binning kernels stage in shared memory.
constexpr int kMaxTilesX = 2048;
constexpr int kMaxTilesY = 2048;
// Most tiles of a view whose lists are built directly, without tile rows
// (Frame::direct_lists).
constexpr int kMaxDirectTiles = 2048;

// Everything a kernel needs to know about one view of a batch.
struct ViewDesc {
  pxs_camera cam;
  float background[3];
  int32_t sh_degree;         // min(options.sh_degree, cloud sh_degree)
  int32_t tiles_x, tiles_y;
  int32_t tile_offset;       // first global tile id of this view
  int32_t row_offset;        // first global tile-row id of this view
  int64_t pixel_offset;      // first pixel of this view in the image arrays
  float min_alpha;
  float transmittance_cutoff;
  float screen_dilation;
  int32_t loss_tile_offset;  // first CTA of this view in the loss kernel's grid
  int32_t l1_block_offset;   // the same for the loss without SSIM
  int64_t target_offset;     // first pixel of this view's target image
  // the gaussians this view renders: [gauss_offset, gauss_offset + gauss_count)
  // of the parameter arrays; slot v * slot_stride + i holds gaussian
  // gauss_offset + i (one cloud: 0 and N for every view; a batch of several
  // independent scenes: each view's own scene)
  int32_t gauss_offset;
  int32_t gauss_count;
};

// Per-step screen-space gradient accumulators of one (view, gaussian) slot, 12
// floats, 16-byte aligned. With z = dL/dp of a pixel's power p = -1/2 d^T A d
// (0 where the alpha cap flattens it), d its centre less the mean, A the
// splat's conic, o its opacity and (u, w) = A d, the per-splat gradients of
// SplatRaster.cpp:337-342 and 455-470 are
//   dL/dmean  = sum of z (u, w)
//   dL/dcov2d = -A (dL/dA) A = 1/2 sum of z (u, w)^T (u, w)
//   dL/do     = sum of z / o
// Sums of z d^T d, dL/dA, would be multiplied by A afterwards; in an elongated
// splat that cancels all but (minor / major axis)^2 of them and brings up the
// rounding of the FP32 sums, while A d cancels pixel by pixel, before the sum.
struct alignas(16) ScreenGrad {
  float s0;         // sum of z
  float dcov[3];    // sums of z u^2, z u w, z w^2
  float dmean[2];
  float dcolor[3];
  float dmean_abs;  // sum of |dL/dmean| per pixel, the densify statistic
  float touched;  // nonzero when any pixel reached the uncapped-alpha branch
  float pad;
};
static_assert(sizeof(ScreenGrad) == 48, "ScreenGrad layout");

// What a (view, gaussian) slot's projection leaves for binning, compositing and
// its adjoint, which gather slots in depth order: one aligned 32-byte sector, so
// that a gather costs one (as three arrays it cost up to three).
struct alignas(32) SlotGeom {
  float4 conic_op;  // conic (a, b, c), opacity
  float2 xy;        // mean
  uint2 rect;       // tile coordinates x0 | x1 << 16, y0 | y1 << 16
};

// Device views of the per-slot projection outputs.
struct ProjectedSoA {
  SlotGeom* geom;
  float4* color;       // r, g, b, clamp flags (bits in .w)
  uint32_t* depth_key; // float bits of depth; kCulledKey when culled
  float4* debug_cov;   // optional: cov2d (xx, xy, yy), radius
};

__host__ __device__ inline int64_t round_up(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

// Kernel launches issued by this library (host counter, bumped at every
// launch site; a captured graph's count is taken while capturing).
extern int64_t g_kernel_launches;
inline void count_launch() { ++g_kernel_launches; }

#if defined(__CUDACC__)
__device__ inline int warp_id() { return threadIdx.x >> 5; }
__device__ inline int lane_id() { return threadIdx.x & 31; }

__device__ inline unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Inclusive warp scan of a 32-bit integer.
__device__ inline int warp_inclusive_scan(int v) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, v, o);
    if (lane_id() >= o) v += n;
  }
  return v;
}

// Looks up which view of a batch a global tile belongs to (views are few).
__device__ inline int view_of_tile(const ViewDesc* views, int n_views, int tile) {
  int v = 0;
  while (v + 1 < n_views && views[v + 1].tile_offset <= tile) ++v;
  return v;
}
#endif  // __CUDACC__

}  // namespace pxs
