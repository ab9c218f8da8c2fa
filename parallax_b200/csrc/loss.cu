// loss.cu -- photometric loss L = (1-w) mean|r-t| + w (1 - mean SSIM) and its
// gradient in one kernel.
//
// photometricLoss / meanSsim (SplatRaster.cpp:582-738) run 13 separable
// 11-tap blurs per channel over whole-image planes. Here a CTA marches down a
// strip of one channel, a thread per column, an image row per iteration:
//   * the row of both images goes to shared memory; each thread blurs its
//     column's x, y, x^2, y^2 and x y horizontally from it and adds the results
//     into eleven running vertical sums per plane in registers, of which one is
//     complete: the statistics of the row five above;
//   * from them the SSIM value and its partials there (zero outside the image,
//     as the reference's zero-padded adjoint requires). The reference blurs five
//     partial planes back; by linearity of the blur the three without a pixel
//     factor are summed first, so three planes go the same way, through shared
//     memory horizontally and eleven running sums vertically;
//   * the row ten above is then complete and its gradient is written.
// So nothing is blurred twice along the march and the vertical blurs never leave
// the registers; only the strip's ten columns at either side and the march's
// twenty extra rows are recomputed. Every blur sums in the reference's tap order;
// the scalar totals are accumulated in double.
#include <algorithm>
#include <cstdio>
#include <exception>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "kernels.h"
#include "runtime.h"

namespace pxs {
namespace {

constexpr int kCols = 128;          // threads, and columns of a strip with its halo
constexpr int kStrip = kCols - 20;  // output columns of a strip
constexpr int kPad = 5;             // columns past either end that the blurs read
constexpr int kRing = 16;           // input rows kept: the output row is 11 behind

struct LossSmem {
  float2 in[kRing][kCols + 2 * kPad];  // rendered, target
  float2 p12[2][kCols + 2 * kPad];     // the partials by variance and covariance
  float p0[2][kCols + 2 * kPad];       // the partial without a pixel factor
};

// View v's share of the flat grid starts at its loss_tile_offset: strips across,
// row blocks down, channels fastest (the three read and write the same lines).
// (kL1: at its l1_block_offset, blocks of consecutive values.)
template <bool kL1>
__device__ __forceinline__ int loss_offset(const ViewDesc& v) {
  return kL1 ? v.l1_block_offset : v.loss_tile_offset;
}
template <bool kL1>
__device__ __forceinline__ int loss_view(const ViewDesc* views, int n_views, int block) {
  int lo = 0, hi = n_views - 1;  // the last view whose first block is at or before this one
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (loss_offset<kL1>(views[mid]) <= block) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// A CTA's two sums into its view's totals; the last CTA of the launch to do so
// (counted in sums[2 n_views]) forms the losses:
// loss = (1-w) * l1 + w * (1 - ssim) per view (SplatRaster.cpp:737); the batch
// loss is the mean over views. mode 1 reports mean SSIM instead.
template <int kThreads>
__device__ __forceinline__ void finish_loss(double l1_sum, double ssim_sum, int v,
                                            const ViewDesc* __restrict__ views, int n_views,
                                            const LossParams& lp, double* __restrict__ sums,
                                            float* __restrict__ per_view,
                                            float* __restrict__ total) {
  __shared__ double red[2][kThreads / 32];
  __shared__ int s_last;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    l1_sum += __shfl_xor_sync(0xffffffffu, l1_sum, o);
    ssim_sum += __shfl_xor_sync(0xffffffffu, ssim_sum, o);
  }
  if (lane_id() == 0) {
    red[0][warp_id()] = l1_sum;
    red[1][warp_id()] = ssim_sum;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int k = 0; k < kThreads / 32; ++k) {
      a += red[0][k];
      b += red[1][k];
    }
    atomicAdd(&sums[2 * v + 0], a);
    atomicAdd(&sums[2 * v + 1], b);
    __threadfence();
    unsigned long long* done = reinterpret_cast<unsigned long long*>(sums + 2 * n_views);
    s_last = atomicAdd(done, 1ull) == (unsigned long long)gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last || threadIdx.x >= 32) return;
  __threadfence();
  float mean = 0.f;  // views in order, whichever lane holds them
  for (int v0 = 0; v0 < n_views; v0 += 32) {
    const int k = v0 + lane_id();
    float loss = 0.f;
    if (k < n_views) {
      const double values = 3.0 * (double)views[k].cam.width * (double)views[k].cam.height;
      const double l1_total = __ldcg(&sums[2 * k + 0]), ssim_total = __ldcg(&sums[2 * k + 1]);
      const float ssim = (float)(ssim_total / values);
      if (lp.mode == 1) {
        loss = ssim;
      } else {
        const float l1 = (float)(l1_total / values);
        loss = lp.ssim_weight <= 0.f
                   ? l1
                   : (1.f - lp.ssim_weight) * l1 + lp.ssim_weight * (1.f - ssim);
      }
      if (per_view != nullptr) per_view[k] = loss;
    }
    for (int j = 0; j < min(32, n_views - v0); ++j) mean += __shfl_sync(0xffffffffu, loss, j);
  }
  if (total != nullptr && lane_id() == 0) *total = mean / (float)n_views;
}

}  // namespace

// mode 0: dL/drgb of photometricLoss; mode 1: d(mean SSIM)/drgb (meanSsim).
// `rows` output rows per CTA (launch_loss).
// Bound by latency at 16 warps per SM (the running sums take 125 registers), with
// about 62% of issue slots and of shared-memory wavefronts taken. The tiled form
// before it, with every blur through shared memory and halos on all sides, took
// 660 instructions per channel and pixel to this one's 340: 8 images of 1920x1440
// in 1628 -> 1043 us, one of 1280x720 in 88 -> 66, one of 320x240 in 27 -> 23.
// Unpaired arithmetic took 1167 us at 8 images; blurring x^2 + y^2 as one plane
// and adding the taps in symmetric pairs first 967, but with other roundings in the
// variances, where the squares cancel: gradients of the parameters moved by up to
// 6e-4 of a typical one against the order kept here.
__global__ void __launch_bounds__(kCols, 4)
    k_loss(const float* __restrict__ rendered, const float* __restrict__ target,
           const ViewDesc* __restrict__ views, int n_views, const LossParams lp, int rows,
           float* __restrict__ grad_out, double* __restrict__ sums,
           float* __restrict__ per_view, float* __restrict__ total) {
  __shared__ LossSmem sm;
  const int v = loss_view<false>(views, n_views, blockIdx.x);
  const ViewDesc& vd = views[v];
  const int W = vd.cam.width, H = vd.cam.height;
  if (W <= 0 || H <= 0) {  // only where no view has a pixel
    finish_loss<kCols>(0.0, 0.0, v, views, n_views, lp, sums, per_view, total);
    return;
  }
  const int strips = (W + kStrip - 1) / kStrip;
  int local = blockIdx.x - vd.loss_tile_offset;
  const int c = local % 3;
  local /= 3;
  const int ox = (local % strips) * kStrip, oy = (local / strips) * rows;
  const int height = min(rows, H - oy);  // output rows of this CTA
  const int t = threadIdx.x;
  const int X = ox - 10 + t;  // this thread's column
  const bool col_in = X >= 0 && X < W;
  const bool output = t >= 10 && t < 10 + kStrip && X < W;
  const int64_t pitch = (int64_t)W * 3;
  const int64_t at = (int64_t)X * 3 + c;
  const float* r_next = rendered + vd.pixel_offset * 3 + at + (oy - 10) * pitch;
  const float* t_next = target + vd.target_offset * 3 + at + (oy - 10) * pitch;
  float* out = grad_out != nullptr ? grad_out + vd.pixel_offset * 3 + at + oy * pitch : nullptr;
  const float w = lp.ssim_weight;
  // 1 / values and 1 / (pixels * 3) of photometricLoss and meanSsim: equal
  const float inv = 1.f / (float)((int64_t)W * H * 3);
  const float c1 = 0.01f * 0.01f, c2 = 0.03f * 0.03f;
  double l1_sum = 0.0, ssim_sum = 0.0;
  // the columns that only pad: zero throughout
  for (int i = t; i < (int)(sizeof(LossSmem) / sizeof(float)); i += kCols)
    reinterpret_cast<float*>(&sm)[i] = 0.f;
  // Running vertical sums: after a row's horizontal blur h, sum j becomes sum
  // j + 1 plus kernel[j] h, so sum 0 is the blur of the last eleven rows. Planes
  // go in pairs through the paired FP32 instructions (half the issue slots):
  // (x, y), (x^2, y^2), and the partials by variance and covariance.
  float2 axy[11], asp[11], b12[11];
  float b0[11], ap[11];
  const float2 zero2 = make_float2(0.f, 0.f);
#pragma unroll
  for (int j = 0; j < 11; ++j) {
    axy[j] = asp[j] = b12[j] = zero2;
    b0[j] = ap[j] = 0.f;
  }
  auto both = [&](int k) { return make_float2(lp.kernel[k], lp.kernel[k]); };
  auto slide2 = [&](float2 (&acc)[11], float2 h) {
#pragma unroll
    for (int j = 0; j < 10; ++j) acc[j] = __ffma2_rn(both(j), h, acc[j + 1]);
    acc[10] = __fmul2_rn(both(10), h);
  };
  const unsigned rows_in = col_in ? (unsigned)H : 0u;  // no row of a column outside
  float2 next = zero2;
  auto load = [&](int Y) {
    next = zero2;
    if ((unsigned)Y < rows_in) next = make_float2(*r_next, *t_next);
    r_next += pitch;
    t_next += pitch;
  };
  load(oy - 10);
  float t_mu = 0.f;  // the last statistics row's partials
  float2 t_vc = zero2;
  const int last_in = height + 20;
  __syncthreads();
  // iteration i: input row oy - 10 + i; its statistics row is five above; the
  // partials of iteration i - 1 are blurred here, and the output row is 21 below i
  for (int i = 0; i <= last_in; ++i) {
    float2* const in = sm.in[(unsigned)i % kRing] + t;
    float2* const p12 = sm.p12[i & 1] + t;
    float* const p0 = sm.p0[i & 1] + t;
    in[kPad] = next;  // (iteration last_in writes a row that nothing reads)
    load(oy - 9 + i);
    p0[kPad] = t_mu;
    p12[kPad] = t_vc;
    // the only barrier of a row: what it orders is written again two (partials)
    // or sixteen rows on, past the next barrier
    __syncthreads();
    if (i >= 11) {
      // horizontal blur of the partials
      float q0 = lp.kernel[0] * p0[0];
      float2 q12 = __fmul2_rn(both(0), p12[0]);
#pragma unroll
      for (int k = 1; k < 11; ++k) {
        q0 += lp.kernel[k] * p0[k];
        q12 = __ffma2_rn(both(k), p12[k], q12);
      }
#pragma unroll
      for (int j = 0; j < 10; ++j) b0[j] = lp.kernel[j] * q0 + b0[j + 1];
      b0[10] = lp.kernel[10] * q0;
      slide2(b12, q12);
      if (i >= 21 && output) {
        const float2 p = sm.in[(unsigned)(i - 11) % kRing][t + kPad];
        // dL/dx = blur(t_mu) + 2x blur(t_var) - 2 blur(t_var mu_x)
        //        + y blur(t_cov) - blur(t_cov mu_y)
        float g = b0[0] + 2.f * p.x * b12[0].x + p.y * b12[0].y;
        if (lp.mode == 0) {
          const float diff = p.x - p.y;
          l1_sum += (double)fabsf(diff);
          const float l1 = (1.f - w) * inv;
          g = (diff > 0.f ? l1 : (diff < 0.f ? -l1 : 0.f)) - w * g;
        }
        if (out != nullptr) {
          *out = g;
          out += pitch;
        }
      }
    }
    if (i == last_in) break;
    // horizontal blur of x, y, x^2 + y^2 and x y
    float2 hxy = zero2, hsq = zero2;
    float hp = 0.f;
#pragma unroll
    for (int k = 0; k < 11; ++k) {
      const float2 p = in[k];
      hxy = __ffma2_rn(both(k), p, hxy);
      hsq = __ffma2_rn(both(k), __fmul2_rn(p, p), hsq);
      hp += lp.kernel[k] * __fmul_rn(p.x, p.y);
    }
    slide2(axy, hxy);
    slide2(asp, hsq);
#pragma unroll
    for (int j = 0; j < 10; ++j) ap[j] = lp.kernel[j] * hp + ap[j + 1];
    ap[10] = lp.kernel[10] * hp;
    // the statistics row's SSIM and partials
    const int Y = oy - 15 + i;
    t_mu = 0.f;
    t_vc = zero2;
    if (i >= 10 && (unsigned)Y < rows_in) {
      const float mu_x = axy[0].x, mu_y = axy[0].y;
      const float var_x = asp[0].x - mu_x * mu_x;
      const float var_y = asp[0].y - mu_y * mu_y;
      const float cov = ap[0] - mu_x * mu_y;
      const float a = 2.f * mu_x * mu_y + c1;
      const float b = 2.f * cov + c2;
      const float cc = mu_x * mu_x + mu_y * mu_y + c1;
      const float d = var_x + var_y + c2;
      // hardware reciprocal approximations (relative error ~1e-7, far inside the
      // 1e-5 loss tolerance; cc >= C1 and d >= C2 - rounding)
      const float rc = __fdividef(1.f, cc), rd = __fdividef(1.f, d);
      const float r_ccd = rc * rd;  // 1 / (cc d)
      const float ssim = (a * b) * r_ccd;
      if (output && Y >= oy && Y < oy + height) ssim_sum += (double)ssim;
      t_mu = inv * (2.f * b * r_ccd) * (mu_y - mu_x * a * rc);
      t_vc.x = -inv * ssim * rd;
      t_vc.y = inv * (2.f * a * r_ccd);
      // the three terms without a pixel factor, blurred as one plane
      t_mu = t_mu - 2.f * t_vc.x * mu_x - t_vc.y * mu_y;
    }
  }
  finish_loss<kCols>(l1_sum, ssim_sum, v, views, n_views, lp, sums, per_view, total);
}

// The loss without SSIM (w = 0): an elementwise pass, `rows` blocks of kL1Values
// values per view's share of the grid. Bound by HBM (36 bytes per pixel).
constexpr int kL1Threads = 256, kL1Values = 2048;

__global__ void __launch_bounds__(kL1Threads)
    k_loss_l1(const float* __restrict__ rendered, const float* __restrict__ target,
              const ViewDesc* __restrict__ views, int n_views, const LossParams lp,
              float* __restrict__ grad_out, double* __restrict__ sums,
              float* __restrict__ per_view, float* __restrict__ total) {
  const int v = loss_view<true>(views, n_views, blockIdx.x);
  const ViewDesc& vd = views[v];
  const int64_t values = (int64_t)vd.cam.width * vd.cam.height * 3;
  const float inv = 1.f / (float)values;
  const int64_t first = (int64_t)(blockIdx.x - vd.l1_block_offset) * kL1Values + threadIdx.x;
  const float* r = rendered + vd.pixel_offset * 3;
  const float* g = target + vd.target_offset * 3;
  double l1_sum = 0.0;
#pragma unroll
  for (int k = 0; k < kL1Values / kL1Threads; ++k) {
    const int64_t i = first + k * kL1Threads;
    if (i >= values) break;
    const float diff = r[i] - g[i];
    l1_sum += (double)fabsf(diff);
    const float sign = diff > 0.f ? 1.f : (diff < 0.f ? -1.f : 0.f);
    if (grad_out != nullptr)
      grad_out[vd.pixel_offset * 3 + i] = (1.f - lp.ssim_weight) * sign * inv;
  }
  finish_loss<kL1Threads>(l1_sum, 0.0, v, views, n_views, lp, sums, per_view, total);
}

int64_t loss_blocks(int width, int height, int rows) {
  if (width <= 0 || height <= 0) return 0;
  if (rows <= 0) return ((int64_t)width * height * 3 + kL1Values - 1) / kL1Values;
  return 3 * (int64_t)((width + kStrip - 1) / kStrip) * ((height + rows - 1) / rows);
}

// A march of R output rows takes R + 21 iterations. An iteration was measured at
// 770, 950, 1300 and 1680 cycles with 1, 2, 3 and 4 CTAs on the SM (a row is a
// chain of loads, blurs and a barrier that one CTA's four warps do not hide): short
// marches spread small images over the SMs, long ones spare large images the
// extra rows. R is the one with the least estimated time; at one view of 1280x720
// 62 us, against 84 at 128 rows and 119 at 8, at 320x240 22 us against 36 at 48 (with
// the order of summation before).
int loss_rows(const int* widths, const int* heights, int n) {
  constexpr int kSms = 148, kPerSm = 4;
  constexpr double kCycles[kPerSm + 1] = {0.0, 770.0, 950.0, 1300.0, 1680.0};
  int best = 8;
  double best_cost = 0.0;
  for (int rows = 8; rows <= 512; rows += std::max(4, rows / 32 * 4)) {
    int64_t blocks = 0;
    for (int v = 0; v < n; ++v) blocks += loss_blocks(widths[v], heights[v], rows);
    const int64_t waves = blocks / (kSms * kPerSm), rest = blocks % (kSms * kPerSm);
    const double cost =
        (rows + 21) * (waves * kCycles[kPerSm] + kCycles[(rest + kSms - 1) / kSms]);
    if (rows == 8 || cost < best_cost) {
      best = rows;
      best_cost = cost;
    }
  }
  return best;
}

void launch_loss(const float* rendered, const float* target, const ViewDesc* views, int n_views,
                 int64_t blocks, int rows, const LossParams& lp, float* grad_out, double* sums,
                 float* per_view, float* total, cudaStream_t stream) {
  if (n_views <= 0) return;
  cudaMemsetAsync(sums, 0, sizeof(double) * (2 * n_views + 1), stream);
  count_launch();
  if (rows > 0)
    k_loss<<<(unsigned)std::max<int64_t>(blocks, 1), kCols, 0, stream>>>(rendered, target, views, n_views, lp, rows,
                                                   grad_out, sums, per_view, total);
  else
    k_loss_l1<<<(unsigned)std::max<int64_t>(blocks, 1), kL1Threads, 0, stream>>>(rendered, target, views, n_views, lp,
                                                           grad_out, sums, per_view, total);
}

}  // namespace pxs

// ------------------------------------------------ allocation-free entry point
//
// pxs_photometric_loss_static serves callers that cannot allocate device
// memory (a host framework whose caching allocator owns the GPU's memory, or
// a loop that must not pay cudaFree's device-wide synchronisation). The loss
// kernel's scratch -- the per-image descriptors it reads and the two double
// sums per image it accumulates into -- lives here, in one file-scope array
// that every GPU loading the library holds until the process exits. Its name
// in host code stands in for the symbol only; the device address comes from
// cudaGetSymbolAddress, looked up once per device on the first call there.
// Every call shares the array and finds the previous call's contents in it:
// the descriptors are rewritten and the sums cleared before each kernel runs,
// and calls that overlap on the GPU race.

namespace pxs {
namespace {

struct StaticLossScratch {
  ViewDesc views[PXS_STATIC_LOSS_MAX_VIEWS];
  double sums[2 * PXS_STATIC_LOSS_MAX_VIEWS + 1];
};
static_assert(sizeof(StaticLossScratch) <= PXS_STATIC_LOSS_SCRATCH_BYTES,
              "the static loss scratch does not hold its views");

static __device__ __align__(256) unsigned char g_loss_scratch[PXS_STATIC_LOSS_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
std::mutex g_scratch_mutex;
StaticLossScratch* g_scratch_addr[kMaxDevices] = {};

// Image v of a batch of same-sized images laid out one after another.
__global__ void k_static_loss_views(StaticLossScratch* scratch, int width, int height,
                                    int n_views, int blocks) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n_views) return;
  ViewDesc d;
  memset(&d, 0, sizeof(d));
  d.cam.width = width;
  d.cam.height = height;
  d.pixel_offset = (int64_t)v * width * height;
  d.target_offset = d.pixel_offset;
  d.loss_tile_offset = d.l1_block_offset = v * blocks;
  scratch->views[v] = d;
}

struct StaticError {
  int status;
  const char* what;
};

// The scratch's device address on the current device; the first call on a
// device looks it up.
StaticLossScratch* static_scratch(int device) {
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (g_scratch_addr[device] == nullptr) {
    void* ptr = nullptr;
    cudaError_t err = cudaGetSymbolAddress(&ptr, g_loss_scratch);
    if (err != cudaSuccess) throw StaticError{PXS_ERR_CUDA, cudaGetErrorString(err)};
    g_scratch_addr[device] = static_cast<StaticLossScratch*>(ptr);
  }
  return g_scratch_addr[device];
}

int static_fail(int status, const char* what, char* error, size_t error_len) {
  if (error != nullptr && error_len > 0) std::snprintf(error, error_len, "%s", what);
  return status;
}

}  // namespace
}  // namespace pxs

extern "C" int pxs_photometric_loss_static(const float* rendered, const float* target,
                                           int32_t width, int32_t height, int32_t n_views,
                                           float ssim_weight, float* dL_drgb,
                                           float* per_view_loss, float* loss, void* stream,
                                           char* error, size_t error_len) {
  using namespace pxs;
  char why[160];
  if (width < 0 || height < 0 || n_views < 0)
    return static_fail(PXS_ERR_INVALID, "negative image size or count", error, error_len);
  if (n_views > PXS_STATIC_LOSS_MAX_VIEWS) {
    std::snprintf(why, sizeof(why),
                  "n_views = %d exceeds the static scratch limit of %d images per call",
                  (int)n_views, PXS_STATIC_LOSS_MAX_VIEWS);
    return static_fail(PXS_ERR_INVALID, why, error, error_len);
  }
  const bool empty = n_views == 0 || width == 0 || height == 0;
  if (!empty && (rendered == nullptr || target == nullptr))
    return static_fail(PXS_ERR_INVALID, "image is null", error, error_len);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  try {
    if (empty) {  // nothing to score: every loss is 0
      if (loss != nullptr) {
        const cudaError_t err = cudaMemsetAsync(loss, 0, sizeof(float), s);
        if (err != cudaSuccess) throw StaticError{PXS_ERR_CUDA, cudaGetErrorString(err)};
      }
      if (per_view_loss != nullptr && n_views > 0) {
        const cudaError_t err = cudaMemsetAsync(per_view_loss, 0, sizeof(float) * n_views, s);
        if (err != cudaSuccess) throw StaticError{PXS_ERR_CUDA, cudaGetErrorString(err)};
      }
      return PXS_OK;
    }
    int device = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess) throw StaticError{PXS_ERR_CUDA, cudaGetErrorString(err)};
    if (device < 0 || device >= kMaxDevices)
      throw StaticError{PXS_ERR_UNAVAILABLE, "device ordinal beyond the supported range"};
    StaticLossScratch* scratch = static_scratch(device);
    cudaGetLastError();  // an earlier, unrelated failure is not this call's
    count_launch();
    int rows = 0;
    if (ssim_weight > 0.f) {
      const std::vector<int> ws(n_views, width), hs(n_views, height);
      rows = loss_rows(ws.data(), hs.data(), n_views);
    }
    const int64_t blocks = loss_blocks(width, height, rows);
    if (blocks * n_views > INT32_MAX) throw StaticError{PXS_ERR_INVALID, "images too large"};
    k_static_loss_views<<<(n_views + 63) / 64, 64, 0, s>>>(scratch, width, height, n_views,
                                                           (int)blocks);
    LossParams lp;
    ssim_kernel_weights(lp.kernel);
    lp.ssim_weight = ssim_weight;
    lp.mode = 0;
    // launch_loss clears scratch->sums on `s` before the kernel adds into them.
    launch_loss(rendered, target, scratch->views, n_views, blocks * n_views, rows, lp, dL_drgb,
                scratch->sums, per_view_loss, loss, s);
    err = cudaGetLastError();
    if (err != cudaSuccess) throw StaticError{PXS_ERR_CUDA, cudaGetErrorString(err)};
    return PXS_OK;
  } catch (const StaticError& e) {
    return static_fail(e.status, e.what, error, error_len);
  } catch (const std::exception& e) {
    return static_fail(PXS_ERR_CUDA, e.what(), error, error_len);
  }
}
