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
// Batches too small for that go by 32x32 tiles (loss_plan).
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
    // horizontal blur of x, y, x^2, y^2 and x y
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

// ---------------------------------------------------------------- small batches
//
// A march's rows follow one another, so a CTA takes (rows + 21) times a row's latency
// however few CTAs there are: below about a megapixel in all, tiles finish first
// (loss_plan). A CTA owns a 32x32 output tile and takes the channels one after
// another: it stages a channel of both images over a 10-pixel halo, blurs the five
// statistic planes onto a 5-pixel halo, forms the SSIM map and its partials there,
// blurs those back onto the tile and writes the gradient. Each blur is register-
// blocked: a thread loads a strip once and slides the 11 taps along it, in the
// march's tap order. Bound by latency with one CTA on an SM, by instructions with two
// (86 KB of shared memory each).
constexpr int TW = 32, TH = 32;
constexpr int IW = TW + 20, IH = TH + 20;  // input region
constexpr int SW = TW + 10, SH = TH + 10;  // statistics region
constexpr int kTileThreads = 320;  // every blur pass below is one round of items

struct TileSmem {
  float in_r[IH][IW];      // rendered, the current channel
  float in_t[IH][IW];      // target
  float hb[5][IH][SW];     // horizontal blur of the five products / of the three partials
  float st[3][SH][SW];     // the three partial planes
};

__global__ void __launch_bounds__(kTileThreads, 2)
    k_loss_tiles(const float* __restrict__ rendered, const float* __restrict__ target,
                 const ViewDesc* __restrict__ views, int n_views, const LossParams lp,
                 float* __restrict__ grad_out, double* __restrict__ sums,
                 float* __restrict__ per_view, float* __restrict__ total) {
  extern __shared__ __align__(16) unsigned char tile_smem[];
  TileSmem& sm = *reinterpret_cast<TileSmem*>(tile_smem);
  const int v = loss_view<false>(views, n_views, blockIdx.x);
  const ViewDesc& vd = views[v];
  const int W = vd.cam.width, H = vd.cam.height;
  if (W <= 0 || H <= 0) {  // only where no view has a pixel
    finish_loss<kTileThreads>(0.0, 0.0, v, views, n_views, lp, sums, per_view, total);
    return;
  }
  const int local = blockIdx.x - vd.loss_tile_offset, across = (W + TW - 1) / TW;
  const int ox = (local % across) * TW, oy = (local / across) * TH;
  const int64_t pix0 = vd.pixel_offset;
  const float* rimg = rendered + pix0 * 3;
  const float* timg = target + vd.target_offset * 3;
  const int tid = threadIdx.x;
  const float w = lp.ssim_weight;
  // 1 / values and 1 / (pixels * 3) of photometricLoss and meanSsim: equal
  const float inv = 1.f / (float)((int64_t)W * H * 3);
  const float c1 = 0.01f * 0.01f, c2 = 0.03f * 0.03f;
  double l1_sum = 0.0, ssim_sum = 0.0;

  for (int c = 0; c < 3; ++c) {
    // stage channel c of both images over the input region, zero outside
    // (the other channels' bytes of the same lines come back from L2)
    for (int q = tid; q < IH * IW; q += kTileThreads) {
      const int lx = q % IW, ly = q / IW;
      const int X = ox - 10 + lx, Y = oy - 10 + ly;
      float a = 0.f, b = 0.f;
      if (X >= 0 && X < W && Y >= 0 && Y < H) {
        const int64_t o = ((int64_t)Y * W + X) * 3 + c;
        a = rimg[o];
        b = timg[o];
      }
      sm.in_r[ly][lx] = a;
      sm.in_t[ly][lx] = b;
    }
    __syncthreads();
    // horizontal blur of the five products over every input row, onto the
    // statistics columns; a thread slides the 11 taps over 7 outputs
    constexpr int HS = 7;
    for (int item = tid; item < IH * (SW / HS); item += kTileThreads) {
      const int r = item / (SW / HS), col0 = (item % (SW / HS)) * HS;
      float xs[HS + 10], ys[HS + 10], xx[HS + 10], yy[HS + 10], xy[HS + 10];
#pragma unroll
      for (int k = 0; k < HS + 10; ++k) {
        xs[k] = sm.in_r[r][col0 + k];
        ys[k] = sm.in_t[r][col0 + k];
        xx[k] = xs[k] * xs[k];
        yy[k] = ys[k] * ys[k];
        xy[k] = xs[k] * ys[k];
      }
#pragma unroll
      for (int o = 0; o < HS; ++o) {
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f, s4 = 0.f;
#pragma unroll
        for (int k = 0; k < 11; ++k) {
          const float kk = lp.kernel[k];
          s0 += kk * xs[o + k];
          s1 += kk * ys[o + k];
          s2 += kk * xx[o + k];
          s3 += kk * yy[o + k];
          s4 += kk * xy[o + k];
        }
        sm.hb[0][r][col0 + o] = s0;
        sm.hb[1][r][col0 + o] = s1;
        sm.hb[2][r][col0 + o] = s2;
        sm.hb[3][r][col0 + o] = s3;
        sm.hb[4][r][col0 + o] = s4;
      }
    }
    __syncthreads();
    // vertical blur -> statistics, then the SSIM map and its partials in
    // place; a thread takes one column and 7 consecutive rows
    constexpr int VS = 7;
    constexpr int VSEG = (SH + VS - 1) / VS;
    for (int item = tid; item < SW * VSEG; item += kTileThreads) {
      const int col = item % SW, r0 = (item / SW) * VS;
      float m[5][VS];
#pragma unroll
      for (int p = 0; p < 5; ++p) {
        float hv[VS + 10];
#pragma unroll
        for (int k = 0; k < VS + 10; ++k) hv[k] = (r0 + k < IH) ? sm.hb[p][r0 + k][col] : 0.f;
#pragma unroll
        for (int o = 0; o < VS; ++o) {
          float acc = 0.f;
#pragma unroll
          for (int k = 0; k < 11; ++k) acc += lp.kernel[k] * hv[o + k];
          m[p][o] = acc;
        }
      }
#pragma unroll
      for (int o = 0; o < VS; ++o) {
        const int r = r0 + o;
        if (r >= SH) break;
        const int X = ox - 5 + col, Y = oy - 5 + r;
        float t_mu = 0.f, t_var = 0.f, t_cov = 0.f, mu_x = m[0][o], mu_y = m[1][o];
        if (X >= 0 && X < W && Y >= 0 && Y < H) {
          const float var_x = m[2][o] - mu_x * mu_x;
          const float var_y = m[3][o] - mu_y * mu_y;
          const float cov = m[4][o] - mu_x * mu_y;
          const float a = 2.f * mu_x * mu_y + c1;
          const float b = 2.f * cov + c2;
          const float cc = mu_x * mu_x + mu_y * mu_y + c1;
          const float d = var_x + var_y + c2;
          // hardware reciprocal approximations (relative error ~1e-7, far
          // inside the 1e-5 loss tolerance; cc >= C1 and d >= C2 - rounding)
          const float rc = __fdividef(1.f, cc), rd = __fdividef(1.f, d);
          const float r_ccd = rc * rd;  // 1 / (cc d)
          const float ssim = (a * b) * r_ccd;
          if (col >= 5 && col < 5 + TW && r >= 5 && r < 5 + TH) ssim_sum += (double)ssim;
          t_mu = inv * (2.f * b * r_ccd) * (mu_y - mu_x * a * rc);
          t_var = -inv * ssim * rd;
          t_cov = inv * (2.f * a * r_ccd);
        } else {
          mu_x = 0.f;
          mu_y = 0.f;
        }
        // dL/dx = blur(t_mu) + 2x blur(t_var) - 2 blur(t_var mu_x)
        //        + y blur(t_cov) - blur(t_cov mu_y); the blur is linear, so
        // the three terms without a pixel factor are blurred as one plane
        sm.st[0][r][col] = t_mu - 2.f * t_var * mu_x - t_cov * mu_y;
        sm.st[1][r][col] = t_var;
        sm.st[2][r][col] = t_cov;
      }
    }
    __syncthreads();
    // horizontal blur of the partials onto the tile's columns, 16 per thread
    constexpr int HS2 = 16;
    for (int item = tid; item < 3 * SH * (TW / HS2); item += kTileThreads) {
      const int p = item / (SH * (TW / HS2));
      const int rem = item % (SH * (TW / HS2));
      const int r = rem / (TW / HS2), col0 = (rem % (TW / HS2)) * HS2;
      float tv[HS2 + 10];
#pragma unroll
      for (int k = 0; k < HS2 + 10; ++k) tv[k] = sm.st[p][r][col0 + k];
#pragma unroll
      for (int o = 0; o < HS2; ++o) {
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < 11; ++k) acc += lp.kernel[k] * tv[o + k];
        sm.hb[p][r][col0 + o] = acc;
      }
    }
    __syncthreads();
    // vertical blur and the gradient, one column and 4 rows per thread
    constexpr int VS2 = 4;
    for (int item = tid; item < TW * (TH / VS2); item += kTileThreads) {
      const int col = item % TW, r0 = (item / TW) * VS2;
      float B[3][VS2];
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        float hv[VS2 + 10];
#pragma unroll
        for (int k = 0; k < VS2 + 10; ++k) hv[k] = sm.hb[p][r0 + k][col];
#pragma unroll
        for (int o = 0; o < VS2; ++o) {
          float acc = 0.f;
#pragma unroll
          for (int k = 0; k < 11; ++k) acc += lp.kernel[k] * hv[o + k];
          B[p][o] = acc;
        }
      }
#pragma unroll
      for (int o = 0; o < VS2; ++o) {
        const int r = r0 + o;
        const int X = ox + col, Y = oy + r;
        if (X >= W || Y >= H) continue;
        const float x = sm.in_r[r + 10][col + 10];
        const float y = sm.in_t[r + 10][col + 10];
        float g = B[0][o];
        g += 2.f * x * B[1][o];
        g += y * B[2][o];
        if (lp.mode == 0) {
          const float diff = x - y;
          l1_sum += (double)fabsf(diff);
          const float sign = diff > 0.f ? 1.f : (diff < 0.f ? -1.f : 0.f);
          g = (1.f - w) * sign * inv - w * g;
        }
        if (grad_out != nullptr) grad_out[(pix0 + (int64_t)Y * W + X) * 3 + c] = g;
      }
    }
    __syncthreads();
  }
  finish_loss<kTileThreads>(l1_sum, ssim_sum, v, views, n_views, lp, sums, per_view, total);
}

// The loss without SSIM (w = 0): an elementwise pass, a view's share of the grid
// being one block per kL1Values of its values. Bound by HBM (36 bytes per pixel).
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

int64_t loss_blocks(int width, int height, LossPlan plan) {
  if (width <= 0 || height <= 0) return 0;
  switch (plan.form) {
    case LossPlan::kL1:
      return ((int64_t)width * height * 3 + kL1Values - 1) / kL1Values;
    case LossPlan::kTiles:
      return (int64_t)((width + TW - 1) / TW) * ((height + TH - 1) / TH);
    default:
      return 3 * (int64_t)((width + kStrip - 1) / kStrip) *
             ((height + plan.rows - 1) / plan.rows);
  }
}

namespace {

// Estimated times in us, fitted to 134 batches of 1 to 64 images of 16 to 2000 pixels a
// side. A march of R output rows takes R + 21 iterations of 960, 1120, 1460 or 1820
// cycles with 1 to 4 CTAs on the SM (a row is a chain of loads, blurs and a barrier
// that one CTA's four warps do not hide), 1680 in a wave that others follow: short
// marches spread small batches over the SMs, long ones spare large ones the rows that
// run in. Tiles take a round of a CTA on every SM after another.
constexpr int kSms = 148;
double march_us(int rows, int64_t blocks) {
  constexpr int kPerSm = 4;
  constexpr double kRow[kPerSm + 1] = {0.0, 960.0, 1120.0, 1460.0, 1820.0}, kFullRow = 1680.0;
  constexpr double kCyclesPerUs = 1965.0;
  const int64_t waves = blocks / (kSms * kPerSm), rest = blocks % (kSms * kPerSm);
  return 7.0 + 4.0 * waves +
         (rows + 21) / kCyclesPerUs * (waves * kFullRow + kRow[(rest + kSms - 1) / kSms]);
}
double tiles_us(int64_t blocks) {
  return blocks <= kSms ? 24.5 : 11.7 + 10.9 * ((blocks + kSms - 1) / kSms);
}

}  // namespace

// Tiles where the quickest march takes longer: one image of 541x541 in 33 us against 39,
// two of 325x182 in 25 against 29, one of 110x2000 in 33 against 45 and eight of
// 128x1000 in 91 against 109; the march one image of 320x240 in 23 against 25, one of
// 1280x720 in 67 against 77.
LossPlan loss_plan(const int* widths, const int* heights, const int* counts, int n) {
  auto blocks_of = [&](LossPlan plan) {
    int64_t blocks = 0;
    for (int k = 0; k < n; ++k)
      blocks += (int64_t)counts[k] * loss_blocks(widths[k], heights[k], plan);
    return blocks;
  };
  LossPlan best{LossPlan::kTiles, 0};
  double best_us = tiles_us(blocks_of(best));
  for (int rows = 8; rows <= 512; rows += std::max(4, rows / 32 * 4)) {
    const LossPlan plan{LossPlan::kMarch, rows};
    const double us = march_us(rows, blocks_of(plan));
    if (us < best_us) {
      best = plan;
      best_us = us;
    }
  }
  return best;
}

void configure_loss_kernel() {
  cudaFuncSetAttribute(k_loss_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)sizeof(TileSmem));
}

void launch_loss(const float* rendered, const float* target, const ViewDesc* views, int n_views,
                 int64_t blocks, LossPlan plan, const LossParams& lp, float* grad_out,
                 double* sums, float* per_view, float* total, cudaStream_t stream) {
  if (n_views <= 0) return;
  cudaMemsetAsync(sums, 0, sizeof(double) * (2 * n_views + 1), stream);
  count_launch();
  const unsigned grid = (unsigned)std::max<int64_t>(blocks, 1);
  switch (plan.form) {
    case LossPlan::kL1:
      k_loss_l1<<<grid, kL1Threads, 0, stream>>>(rendered, target, views, n_views, lp, grad_out,
                                                 sums, per_view, total);
      break;
    case LossPlan::kTiles:
      k_loss_tiles<<<grid, kTileThreads, sizeof(TileSmem), stream>>>(
          rendered, target, views, n_views, lp, grad_out, sums, per_view, total);
      break;
    default:
      k_loss<<<grid, kCols, 0, stream>>>(rendered, target, views, n_views, lp, plan.rows,
                                         grad_out, sums, per_view, total);
  }
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
// device looks it up and raises the tiled kernel's shared-memory limit.
StaticLossScratch* static_scratch(int device) {
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (g_scratch_addr[device] == nullptr) {
    void* ptr = nullptr;
    cudaError_t err = cudaGetSymbolAddress(&ptr, g_loss_scratch);
    if (err != cudaSuccess) throw StaticError{PXS_ERR_CUDA, cudaGetErrorString(err)};
    err = cudaFuncSetAttribute(k_loss_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sizeof(TileSmem));
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
    LossPlan plan;
    if (ssim_weight > 0.f) plan = loss_plan(&width, &height, &n_views, 1);
    const int64_t blocks = loss_blocks(width, height, plan);
    if (blocks * n_views > INT32_MAX) throw StaticError{PXS_ERR_INVALID, "images too large"};
    k_static_loss_views<<<(n_views + 63) / 64, 64, 0, s>>>(scratch, width, height, n_views,
                                                           (int)blocks);
    LossParams lp;
    ssim_kernel_weights(lp.kernel);
    lp.ssim_weight = ssim_weight;
    lp.mode = 0;
    // launch_loss clears scratch->sums on `s` before the kernel adds into them.
    launch_loss(rendered, target, scratch->views, n_views, blocks * n_views, plan, lp, dL_drgb,
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
