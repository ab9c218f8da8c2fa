// adam.cu -- the optimiser step, fused with clearing the gradients and with
// folding this step's densification statistics into the running totals.
//
// applyGradients (SplatTrainer.cpp:218-256) with adamDelta (:56-65). Compiled
// with -fmad=false: with IEEE division and square root the update is bit-identical
// to the reference's for identical gradients.
#include <algorithm>
#include <limits>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace pxs {

// `plain`: every scalar is finite and epsilon and the corrections are positive.
// Then a parameter that has never had a gradient (m = v = 0) moves by -lr 0 /
// (0 + epsilon) = -0, which is left out: the divisions of 0 by a correction
// would leave the fast path of IEEE division, and in a step that sees part of
// the cloud most parameters are such (with their clearing 0.449 -> 0.296 ms at 1M
// gaussians, 8 views; 0.119 -> 0.051 ms at 151,721, one view).
__device__ __forceinline__ float adam_delta(float& m, float& v, float g, float lr, float b1,
                                            float b2, float eps, float c1, float c2,
                                            bool plain) {
  m = b1 * m + (1.f - b1) * g;
  v = b2 * v + (1.f - b2) * g * g;
  const bool still = plain && m == 0.f && v == 0.f;
  const float m_hat = (still ? 1.f : m) / c1;
  const float v_hat = (still ? 1.f : v) / c2;
  const float delta = -lr * m_hat / (sqrtf(v_hat) + eps);
  return still ? -m : delta;
}

__device__ __forceinline__ bool plain_scalars(const StepScalars& s) {
  const float rates = fabsf(s.lr[0]) + fabsf(s.lr[1]) + fabsf(s.lr[2]) + fabsf(s.lr[3]) +
                      fabsf(s.lr[4]) + fabsf(s.lr[5]);
  return s.epsilon > 0.f && s.correction1 > 0.f && s.correction2 > 0.f && isfinite(rates) &&
         isfinite(s.epsilon) && isfinite(s.correction1) && isfinite(s.correction2);
}

// Quaternion::norm / normalize over (x, y, z, w) storage (SplatTrainer.cpp:247-248).
__device__ __forceinline__ void normalize(float (&q)[4]) {
  const float sq = (q[1] * q[1] + q[3] * q[3]) + (q[2] * q[2] + q[0] * q[0]);
  const float norm = sqrtf(sq);
  if (norm > 1e-6f) {
#pragma unroll
    for (int a = 0; a < 4; ++a) q[a] = q[a] / norm;
  } else {
    q[0] = 1.f;
    q[1] = q[2] = q[3] = 0.f;
  }
}

// accumulateStatistics (SplatTrainer.cpp:258-263), then this step's stats clear.
__device__ __forceinline__ void fold_statistics(int g, int zero_grads, float* screen_gradient,
                                                int32_t* visible_count, float* acc_gradient,
                                                int32_t* acc_views) {
  if (screen_gradient == nullptr) return;
  if (acc_gradient != nullptr) {
    acc_gradient[g] += screen_gradient[g];
    acc_views[g] += visible_count[g];
  }
  if (zero_grads) {
    screen_gradient[g] = 0.f;
    visible_count[g] = 0;
  }
}

// The groups of V floats of the flat P x N arrays (k_adam). The rows' sections
// end at floats 3N, 6N, 10N, 11N, 14N and P N: the first group that begins at
// or past each end, and the group that straddles it (the largest Index: none).
// 32 bits count the groups of four of any arrays that fit the device.
template <int V>
struct AdamGroups {
  using Index = std::conditional_t<V == 4, uint32_t, int64_t>;
  Index next[6];
  Index odd[6];
  Index skipped;  // groups wholly inside the rotation rows
};

constexpr int kAdamThreads = 256, kAdamCtas = 6;

// The form for every count and alignment. The parameters outside the rotation
// are one elementwise problem: the flat P x N arrays are cut into groups of V
// consecutive floats (V = 4, 16-byte loads and stores, where the arrays start
// on 16 bytes, whatever N is: groups run across rows), one group per thread,
// blocks [rot_blocks, grid). Blocks [0, rot_blocks) take a gaussian per thread:
// its four rotation rows together, so the quaternion is renormalised in
// registers, and its densify statistics. A group that straddles the rotation
// rows' ends, or the array's, goes element by element.
//
// Bound by HBM: 28 bytes per float (32 when it clears the gradients), with about
// 70 instructions per float of IEEE divisions and square root that keep the
// reference's bits; 40 registers (6 CTAs per SM, a few bytes spilled around the
// divisions' slow path) measured best. 333,333 gaussians SH3: 134.5 -> 102.3 us
// (5.4 TB/s; rows of a count that is not a multiple of 4 took a gaussian per
// thread before).
template <int V>
__global__ void __launch_bounds__(kAdamThreads, kAdamCtas)
    k_adam(float* __restrict__ params, float* __restrict__ grads, float* __restrict__ m,
           float* __restrict__ v, int N, int S, const StepScalars* __restrict__ scalars,
           int zero_grads, float* __restrict__ screen_gradient,
           int32_t* __restrict__ visible_count, float* __restrict__ acc_gradient,
           int32_t* __restrict__ acc_views, const int32_t* __restrict__ skip,
           const float* __restrict__ position_scale, int rot_blocks, AdamGroups<V> groups) {
  // a step whose tile pairs overflowed is redone by the host: leave the state alone
  if (skip != nullptr && *skip != 0) return;
  const StepScalars& s = *scalars;
  const int64_t n = N;
  const bool plain = plain_scalars(s);
  if ((int)blockIdx.x < rot_blocks) {
    const int g = blockIdx.x * kAdamThreads + threadIdx.x;
    if (g >= N) return;
    float q[4], gg[4], mm[4], vv[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int64_t i = (PXS_C_ROTATION + a) * n + g;
      q[a] = params[i];
      gg[a] = grads[i];
      mm[a] = m[i];
      vv[a] = v[i];
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int64_t i = (PXS_C_ROTATION + a) * n + g;
      q[a] = q[a] + adam_delta(mm[a], vv[a], gg[a], s.lr[2], s.beta1, s.beta2, s.epsilon,
                               s.correction1, s.correction2, plain);
      m[i] = mm[a];
      v[i] = vv[a];
      if (zero_grads) grads[i] = 0.f;
    }
    normalize(q);
#pragma unroll
    for (int a = 0; a < 4; ++a) params[(PXS_C_ROTATION + a) * n + g] = q[a];
    fold_statistics(g, zero_grads, screen_gradient, visible_count, acc_gradient, acc_views);
    return;
  }
  // group k: floats [k V, k V + V); the groups wholly inside the rotation rows
  // are left out
  using Index = typename AdamGroups<V>::Index;
  Index k = (Index)(blockIdx.x - rot_blocks) * kAdamThreads + threadIdx.x;
  if (k >= groups.next[1]) k += groups.skipped;
  if (k >= groups.next[5]) return;
  // positionLearningRate (SplatTrainer.cpp:200-208) ends with "* extent": with
  // several scenes lr[0] holds the rest and each gaussian its scene's extent
  const bool scaled = position_scale != nullptr && k < groups.next[0];
  float lr = s.lr[5];
  bool whole = V > 1 && k != groups.odd[5];
  if (k < groups.next[4]) {
    lr = k >= groups.next[3] ? s.lr[4]
         : k >= groups.next[1] ? s.lr[3]
         : k >= groups.next[0] ? s.lr[1]
                               : s.lr[0];
    whole = whole && !scaled && k != groups.odd[0] && k != groups.odd[1] &&
            k != groups.odd[2] && k != groups.odd[3] && k != groups.odd[4];
  }
  if (whole) {
    const float4 p4 = reinterpret_cast<const float4*>(params)[k];
    const float4 g4 = reinterpret_cast<const float4*>(grads)[k];
    const float4 m4 = reinterpret_cast<const float4*>(m)[k];
    const float4 v4 = reinterpret_cast<const float4*>(v)[k];
    float pp[4] = {p4.x, p4.y, p4.z, p4.w}, gg[4] = {g4.x, g4.y, g4.z, g4.w};
    float mm[4] = {m4.x, m4.y, m4.z, m4.w}, vv[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      pp[j] += adam_delta(mm[j], vv[j], gg[j], lr, s.beta1, s.beta2, s.epsilon, s.correction1,
                          s.correction2, plain);
    reinterpret_cast<float4*>(params)[k] = make_float4(pp[0], pp[1], pp[2], pp[3]);
    reinterpret_cast<float4*>(m)[k] = make_float4(mm[0], mm[1], mm[2], mm[3]);
    reinterpret_cast<float4*>(v)[k] = make_float4(vv[0], vv[1], vv[2], vv[3]);
    if (zero_grads) reinterpret_cast<float4*>(grads)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
#pragma unroll 1
  for (int j = 0; j < V; ++j) {
    const int64_t e = (int64_t)k * V + j;
    const int row = (int)(e / n);
    if (row >= 14 + 3 * S) return;
    if (row >= PXS_C_ROTATION && row < PXS_C_OPACITY) continue;
    float rate = row < PXS_C_LOG_SCALE ? s.lr[0]
                 : row < PXS_C_ROTATION ? s.lr[1]
                 : row == PXS_C_OPACITY ? s.lr[3]
                 : row < PXS_C_SH_REST  ? s.lr[4]
                                        : s.lr[5];
    if (row < PXS_C_LOG_SCALE && position_scale != nullptr) rate *= position_scale[e - row * n];
    float mm = m[e], vv = v[e];
    params[e] += adam_delta(mm, vv, grads[e], rate, s.beta1, s.beta2, s.epsilon, s.correction1,
                            s.correction2, plain);
    m[e] = mm;
    v[e] = vv;
    if (zero_grads) grads[e] = 0.f;
  }
}

// The same where N is a multiple of four and so every row starts on 16 bytes: no
// group straddles two rows, and the rotation goes by groups too. A rotation block
// takes 256 gaussians, a quarter of its threads per row; the new quaternions pass
// through shared memory to a thread each, which normalises it, and back.
//
// 48 registers (5 CTAs per SM) without a spill: held to 40, its spills are on the way of
// every thread (71 -> 82 us for 865,748 gaussians without SH). Times in us here / by
// k_adam / a thread per gaussian group and row, with all four rotation rows in one
// thread, cold and with the gradients cleared: 73 / 78 / 75 (865,748, no SH), 42 / 44 / 42
// (400,000, no SH), 109 / 115 / 113 (865,748 SH1), 296 / 309 / 311 (1M SH3); it reaches
// 6.2 TB/s at the last.
constexpr int kRowsCtas = 5;

__global__ void __launch_bounds__(kAdamThreads, kRowsCtas)
    k_adam_rows(float* __restrict__ params, float* __restrict__ grads, float* __restrict__ m,
                float* __restrict__ v, int N, int S, const StepScalars* __restrict__ scalars,
                int zero_grads, float* __restrict__ screen_gradient,
                int32_t* __restrict__ visible_count, float* __restrict__ acc_gradient,
                int32_t* __restrict__ acc_views, const int32_t* __restrict__ skip,
                const float* __restrict__ position_scale, int rot_blocks) {
  __shared__ __align__(16) float s_q[4][kAdamThreads];
  if (skip != nullptr && *skip != 0) return;
  const StepScalars& s = *scalars;
  const bool plain = plain_scalars(s);
  const uint32_t n4 = (uint32_t)N / 4;
  const bool rotation = (int)blockIdx.x < rot_blocks;
  uint32_t k;  // the group
  float lr;
  bool live = true;
  if (rotation) {
    const uint32_t g4 = blockIdx.x * (kAdamThreads / 4) + threadIdx.x % (kAdamThreads / 4);
    k = (PXS_C_ROTATION + threadIdx.x / (kAdamThreads / 4)) * n4 + g4;
    lr = s.lr[2];
    live = g4 < n4;
  } else {
    k = (blockIdx.x - rot_blocks) * kAdamThreads + threadIdx.x;
    if (k >= PXS_C_ROTATION * n4) k += 4 * n4;
    if (k >= (14 + 3 * S) * n4) return;
    lr = k >= 14 * n4                ? s.lr[5]
         : k >= 11 * n4              ? s.lr[4]
         : k >= PXS_C_OPACITY * n4   ? s.lr[3]
         : k >= PXS_C_LOG_SCALE * n4 ? s.lr[1]
                                     : s.lr[0];
  }
  if (live) {
    const float4 p4 = reinterpret_cast<const float4*>(params)[k];
    const float4 g4 = reinterpret_cast<const float4*>(grads)[k];
    const float4 m4 = reinterpret_cast<const float4*>(m)[k];
    const float4 v4 = reinterpret_cast<const float4*>(v)[k];
    float rate[4] = {lr, lr, lr, lr};
    if (position_scale != nullptr && k < PXS_C_LOG_SCALE * n4) {
      const float* at = position_scale + 4 * (k >= 2 * n4 ? k - 2 * n4 : k >= n4 ? k - n4 : k);
#pragma unroll
      for (int j = 0; j < 4; ++j) rate[j] *= at[j];
    }
    float pp[4] = {p4.x, p4.y, p4.z, p4.w}, gg[4] = {g4.x, g4.y, g4.z, g4.w};
    float mm[4] = {m4.x, m4.y, m4.z, m4.w}, vv[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      pp[j] += adam_delta(mm[j], vv[j], gg[j], rate[j], s.beta1, s.beta2, s.epsilon,
                          s.correction1, s.correction2, plain);
    const float4 out = make_float4(pp[0], pp[1], pp[2], pp[3]);
    if (rotation) reinterpret_cast<float4*>(s_q)[threadIdx.x] = out;
    else reinterpret_cast<float4*>(params)[k] = out;
    reinterpret_cast<float4*>(m)[k] = make_float4(mm[0], mm[1], mm[2], mm[3]);
    reinterpret_cast<float4*>(v)[k] = make_float4(vv[0], vv[1], vv[2], vv[3]);
    if (zero_grads) reinterpret_cast<float4*>(grads)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (!rotation) return;
  __syncthreads();
  const int t = threadIdx.x, g = blockIdx.x * kAdamThreads + t;
  float q[4] = {s_q[0][t], s_q[1][t], s_q[2][t], s_q[3][t]};
  normalize(q);
#pragma unroll
  for (int a = 0; a < 4; ++a) s_q[a][t] = q[a];
  __syncthreads();
  if (live) reinterpret_cast<float4*>(params)[k] = reinterpret_cast<const float4*>(s_q)[t];
  if (g < N)
    fold_statistics(g, zero_grads, screen_gradient, visible_count, acc_gradient, acc_views);
}

namespace {

template <int V>
void launch_adam_groups(float* params, float* grads, float* m, float* v, int N, int S,
                        const StepScalars* scalars, int zero_grads, float* screen_gradient,
                        int32_t* visible_count, float* acc_gradient, int32_t* acc_views,
                        const int32_t* skip, cudaStream_t stream, const float* position_scale) {
  using Index = typename AdamGroups<V>::Index;
  const int64_t ends[6] = {3, 6, 10, 11, 14, 14 + 3 * (int64_t)S};  // rows
  AdamGroups<V> groups;
  for (int i = 0; i < 6; ++i) {
    const int64_t end = ends[i] * N;
    groups.next[i] = (Index)((end + V - 1) / V);
    groups.odd[i] = end % V != 0 ? (Index)(end / V) : std::numeric_limits<Index>::max();
  }
  groups.skipped = (Index)std::max<int64_t>(ends[2] * N / V - (int64_t)groups.next[1], 0);
  const int rot_blocks = (N + kAdamThreads - 1) / kAdamThreads;
  const int64_t blocks = rot_blocks + ((int64_t)groups.next[5] - (int64_t)groups.skipped +
                                       kAdamThreads - 1) / kAdamThreads;
  count_launch();
  k_adam<V><<<(unsigned)blocks, kAdamThreads, 0, stream>>>(
      params, grads, m, v, N, S, scalars, zero_grads, screen_gradient, visible_count,
      acc_gradient, acc_views, skip, position_scale, rot_blocks, groups);
}

void launch_adam_rows(float* params, float* grads, float* m, float* v, int N, int S,
                      const StepScalars* scalars, int zero_grads, float* screen_gradient,
                      int32_t* visible_count, float* acc_gradient, int32_t* acc_views,
                      const int32_t* skip, cudaStream_t stream, const float* position_scale) {
  const int rot_blocks = (N + kAdamThreads - 1) / kAdamThreads;
  const int64_t groups = (10 + 3 * (int64_t)S) * (N / 4);
  count_launch();
  k_adam_rows<<<(unsigned)(rot_blocks + (groups + kAdamThreads - 1) / kAdamThreads),
                kAdamThreads, 0, stream>>>(params, grads, m, v, N, S, scalars, zero_grads,
                                           screen_gradient, visible_count, acc_gradient,
                                           acc_views, skip, position_scale, rot_blocks);
}

template <typename... Args>
void launch_adam_kernel(float* params, float* grads, float* m, float* v, int N, int S,
                        Args... args) {
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  const bool wide = aligned(params) && aligned(grads) && aligned(m) && aligned(v);
  if (wide && N % 4 == 0)
    launch_adam_rows(params, grads, m, v, N, S, args...);
  else if (wide)
    launch_adam_groups<4>(params, grads, m, v, N, S, args...);
  else
    launch_adam_groups<1>(params, grads, m, v, N, S, args...);
}

}  // namespace

void launch_adam(float* params, float* grads, float* m, float* v, int N, int S,
                 const StepScalars* scalars, int zero_grads, float* screen_gradient,
                 int32_t* visible_count, float* acc_gradient, int32_t* acc_views,
                 cudaStream_t stream, const float* position_scale) {
  if (N <= 0) return;
  launch_adam_kernel(params, grads, m, v, N, S, scalars, zero_grads, screen_gradient,
                     visible_count, acc_gradient, acc_views, static_cast<const int32_t*>(nullptr),
                     stream, position_scale);
}

void launch_adam_checked(float* params, float* grads, float* m, float* v, int N, int S,
                         const StepScalars* scalars, float* screen_gradient,
                         int32_t* visible_count, float* acc_gradient, int32_t* acc_views,
                         const int32_t* skip, cudaStream_t stream,
                         const float* position_scale) {
  if (N <= 0) return;
  launch_adam_kernel(params, grads, m, v, N, S, scalars, 1, screen_gradient, visible_count,
                     acc_gradient, acc_views, skip, stream, position_scale);
}

// resetOpacity (SplatTrainer.cpp:301-309): cap the logit, clear its moments.
__global__ void k_reset_opacity(float* __restrict__ params, float* __restrict__ m,
                                float* __restrict__ v, int N, float ceiling) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= N) return;
  const int64_t i = (int64_t)PXS_C_OPACITY * N + g;
  const float x = params[i];
  params[i] = ceiling < x ? ceiling : x;  // std::min(x, ceiling)
  m[i] = 0.f;
  v[i] = 0.f;
}

void launch_reset_opacity(float* params, float* m, float* v, int N, float ceiling,
                          cudaStream_t stream) {
  if (N > 0) {
    count_launch();
    k_reset_opacity<<<(N + 255) / 256, 256, 0, stream>>>(params, m, v, N, ceiling);
  }
}

}  // namespace pxs

namespace pxs {

// The data-parallel reduction block's small parts (see pxs_trainer_accumulate):
// the visible counts as floats (exact for counts below 2^24) and the loss tail
// (mean loss x views, views), so one collective sums everything.
__global__ void k_pack_reduction(const int32_t* __restrict__ visible, float* __restrict__ visible_f,
                                 int N, const float* __restrict__ loss_mean, int n_views,
                                 float* __restrict__ tail) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g < N) visible_f[g] = (float)visible[g];
  if (g == 0) {
    tail[0] = loss_mean[0] * (float)n_views;
    tail[1] = (float)n_views;
  }
}

__global__ void k_unpack_visible(const float* __restrict__ visible_f,
                                 int32_t* __restrict__ visible, int N) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g < N) visible[g] = (int32_t)rintf(visible_f[g]);
}

void launch_pack_reduction(const int32_t* visible, float* visible_f, int N,
                           const float* loss_mean, int n_views, float* tail,
                           cudaStream_t stream) {
  count_launch();
  k_pack_reduction<<<(std::max(N, 1) + 255) / 256, 256, 0, stream>>>(visible, visible_f, N,
                                                                     loss_mean, n_views, tail);
}

void launch_unpack_visible(const float* visible_f, int32_t* visible, int N, cudaStream_t stream) {
  if (N <= 0) return;
  count_launch();
  k_unpack_visible<<<(N + 255) / 256, 256, 0, stream>>>(visible_f, visible, N);
}

}  // namespace pxs
