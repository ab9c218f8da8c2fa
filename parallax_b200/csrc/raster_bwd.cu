// raster_bwd.cu -- the adjoint of front-to-back compositing.
//
// rasterizeSplatsBackward, pixel pass (SplatRaster.cpp:346-433): each pixel
// walks its tile's list back to front from its last contributor (recorded by
// the forward kernel), dividing the transmittance back out rather than storing
// it per pair, and the per-splat screen-space gradients are summed over the
// tile's pixels (ScreenGrad):
//   * per warp and two entries at a time with a 21-shuffle transpose reduction
//     (warp_reduce);
//   * once per (warp, splat) into global memory: each of eleven lanes holds one
//     complete sum and adds it to its float of the slot's accumulators, one
//     reduction instruction for both entries.
// The branch decisions (power > 0, the alpha floor, the 0.99 cap) are taken
// with the forward kernel's exact rounding (raster_common.cuh); the gradient
// arithmetic itself may use fused multiply-adds.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "raster_common.cuh"

namespace pxs {
namespace {

constexpr unsigned kFull = 0xffffffffu;
// Fire-and-forget global addition.
__device__ __forceinline__ void red_add(float* address, float x) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(address), "f"(x) : "memory");
}

// One entry's sums over a lane's pixels (ScreenGrad): z; z u^2, z u w, z w^2;
// z u, z w; the colour gradient; |dmean|.
struct LaneSums {
  float z, uu, uw, ww, u, w, c0, c1, c2, ab;
};

// Where a lane's result of warp_reduce belongs: the float of the slot's
// ScreenGrad, or -1. Lanes 0-15 hold entry A's sums, lanes 16-31 entry B's.
__device__ __forceinline__ int sum_index(int lane) {
  const bool b3 = lane & 8, b2 = lane & 4, b1 = lane & 2, b0 = lane & 1;
  if (b0 && b1) return -1;
  if (!b2) return (b3 ? 5 : 0) + (b0 ? 4 : b1 ? 2 : 0);
  return b0 ? (b3 ? 10 : -1) : (b3 ? 5 : 0) + (b1 ? 3 : 1);
}

// Sums a warp's LaneSums of two entries A and B into the eleven accumulators of
// each one's slot. The halves of the warp take one entry each, then lanes 8, 4,
// 2 and 1 apart split what is left of its ten sums: 21 shuffles for the two
// entries, against 24 for one reduction of ten values each, in the latency of
// one. The touched flags need no sum; lane 13 of each half carries them.
__device__ __forceinline__ float warp_reduce(const LaneSums& a, float toucheda,
                                             const LaneSums& b, float touchedb, int lane) {
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4, b1 = lane & 2, b0 = lane & 1;
  auto split = [&](bool upper, int apart, float x, float y) {
    return (upper ? y : x) + __shfl_xor_sync(kFull, upper ? x : y, apart);
  };
  auto half = [&](float x, float y) { return split(b4, 16, x, y); };
  // accumulators 0-4 to the lanes without bit 3, 5-9 to those with it
  const float x0 = split(b3, 8, half(a.z, b.z), half(a.w, b.w));
  const float x1 = split(b3, 8, half(a.uu, b.uu), half(a.c0, b.c0));
  const float x2 = split(b3, 8, half(a.uw, b.uw), half(a.c1, b.c1));
  const float x3 = split(b3, 8, half(a.ww, b.ww), half(a.c2, b.c2));
  const float x4 = split(b3, 8, half(a.u, b.u), half(a.ab, b.ab));
  const float y0 = split(b2, 4, x0, x1), y1 = split(b2, 4, x2, x3);
  const float y2 = x4 + __shfl_xor_sync(kFull, x4, 4);
  const float r0 = split(b1, 2, y0, y1), r1 = y2 + __shfl_xor_sync(kFull, y2, 2);
  const float t = split(b0, 1, r0, r1);
  return (lane & 15) == 13 ? (b4 ? touchedb : toucheda) : t;
}

// Two entries' sums into their slots' accumulators, by the whole warp; `index`
// is the lane's sum_index. (Entries that a single lane takes once had a path
// of their own, without the reduction; finding them cost more than it saved.)
__device__ __forceinline__ void add_entries(ScreenGrad* slot_a, const LaneSums& a, bool toucheda,
                                            ScreenGrad* slot_b, const LaneSums& b, bool touchedb,
                                            int lane, int index) {
  const float any_a = __any_sync(kFull, toucheda) ? 1.f : 0.f;
  const float any_b = __any_sync(kFull, touchedb) ? 1.f : 0.f;
  const float sum = warp_reduce(a, any_a, b, any_b, lane);
  float* dst = reinterpret_cast<float*>(lane < 16 ? slot_a : slot_b);
  if (index >= 0) red_add(dst + index, sum);
}

// The same for one entry.
__device__ __forceinline__ void add_entry(ScreenGrad* slot, const LaneSums& v, bool touched,
                                          int lane, int index) {
  const LaneSums none = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const float any = __any_sync(kFull, touched) ? 1.f : 0.f;
  const float sum = warp_reduce(v, any, none, 0.f, lane);
  if (index >= 0 && lane < 16) red_add(reinterpret_cast<float*>(slot) + index, sum);
}

}  // namespace

template <int PX>
__global__ void __launch_bounds__(TileGeom<PX>::kThreads)
    k_backward(const int2* __restrict__ ranges, const uint32_t* __restrict__ pair_slots,
               const SlotGeom* __restrict__ geom,
               const float4* __restrict__ color, const ViewDesc* __restrict__ views,
               int n_views, const float* __restrict__ T_final,
               const int32_t* __restrict__ last_in, const float* __restrict__ dL_drgb,
               ScreenGrad* __restrict__ screen) {
  constexpr int kThreads = TileGeom<PX>::kThreads;
  __shared__ uint32_t s_slot[kBatch];
  __shared__ float2 s_xy[kBatch];
  __shared__ float4 s_co[kBatch];
  __shared__ float4 s_col[kBatch];  // r, g, b, power floor
  __shared__ uint32_t s_mask[kBatch];
  __shared__ int s_hi;
  const TileInfo<PX> info = tile_info<PX>(views, n_views, ranges);
  const ViewDesc& vd = views[info.view];
  const float min_alpha = vd.min_alpha;
  const float fx = (float)info.px + 0.5f;
  const float bg0 = vd.background[0], bg1 = vd.background[1], bg2 = vd.background[2];
  // per pixel: dL/drgb, the running transmittance, the last contributor, and
  // the colour behind the current entry against dL/drgb: the adjoint only needs
  // the suffix colour (the reference's accum_rec) through that product, and
  // starting it at the background's accounts for the background's share
  float fy[PX], dLp0[PX], dLp1[PX], dLp2[PX], T[PX], behind[PX];
  int my_last[PX];
  int thread_hi = info.range.x;
#pragma unroll
  for (int p = 0; p < PX; ++p) {
    const int py = info.py0 + p;
    fy[p] = (float)py + 0.5f;
    dLp0[p] = dLp1[p] = dLp2[p] = 0.f;
    T[p] = 1.f;
    my_last[p] = info.range.x;
    if (info.px < vd.cam.width && py < vd.cam.height) {
      const int64_t pixel = vd.pixel_offset + (int64_t)py * vd.cam.width + info.px;
      dLp0[p] = dL_drgb[pixel * 3 + 0];
      dLp1[p] = dL_drgb[pixel * 3 + 1];
      dLp2[p] = dL_drgb[pixel * 3 + 2];
      T[p] = T_final[pixel];
      my_last[p] = last_in[pixel];
    }
    behind[p] = bg0 * dLp0[p] + bg1 * dLp1[p] + bg2 * dLp2[p];
    thread_hi = max(thread_hi, my_last[p]);
  }
  const int lane = lane_id(), warp = warp_id(), index = sum_index(lane_id());
  const int warp_hi = __reduce_max_sync(kFull, thread_hi);
  if (threadIdx.x == 0) s_hi = info.range.x;
  __syncthreads();
  if (lane == 0 && warp_hi > info.range.x) atomicMax(&s_hi, warp_hi);
  __syncthreads();
  const int hi = s_hi;

  for (int batch_end = hi; batch_end > info.range.x; batch_end -= kBatch) {
    const int batch_start = max(info.range.x, batch_end - kBatch);
    const int n = batch_end - batch_start;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kThreads) {
      const uint32_t slot = pair_slots[batch_start + i];
      const float4 co = geom[slot].conic_op;
      const float2 mean = geom[slot].xy;
      float4 c = color[slot];
      c.w = power_floor(co.w, min_alpha);
      s_slot[i] = slot;
      s_xy[i] = mean;
      s_co[i] = co;
      s_col[i] = c;
      s_mask[i] = warp_mask<PX>(mean, co, c.w, info.tile_px, info.tile_py);
    }
    __syncthreads();
    const int j_top = min(n, warp_hi - batch_start) - 1;  // warp-uniform
    for (int j = j_top; j >= 0; --j) {
      if (!((s_mask[j] >> warp) & 1u)) continue;  // the splat cannot reach this warp's pixels
      const int e = batch_start + j;
      const float2 m = s_xy[j];
      const float4 co = s_co[j];
      const float4 c = s_col[j];
      const float dx = fx - m.x;
      LaneSums v = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      bool contrib = false, touched = false;
#pragma unroll
      for (int p = 0; p < PX; ++p) {
        if (e < my_last[p]) {
          const float dy = fy[p] - m.y;
          const float power = splat_power(co, dx, dy);
          if (!(power > 0.f) && !(power < c.w)) {
            const float raw_alpha = __fmul_rn(co.w, splat_exp(power));
            const float alpha = raw_alpha < kMaxAlpha ? raw_alpha : kMaxAlpha;
            if (!(alpha < min_alpha)) {
              contrib = true;
              T[p] *= rcp_approx_ftz(1.f - alpha);
              const float weight = alpha * T[p];
              v.c0 += weight * dLp0[p];
              v.c1 += weight * dLp1[p];
              v.c2 += weight * dLp2[p];
              // the colour minus what lies behind, against dL/drgb
              const float d = c.x * dLp0[p] + c.y * dLp1[p] + c.z * dLp2[p] - behind[p];
              behind[p] += alpha * d;
              if (raw_alpha < kMaxAlpha) {  // the cap flattens the gradient
                touched = true;
                const float z = raw_alpha * (d * T[p]);
                const float u = co.x * dx + co.y * dy, w = co.y * dx + co.z * dy;
                const float zu = z * u, zw = z * w;
                v.z += z;
                v.uu += zu * u;
                v.uw += zu * w;
                v.ww += zw * w;
                v.u += zu;
                v.w += zw;
                v.ab += sqrt_approx_ftz(zu * zu + zw * zw);
              }
            }
          }
        }
      }
      if (__any_sync(kFull, contrib))
        add_entry(&screen[s_slot[j]], v, touched, lane, index);
    }
  }
}

// Warp w's bit in a tile-list entry's mask for the adjoint with PX pixels per
// thread, from the forward's block bits (bit b: some pixel of 8x8 block b of
// the two-pixel layout took the entry). With four pixels per thread warp w
// covers the two-pixel blocks w and w + 2.
template <int PX>
__device__ __forceinline__ uint32_t mask_from_block_bits(uint32_t bits) {
  if constexpr (PX == 2) return bits;
  else return (bits | (bits >> 2)) & 3u;
}

// The paired-FP32 forms of k_backward, with NP pairs of vertically adjacent
// pixels per thread (NP = 1: two pixels, 8x8 blocks per warp; NP = 2: four
// pixels, 8x16 blocks). The gradient arithmetic of a pair runs as the halves
// of paired FP32 instructions (fma/add/mul .f32x2). The branch decisions are
// the forward's, from operations that round as its own (splat_power2, alpha
// = opacity * exp). The body has no branches on them: a pixel that does not
// take an entry runs the paired arithmetic with alpha = 0, so its transmittance
// (multiplied by 1), what lies behind it and its sums are unchanged; almost
// every warp has some lane that takes the entry, so branching around the
// arithmetic only added divergence handling. A thread adds its pairs'
// contributions before the warp reduction, so one reduction serves 2 NP pixels
// per lane.
//
// The kernel is bound by instruction issue (77% of cycles over whole waves,
// ALU pipe 56%, FMA 44%), so its cost is instructions per entry and warp, about
// 208 of them when ten gradients per pixel were formed, reduced entry by entry
// and added with shared-memory atomics (a compare-and-swap loop for floats):
//   - the conic and opacity factors once per slot (ScreenGrad), the colour
//     behind as its product with dL/drgb, sums straight to global memory;
//   - two entries per reduction, which also halves the reduction's latency
//     where few warps hide it (small images).
// 7.02 -> 4.69 ms per step of 8 views of 1920x1440 with 1M gaussians, 4.18 ->
// 2.81 ms over 40 views of ten small scenes, 0.131 -> 0.072 ms for one 320x240
// view of 20k. Summing z, z d, z d^T d instead (seven lane sums, dx applied
// once per column) ran in 4.39 ms but lost precision in elongated splats
// (ScreenGrad). 56 registers since each tile schedule has its own kernel: 4.50 ms
// (for_each_tile); held to 48 (10 CTAs per SM) 4.57.
// kB entries are staged per batch (RasterConfig::backward_batch: 64, 128 or
// 256 with two pixels per thread; 128 with four, where fewer threads share a
// batch); kPersist and `order` map CTAs to tiles (for_each_tile).
template <int NP, int kB, bool kBits, bool kPersist>
__global__ void __launch_bounds__(TileGeom<2 * NP>::kThreads)
    k_backward_pairs(const int2* __restrict__ ranges, const uint32_t* __restrict__ pair_slots,
                     const SlotGeom* __restrict__ geom,
                     const float4* __restrict__ color, const ViewDesc* __restrict__ views,
                     int n_views, const float* __restrict__ T_final,
                     const int32_t* __restrict__ last_in, const float* __restrict__ dL_drgb,
                     ScreenGrad* __restrict__ screen, const uint8_t* __restrict__ block_bits,
                     const int* __restrict__ order, int* __restrict__ ticket,
                     int total_tiles) {
  constexpr int PX = 2 * NP;
  constexpr int kThreads = TileGeom<PX>::kThreads;
  constexpr int kWarps = TileGeom<PX>::kWarps;
  __shared__ uint32_t s_slot[kB];
  __shared__ float2 s_xy[kB];  // -mean
  __shared__ float4 s_co[kB];  // conic, -opacity
  __shared__ float4 s_col[kB];  // r, g, b (w unused)
  __shared__ uint32_t s_mask[kB];
  __shared__ uint8_t s_list[kWarps][kB];  // a warp's entries of the batch
  __shared__ int s_hi;
  static_assert(kB <= 256, "batch indices are bytes");
  for_each_tile<kPersist>(order, ticket, total_tiles, [&](int tile) {
  const TileInfo<PX> info = tile_info<PX>(views, n_views, ranges, tile);
  const ViewDesc& vd = views[info.view];
  const float min_alpha = vd.min_alpha;
  const float fx = (float)info.px + 0.5f;
  // (no alpha reaches a floor above the cap)
  const float neg_min_alpha = min_alpha > kMaxAlpha ? -INFINITY : -min_alpha;
  const float2 zero2 = make_float2(0.f, 0.f);
  // per pixel: -dL/drgb, the running transmittance, the last contributor, and
  // the colour behind the current entry against dL/drgb (see k_backward)
  float2 fy[NP], nL0[NP], nL1[NP], nL2[NP], T[NP], behind[NP];
  int last0[NP], last1[NP];
  int hi_mine = info.range.x;
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    const int py = info.py0 + 2 * q;
    fy[q] = make_float2((float)py + 0.5f, (float)(py + 1) + 0.5f);
    nL0[q] = nL1[q] = nL2[q] = zero2;
    T[q] = make_float2(1.f, 1.f);
    last0[q] = last1[q] = info.range.x;
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      if (info.px < vd.cam.width && py + p < vd.cam.height) {
        const int64_t pixel = vd.pixel_offset + (int64_t)(py + p) * vd.cam.width + info.px;
        const float d0 = -dL_drgb[pixel * 3 + 0], d1 = -dL_drgb[pixel * 3 + 1];
        const float d2 = -dL_drgb[pixel * 3 + 2], tf = T_final[pixel];
        const int l = last_in[pixel];
        if (p == 0) {
          nL0[q].x = d0; nL1[q].x = d1; nL2[q].x = d2; T[q].x = tf; last0[q] = l;
        } else {
          nL0[q].y = d0; nL1[q].y = d1; nL2[q].y = d2; T[q].y = tf; last1[q] = l;
        }
      }
    }
    const float b0 = -vd.background[0], b1 = -vd.background[1], b2 = -vd.background[2];
    behind[q] = __ffma2_rn(make_float2(b2, b2), nL2[q],
                           __ffma2_rn(make_float2(b1, b1), nL1[q],
                                      __fmul2_rn(make_float2(b0, b0), nL0[q])));
    hi_mine = max(hi_mine, max(last0[q], last1[q]));
  }
  const int lane = lane_id(), warp = warp_id(), index = sum_index(lane_id());
  const int warp_hi = __reduce_max_sync(kFull, hi_mine);
  if (threadIdx.x == 0) s_hi = info.range.x;
  __syncthreads();
  if (lane == 0 && warp_hi > info.range.x) atomicMax(&s_hi, warp_hi);
  __syncthreads();
  const int hi = s_hi;

  for (int batch_end = hi; batch_end > info.range.x; batch_end -= kB) {
    const int batch_start = max(info.range.x, batch_end - kB);
    const int n = batch_end - batch_start;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kThreads) {
      const uint32_t slot = pair_slots[batch_start + i];
      const float4 co = geom[slot].conic_op;
      const float2 mean = geom[slot].xy;
      s_slot[i] = slot;
      s_xy[i] = make_float2(-mean.x, -mean.y);  // negated: fx + (-mx) is fx - mx
      s_co[i] = make_float4(co.x, co.y, co.z, -co.w);
      s_col[i] = color[slot];
      // which warps took the entry in the forward pass (exact), else which
      // ones its footprint can reach
      s_mask[i] = kBits
                      ? mask_from_block_bits<PX>(block_bits[batch_start + i])
                      : warp_mask<PX>(mean, co, power_floor(co.w, min_alpha), info.tile_px,
                                      info.tile_py);
    }
    __syncthreads();
    const int j_top = min(n, warp_hi - batch_start) - 1;  // warp-uniform
    // the entries some pixel of this warp takes (or can reach), ascending;
    // built by the whole warp, which is converged here
    int n_mine = 0;
    for (int j0 = 0; j0 <= j_top; j0 += 32) {
      const int jj = j0 + lane;
      const bool mine = jj <= j_top && ((s_mask[jj] >> warp) & 1u);
      const unsigned b = __ballot_sync(kFull, mine);
      if (mine) s_list[warp][n_mine + __popc(b & lanemask_lt())] = (uint8_t)jj;
      n_mine += __popc(b);
    }
    __syncwarp();
    // entry j's sums over this lane's pixels; whether a pixel took it, and one
    // below the cap
    auto visit = [&](int j, LaneSums& v, bool& contrib, bool& touched) {
      const int e = batch_start + j;
      const float2 nm = s_xy[j];
      const float4 co = s_co[j];
      const float4 c = s_col[j];
      const float dx = fx + nm.x;
      contrib = touched = false;
      // pair q's sums: assigned by the first pair, added by the next
      auto put = [&](int q, float& to, float x) { to = q == 0 ? x : to + x; };
      const float adx = co.x * dx, bdx = co.y * dx;
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        const float2 dy = add2_rn(fy[q], make_float2(nm.y, nm.y));
        const float2 power = splat_power2(co, dx, dy);
        // no power-floor test: below the floor alpha is certainly under
        // min_alpha, so the alpha test below decides the same
        const bool in0 = e < last0[q] && !(power.x > 0.f);
        const bool in1 = e < last1[q] && !(power.y > 0.f);
        // -opacity exp(power), 0 where the pixel does not take the entry (the
        // opacity is staged negated: the tests are mirrored), then -alpha
        float2 nr = mul2_rn(make_float2(co.w, co.w),
                                  make_float2(splat_exp(power.x), splat_exp(power.y)));
        const bool c0 = in0 && !(nr.x > neg_min_alpha);
        const bool c1 = in1 && !(nr.y > neg_min_alpha);
        contrib = contrib || c0 || c1;
        nr.x = c0 ? nr.x : 0.f;
        nr.y = c1 ? nr.y : 0.f;
        const float2 na = make_float2(nr.x > -kMaxAlpha ? nr.x : -kMaxAlpha,
                                      nr.y > -kMaxAlpha ? nr.y : -kMaxAlpha);
        // where the pixel does not take the entry 1 - alpha is 1, its
        // reciprocal exactly 1, and T stays as it is
        const float2 om = __fadd2_rn(make_float2(1.f, 1.f), na);
        T[q] = __fmul2_rn(T[q], make_float2(rcp_approx_ftz(om.x), rcp_approx_ftz(om.y)));
        const float2 nw = __fmul2_rn(na, T[q]);  // minus the colour weight
        const float2 w0 = __fmul2_rn(nw, nL0[q]);
        const float2 w1 = __fmul2_rn(nw, nL1[q]);
        const float2 w2 = __fmul2_rn(nw, nL2[q]);
        put(q, v.c0, w0.x + w0.y);
        put(q, v.c1, w1.x + w1.y);
        put(q, v.c2, w2.x + w2.y);
        // minus (the colour less what lies behind, SplatRaster.cpp:399-405)
        // against dL/drgb; the entry then joins what lies behind for the
        // entries in front of it: behind += alpha (colour . dL - behind),
        // which leaves a pixel that does not take the entry unchanged
        const float2 nd = __ffma2_rn(
            make_float2(c.z, c.z), nL2[q],
            __ffma2_rn(make_float2(c.y, c.y), nL1[q],
                       __ffma2_rn(make_float2(c.x, c.x), nL0[q], behind[q])));
        behind[q] = __ffma2_rn(na, nd, behind[q]);
        // dL/dpower = opacity exp(power) dL/dalpha; 0 at the 0.99 cap, which
        // flattens the gradient, and outside the pixel's entries (selected, so
        // an exponential that overflowed there does not spread)
        const bool t0 = c0 && nr.x > -kMaxAlpha, t1 = c1 && nr.y > -kMaxAlpha;
        touched = touched || t0 || t1;
        const float2 z = __fmul2_rn(make_float2(t0 ? nr.x : 0.f, t1 ? nr.y : 0.f),
                                    __fmul2_rn(nd, T[q]));
        const float2 u = __ffma2_rn(make_float2(co.y, co.y), dy, make_float2(adx, adx));
        const float2 w = __ffma2_rn(make_float2(co.z, co.z), dy, make_float2(bdx, bdx));
        const float2 zu = __fmul2_rn(z, u), zw = __fmul2_rn(z, w);
        const float2 zuu = __fmul2_rn(zu, u), zuw = __fmul2_rn(zu, w), zww = __fmul2_rn(zw, w);
        put(q, v.z, z.x + z.y);
        put(q, v.uu, zuu.x + zuu.y);
        put(q, v.uw, zuw.x + zuw.y);
        put(q, v.ww, zww.x + zww.y);
        put(q, v.u, zu.x + zu.y);
        put(q, v.w, zw.x + zw.y);
        // |dL/dmean| per pixel, for the densification statistic (a sum compared
        // against a threshold): the square-root approximation. Not |z| |A d|: in a
        // splat of next to no width |A d|^2 overflows at pixels that have z = 0
        const float2 sq = __ffma2_rn(zu, zu, __fmul2_rn(zw, zw));
        put(q, v.ab, sqrt_approx_ftz(sq.x) + sqrt_approx_ftz(sq.y));
      }
    };
    // back to front, two entries at a time (one reduction serves both), then
    // the odd one
    int qi = n_mine - 1;
    for (; qi > 0; qi -= 2) {
      const int ja = s_list[warp][qi], jb = s_list[warp][qi - 1];
      LaneSums va, vb;
      bool ca, cb, ta, tb;
      visit(ja, va, ca, ta);
      visit(jb, vb, cb, tb);
      if (kBits || __any_sync(kFull, ca || cb))
        add_entries(&screen[s_slot[ja]], va, ta, &screen[s_slot[jb]], vb, tb, lane, index);
    }
    if (qi == 0) {
      const int j = s_list[warp][0];
      LaneSums v;
      bool contrib, touched;
      visit(j, v, contrib, touched);
      if (kBits || __any_sync(kFull, contrib))
        add_entry(&screen[s_slot[j]], v, touched, lane, index);
    }
  }
  });
}

namespace {

template <int PX>
void backward_px(const int2* ranges, const uint32_t* pair_slots, const SlotGeom* geom, const float4* color, const ViewDesc* views, int n_views,
                 int total_tiles, const float* T_final, const int32_t* last,
                 const float* dL_drgb, ScreenGrad* screen, cudaStream_t stream) {
  k_backward<PX><<<total_tiles, TileGeom<PX>::kThreads, 0, stream>>>(
      ranges, pair_slots, geom, color, views, n_views, T_final, last, dL_drgb, screen);
}

}  // namespace

template <int NP, int B, bool kBits>
void backward_pairs_launch(const int2* ranges, const uint32_t* pair_slots, const SlotGeom* geom, const float4* color, const ViewDesc* views,
                           int n_views, int total_tiles, const float* T_final,
                           const int32_t* last, const float* dL_drgb, ScreenGrad* screen,
                           cudaStream_t stream, const uint8_t* block_bits,
                           const int* tile_order, int* ticket) {
  const int schedule = tile_order == nullptr ? kTileOrder : raster_config().backward_schedule;
  const int threads = TileGeom<2 * NP>::kThreads;
  if (schedule == kPersistent) {
    const auto persistent = k_backward_pairs<NP, B, kBits, true>;
    cudaMemsetAsync(ticket, 0, sizeof(int), stream);
    persistent<<<std::min(total_tiles, resident_ctas(persistent, threads)), threads, 0, stream>>>(
        ranges, pair_slots, geom, color, views, n_views, T_final, last, dL_drgb, screen,
        block_bits, tile_order, ticket, total_tiles);
  } else {
    k_backward_pairs<NP, B, kBits, false><<<total_tiles, threads, 0, stream>>>(
        ranges, pair_slots, geom, color, views, n_views, T_final, last, dL_drgb, screen,
        block_bits, tile_order, ticket, total_tiles);
  }
}

void launch_backward(const int2* ranges, const uint32_t* pair_slots, const SlotGeom* geom, const float4* color, const ViewDesc* views,
                     int n_views, int total_tiles, const float* T_final, const int32_t* last,
                     const float* dL_drgb, ScreenGrad* screen, cudaStream_t stream,
                     const uint8_t* block_bits, const int* tile_order, int* ticket) {
  if (total_tiles <= 0) return;
  count_launch();
#define PXS_BWD(NP, B)                                                                         \
  (block_bits != nullptr                                                                       \
       ? backward_pairs_launch<NP, B, true>(ranges, pair_slots, geom, color, views,    \
                                            n_views, total_tiles, T_final, last, dL_drgb,      \
                                            screen, stream, block_bits, tile_order, ticket)    \
       : backward_pairs_launch<NP, B, false>(ranges, pair_slots, geom, color, views,   \
                                             n_views, total_tiles, T_final, last, dL_drgb,     \
                                             screen, stream, block_bits, tile_order, ticket))
  switch (raster_config().backward_px) {
    case 1:
      backward_px<1>(ranges, pair_slots, geom, color, views, n_views, total_tiles,
                     T_final, last, dL_drgb, screen, stream);
      break;
    case 4:
      PXS_BWD(2, kBatch / 2);
      break;
    default: {
      const int b = raster_config().backward_batch;
      if (b == 64) PXS_BWD(1, 64);
      else if (b == 128) PXS_BWD(1, 128);
      else PXS_BWD(1, 256);
    }
  }
#undef PXS_BWD
}

}  // namespace pxs
