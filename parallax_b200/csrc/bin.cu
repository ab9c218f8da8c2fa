// bin.cu -- per-tile key lists from the depth-sorted splats, by tile rows.
//
// The reference appends each splat, in depth order, to every 16-px tile its
// 3-sigma box touches (buildTiles, SplatRaster.cpp:104-151), so a tile's list
// is near to far. Sorting the (tile, splat) pairs themselves moves every pair
// through memory once per radix pass. Here the rectangle structure is used
// instead:
//   1. each visible splat has one record per tile row it covers (about one
//      seventh as many as pairs), wanted grouped by row and near to far
//      within a row: each view's depth-sorted slots are cut into chunks of
//      1024; a CTA per chunk counts, per tile row, the splats covering it; an
//      exclusive scan of the counts in (row, chunk) order gives each chunk
//      its base in each row, and the chunk writes its records there (as in
//      step 3 with rows for columns) -- a stable counting sort by row with no
//      sort pass;
//   2. each row is cut into chunks of 1024 records; one CTA per chunk counts,
//      per column, the records covering it; a per-row pass turns those into
//      each chunk's base within every tile of the row and the tiles' lengths;
//      an exclusive scan over the tiles gives the tile ranges;
//   3. one CTA per chunk sets its records' bits in a 1024-bit map per column; a
//      pair's place in its tile's list is the chunk's base plus the number of
//      earlier bits of the column.
// Images of few tiles skip the rows (Frame::direct_lists).
// Over the splats' 3-sigma squares (Frame::project's whole_lists, for
// pxs_tile_lists) the result -- ranges and slot lists -- is exactly the
// reference's, with equal depths in gaussian order (the depth sort is stable over
// slots). The steps and images instead list only the tiles a splat can reach
// (raster_common.cuh: splat_footprint for its box, row_columns per tile row): the
// same pixels take the same entries, from lists about half as long (29 against
// 54 tiles per splat at 1920x1440 in clouds of 1M, 15 against 26 at 1280x720).
// With 8 views of 1M gaussians at 1920x1440 binning went from 2.76 to 2.38 ms,
// compositing, which stages the entries, from 2.63 to 2.27, its adjoint from
// 4.70 to 4.60.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "raster_common.cuh"

namespace pxs {
namespace {

constexpr int kWarps = 8;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ int view_of_row(const ViewDesc* __restrict__ views, int n_views,
                                           int row) {
  int v = 0;
  while (v + 1 < n_views && views[v + 1].row_offset <= row) ++v;
  return v;
}

}  // namespace

// Rows are cut into chunks of at most kChunk records so the work balances
// whatever the rows' lengths. Row r's records are [offsets[r * cpv],
// offsets[(r + 1) * cpv]) (the total for the last row), clamped to the capacity;
// records past it raise the overflow flag. chunks[c] = (row, begin, end);
// n_chunks[0] is the count. One CTA builds the table, 1024 rows at a time: a
// block-wide scan over the rows' chunk counts, then a chunk per thread.
constexpr int kChunk = 1024;
constexpr int kPerLane = kChunk / (kWarps * 32);  // records per lane per chunk

__global__ void __launch_bounds__(1024)
    k_row_chunks(const int64_t* __restrict__ offsets, int cpv, const int64_t* __restrict__ total,
                 int64_t capacity, int total_rows, int max_chunks, int4* __restrict__ chunks,
                 int32_t* __restrict__ n_chunks, int32_t* __restrict__ overflow) {
  __shared__ int warp_sums[32];
  __shared__ int first[1024], begin[1024], end[1024];
  const int t = threadIdx.x;
  int carry = 0;
  for (int base = 0; base < total_rows; base += 1024) {
    const int row = base + t;
    int64_t b = 0, e = 0;
    if (row < total_rows) {
      b = offsets[(int64_t)row * cpv];
      e = row + 1 < total_rows ? offsets[(int64_t)(row + 1) * cpv] : *total;
      if (e > capacity) atomicExch(overflow, 1);
      b = min(b, capacity);
      e = min(e, capacity);
    }
    begin[t] = (int)b;
    end[t] = (int)e;
    const int count = (int)((e - b + kChunk - 1) / kChunk);
    int x = count;  // block-wide inclusive scan
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(kFull, x, o);
      if (lane_id() >= o) x += n;
    }
    if (lane_id() == 31) warp_sums[warp_id()] = x;
    __syncthreads();
    if (warp_id() == 0) {
      int y = warp_sums[lane_id()];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(kFull, y, o);
        if (lane_id() >= o) y += n;
      }
      warp_sums[lane_id()] = y;
    }
    __syncthreads();
    first[t] = (warp_id() > 0 ? warp_sums[warp_id() - 1] : 0) + x - count;
    const int n = warp_sums[31];
    __syncthreads();
    for (int c = t; c < n && carry + c < max_chunks; c += 1024) {
      // the last row whose first chunk is at or before c (a row without chunks
      // shares its first with the next one)
      int lo = 0, hi = 1023;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (first[mid] <= c) lo = mid;
        else hi = mid - 1;
      }
      const int from = begin[lo] + (c - first[lo]) * kChunk;
      chunks[carry + c] = make_int4(base + lo, from, min(end[lo], from + kChunk), 0);
    }
    carry += n;
    __syncthreads();
  }
  if (t == 0) n_chunks[0] = min(carry, max_chunks);
}

// Per-warp counts of the lanes' ranges range[k] = lo | hi << 16 (empty when
// hi < lo) over the columns of `row` (zeroed by the caller, `extent` wide):
// each range adds +1 at lo and -1 past hi (two shared-memory atomics however
// wide it is), then the warp prefix-sums its row.
template <int K>
__device__ __forceinline__ void warp_range_counts(const uint32_t (&range)[K], int extent,
                                                  int32_t* row) {
  const int lane = lane_id();
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int lo = range[k] & 0xFFFF, hi = range[k] >> 16;
    if (hi >= lo) {
      atomicAdd(&row[lo], 1);
      if (hi + 1 < extent) atomicAdd(&row[hi + 1], -1);
    }
  }
  __syncwarp();
  int carry = 0;
  for (int c0 = 0; c0 < extent; c0 += 32) {
    const int c = c0 + lane;
    int v = c < extent ? row[c] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(kFull, v, o);
      if (lane >= o) v += n;
    }
    if (c < extent) row[c] = carry + v;
    carry += __shfl_sync(kFull, v, 31);
  }
  __syncwarp();
}

// Per-warp column counts of one chunk of row records into s_cnt
// [kWarps][max_tiles_x] (zeroed by the caller). Each record's column range
// was stored beside it when the records were written (rec_xr), so it is read
// with the record instead of gathered through the record's slot.
__device__ __forceinline__ void chunk_column_counts(const int4& ch, const uint32_t* __restrict__ rec_slots,
                                                    const uint32_t* __restrict__ rec_xr, int max_tiles_x,
                                                    int tiles_x, int32_t* s_cnt,
                                                    uint32_t (&slot)[kPerLane],
                                                    uint32_t (&xr)[kPerLane]) {
  const int w = warp_id(), lane = lane_id();
  const int w_begin = ch.y + w * (kChunk / kWarps);
#pragma unroll
  for (int k = 0; k < kPerLane; ++k) {
    const int rec = w_begin + k * 32 + lane;
    slot[k] = 0u;
    xr[k] = 1u;  // x0 = 1 > x1 = 0: covers nothing
    if (rec < ch.z) {
      slot[k] = rec_slots[rec];
      xr[k] = rec_xr[rec];
    }
  }
  warp_range_counts(xr, tiles_x, s_cnt + w * max_tiles_x);
}

// Per chunk: how many of its records cover each column.
__global__ void __launch_bounds__(kWarps * 32)
    k_chunk_counts(const int4* __restrict__ chunks, const int32_t* __restrict__ n_chunks,
                   const uint32_t* __restrict__ rec_slots, const uint32_t* __restrict__ rec_xr,
                   const ViewDesc* __restrict__ views, int n_views, int max_tiles_x,
                   int32_t* __restrict__ chunk_counts) {
  extern __shared__ int32_t s_cnt[];  // [kWarps][max_tiles_x]
  if ((int)blockIdx.x >= n_chunks[0]) return;
  const int4 ch = chunks[blockIdx.x];
  const ViewDesc& vd = views[view_of_row(views, n_views, ch.x)];
  const int tiles_x = vd.tiles_x;
  for (int i = threadIdx.x; i < kWarps * tiles_x; i += blockDim.x)
    s_cnt[(i / tiles_x) * max_tiles_x + (i % tiles_x)] = 0;
  __syncthreads();
  uint32_t slot[kPerLane], xr[kPerLane];
  chunk_column_counts(ch, rec_slots, rec_xr, max_tiles_x, tiles_x, s_cnt, slot, xr);
  __syncthreads();
  for (int c = threadIdx.x; c < tiles_x; c += blockDim.x) {
    int total = 0;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) total += s_cnt[k * max_tiles_x + c];
    chunk_counts[(int64_t)blockIdx.x * max_tiles_x + c] = total;
  }
}

// Per row: each chunk's base within each tile of the row (exclusive over the
// row's chunks, in order) and the tile's length. The row's chunks are
// consecutive in the table, found from the first one by a binary search.
__global__ void __launch_bounds__(256)
    k_row_tiles(const int4* __restrict__ chunks, const int32_t* __restrict__ n_chunks,
                const ViewDesc* __restrict__ views, int n_views, int max_tiles_x,
                const int32_t* __restrict__ chunk_counts, int32_t* __restrict__ chunk_base,
                int32_t* __restrict__ tile_counts) {
  const int row = blockIdx.x;
  const int v = view_of_row(views, n_views, row);
  const ViewDesc& vd = views[v];
  const int tiles_x = vd.tiles_x;
  const int nc = n_chunks[0];
  // first chunk with chunks[c].x >= row
  int lo = 0, hi = nc;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (chunks[mid].x < row) lo = mid + 1;
    else hi = mid;
  }
  const int first = lo;  // then the first past the row
  for (hi = nc; lo < hi;) {
    const int mid = (lo + hi) >> 1;
    if (chunks[mid].x <= row) lo = mid + 1;
    else hi = mid;
  }
  const int64_t tile0 = (int64_t)vd.tile_offset + (int64_t)(row - vd.row_offset) * tiles_x;
  for (int c = threadIdx.x; c < tiles_x; c += blockDim.x) {
    int run = 0;
#pragma unroll 8
    for (int k = first; k < lo; ++k) {
      const int t = chunk_counts[(int64_t)k * max_tiles_x + c];
      chunk_base[(int64_t)k * max_tiles_x + c] = run;
      run += t;
    }
    tile_counts[tile0 + c] = run;
  }
}

// ranges[t] = [offset, offset + count); a tile whose list would pass the pair
// capacity is left empty and raises the overflow flag.
__global__ void k_ranges_from_offsets(const int32_t* __restrict__ counts,
                                      const int64_t* __restrict__ offsets, int64_t n_tiles,
                                      int64_t capacity, int2* __restrict__ ranges,
                                      int32_t* __restrict__ overflow) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tiles) return;
  const int64_t begin = offsets[t], end = begin + counts[t];
  if (end > capacity) {
    ranges[t] = make_int2(0, 0);
    atomicExch(overflow, 1);
  } else {
    ranges[t] = make_int2((int)begin, (int)end);
  }
}

// Writes each chunk's records into its row's tile lists, in record (depth)
// order. The chunk's records are 1024 bits per column, 32 words: a record sets its
// bit in each of its columns, then a half warp per column, two words per lane,
// counts the words' bits, scans the counts and writes the set bits' slots from
// the column's base on. Wider images go kMapCols columns at a time.
//
// Bound by instructions. Ranking 32 records at a time in per-warp bitmaps, staging
// the pairs in shared memory by column and copying them out took 3.6 warp
// instructions per pair and 1.06 ms for 8 views of 1M gaussians at 1920x1440 (228M
// pairs); this form 0.75 ms, and 0.83 with the lanes kept together by a vote per bit.
constexpr int kMapCols = 512;
constexpr int kMapWords = kChunk / 32;
static_assert(kMapWords == 32, "two words per lane of a half warp");

__global__ void __launch_bounds__(kWarps * 32)
    k_chunk_expand(const int4* __restrict__ chunks, const int32_t* __restrict__ n_chunks,
                   const uint32_t* __restrict__ rec_slots, const uint32_t* __restrict__ rec_xr,
                   const ViewDesc* __restrict__ views, int n_views, int max_tiles_x,
                   const int32_t* __restrict__ chunk_base,
                   const int64_t* __restrict__ tile_offsets, int64_t capacity,
                   uint32_t* __restrict__ tile_slots) {
  extern __shared__ uint32_t s_map[];  // [kMapWords][pitch], an odd pitch
  __shared__ uint32_t s_slot[kChunk];
  __shared__ uint32_t s_dst[kMapCols];  // each column's first list position
  if ((int)blockIdx.x >= n_chunks[0]) return;
  const int4 ch = chunks[blockIdx.x];
  const ViewDesc& vd = views[view_of_row(views, n_views, ch.x)];
  const int tiles_x = vd.tiles_x;
  const int w = warp_id(), lane = lane_id();
  uint32_t xr[kPerLane];
#pragma unroll
  for (int k = 0; k < kPerLane; ++k) {
    const int i = w * (kChunk / kWarps) + k * 32 + lane, rec = ch.y + i;
    xr[k] = 1u;  // 1 > 0: covers nothing
    if (rec < ch.z) {
      s_slot[i] = rec_slots[rec];
      xr[k] = rec_xr[rec];
    }
  }
  const int64_t tile0 = (int64_t)vd.tile_offset + (int64_t)(ch.x - vd.row_offset) * tiles_x;
  const uint32_t cap = (uint32_t)capacity;  // at most 2^31 - 1
  for (int c0 = 0; c0 < tiles_x; c0 += kMapCols) {
    const int cols = min(kMapCols, tiles_x - c0);
    const int pitch = cols | 1;
    for (int i = threadIdx.x; i < kMapWords * pitch; i += blockDim.x) s_map[i] = 0u;
    // list positions in 32 bits: nothing past the capacity is written
    for (int c = threadIdx.x; c < cols; c += blockDim.x)
      s_dst[c] = (uint32_t)min(
          tile_offsets[tile0 + c0 + c] + chunk_base[(int64_t)blockIdx.x * max_tiles_x + c0 + c],
          capacity);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kPerLane; ++k) {
      uint32_t* row = s_map + (w * kPerLane + k) * pitch;
      const int lo = max((int)(xr[k] & 0xFFFF) - c0, 0);
      const int hi = min((int)(xr[k] >> 16) - c0, cols - 1);
      for (int c = lo; c <= hi; ++c) atomicOr(&row[c], 1u << lane);
    }
    __syncthreads();
    const int half = lane >> 4, i = lane & 15;
    for (int cc = 2 * w; cc < cols; cc += 2 * kWarps) {
      const int c = cc + half;
      uint32_t m0 = 0u, m1 = 0u, at = 0u;
      if (c < cols) {
        m0 = s_map[2 * i * pitch + c];
        m1 = s_map[(2 * i + 1) * pitch + c];
        at = s_dst[c];
      }
      const int n = __popc(m0) + __popc(m1);
      int x = n;
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {
        const int y = __shfl_up_sync(kFull, x, o, 16);
        if (i >= o) x += y;
      }
      at += (uint32_t)(x - n);
      const uint32_t* slots = s_slot + 64 * i;
      while (m0 != 0u) {
        if (at < cap) tile_slots[at] = slots[__ffs(m0) - 1];
        m0 &= m0 - 1u;
        ++at;
      }
      __syncwarp();
      slots += 32;
      while (m1 != 0u) {
        if (at < cap) tile_slots[at] = slots[__ffs(m1) - 1];
        m1 &= m1 - 1u;
        ++at;
      }
    }
    if (c0 + kMapCols < tiles_x) __syncthreads();  // the map is read before it is cleared
  }
}

// ------------------------------------------------------------ tile-row records
//
// The records -- one (tile row, slot) per row a visible splat covers -- are
// wanted grouped by row (rows of every view one after another) and, within a
// row, in depth order. Each view's depth-sorted slots are cut into chunks of
// kSlotChunk; a chunk counts, per tile row of its view, the splats covering
// it; an exclusive scan of those counts in (row, chunk) order gives every
// chunk its base in every row; the chunk then sets its splats' bits in a
// 1024-bit map per row and writes each row's records there in bit order. This
// is the stable counting sort of the records by row, with no sort pass.
constexpr int kSlotChunk = 1024;
constexpr int kSlotPerLane = kSlotChunk / (kWarps * 32);  // slots per lane per chunk

// Lane slots of a chunk starting at `begin` of the depth-sorted slots, and
// their tile-row ranges and (with xr) tile-column ranges, empty for a culled
// slot. A culled slot is known by its sorted key (kCulledKey, read beside the
// slot), so the only gather by slot is its rectangle; a visible slot's
// rectangle is never empty (its footprint meets the image).
__device__ __forceinline__ void chunk_slot_rows(const uint32_t* __restrict__ sorted_slots,
                                                const uint32_t* __restrict__ sorted_keys,
                                                const SlotGeom* __restrict__ geom, int64_t begin,
                                                uint32_t (&slot)[kSlotPerLane],
                                                uint32_t (&yr)[kSlotPerLane],
                                                uint32_t (*xr)[kSlotPerLane] = nullptr) {
  const int w = warp_id(), lane = lane_id();
  bool live[kSlotPerLane];
#pragma unroll
  for (int k = 0; k < kSlotPerLane; ++k) {
    const int64_t i = begin + w * (kSlotChunk / kWarps) + k * 32 + lane;
    slot[k] = sorted_slots[i];
    live[k] = sorted_keys[i] != kCulledKey;
    yr[k] = 1u;  // y0 = 1 > y1 = 0: no rows
    if (xr != nullptr) (*xr)[k] = 1u;
  }
#pragma unroll
  for (int k = 0; k < kSlotPerLane; ++k)
    if (live[k]) {
      const uint2 r = geom[slot[k]].rect;
      yr[k] = r.y;
      if (xr != nullptr) (*xr)[k] = r.x;
    }
}

// counts[(row_offset + y) * cpv + c]: splats of chunk c of view v (block
// v * cpv + c) covering tile row y of the view.
__global__ void __launch_bounds__(kWarps * 32)
    k_slot_row_counts(const uint32_t* __restrict__ sorted_slots,
                      const uint32_t* __restrict__ sorted_keys,
                      const SlotGeom* __restrict__ geom,
                      const ViewDesc* __restrict__ views, int64_t slot_stride, int cpv,
                      int max_tiles_y, int32_t* __restrict__ counts) {
  extern __shared__ int32_t s_cnt[];  // [kWarps][max_tiles_y]
  const int v = blockIdx.x / cpv, c = blockIdx.x % cpv;
  const ViewDesc& vd = views[v];
  const int tiles_y = vd.tiles_y;
  for (int i = threadIdx.x; i < kWarps * tiles_y; i += blockDim.x)
    s_cnt[(i / tiles_y) * max_tiles_y + (i % tiles_y)] = 0;
  __syncthreads();
  uint32_t slot[kSlotPerLane], yr[kSlotPerLane];
  chunk_slot_rows(sorted_slots, sorted_keys, geom,
                  (int64_t)v * slot_stride + (int64_t)c * kSlotChunk, slot, yr);
  warp_range_counts(yr, tiles_y, s_cnt + warp_id() * max_tiles_y);
  __syncthreads();
  for (int y = threadIdx.x; y < tiles_y; y += blockDim.x) {
    int total = 0;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) total += s_cnt[k * max_tiles_y + y];
    counts[(int64_t)(vd.row_offset + y) * cpv + c] = total;
  }
}

// The chunk's records at offsets[(row_offset + y) * cpv + c] onwards in each
// row y, in slot order; nothing at or past `capacity`. As in k_chunk_expand the
// chunk is 1024 bits per row (kMapRows rows at a time); a warp per row lists the
// set bits' places, then takes a record per lane: its slot, and its columns cut
// to the ones its splat reaches in that row (row_columns on shapes kept in shared
// memory; without `tight` they stay the rectangle's). Bound by shared memory (the
// shapes' reads meet random banks; in two arrays of halves eight lanes spread over
// eight bank groups instead of four, the stage 1.98 -> 1.945 ms at 8 views of 1M) at
// 3 CTAs per SM. Before that, ranking in per-warp bitmaps took 0.57 against 0.60 ms
// at 8 views of 1M gaussians, 1920x1440, but the binning stage 446 against 423 us
// over 40 views of ten small scenes and 347 against 336 at 2 views of 700k, 1280x720.
constexpr int kMapRows = 512;
struct RowExpandSmem {
  float4 shape[2][kSlotChunk];         // the halves of the splats' RowShape
  uint32_t slot[kSlotChunk];
  uint16_t place[kWarps][kSlotChunk];  // a row's records: their splats' places
  uint32_t dst[kMapRows];              // each row's first record
};
static_assert(kSlotChunk == 32 * 32, "a word per lane");
static_assert(sizeof(RowShape) == 32, "two 16-byte halves");

__global__ void __launch_bounds__(kWarps * 32)
    k_slot_row_expand(const uint32_t* __restrict__ sorted_slots,
                      const uint32_t* __restrict__ sorted_keys,
                      const SlotGeom* __restrict__ geom, int tight,
                      const ViewDesc* __restrict__ views, int64_t slot_stride, int cpv,
                      const int64_t* __restrict__ offsets, int64_t capacity,
                      uint32_t* __restrict__ rec_slots, uint32_t* __restrict__ rec_xr) {
  extern __shared__ __align__(32) unsigned char row_smem[];
  RowExpandSmem& sm = *reinterpret_cast<RowExpandSmem*>(row_smem);
  uint32_t* const map = reinterpret_cast<uint32_t*>(row_smem + sizeof(RowExpandSmem));
  const int v = blockIdx.x / cpv, c = blockIdx.x % cpv;
  const ViewDesc& vd = views[v];
  const int tiles_y = vd.tiles_y;
  const int w = warp_id(), lane = lane_id();
  uint32_t slot[kSlotPerLane], yr[kSlotPerLane];
  uint32_t xr[kSlotPerLane];  // the box's column ranges
  chunk_slot_rows(sorted_slots, sorted_keys, geom,
                  (int64_t)v * slot_stride + (int64_t)c * kSlotChunk, slot, yr, &xr);
  const int place = w * (kSlotChunk / kWarps) + lane;  // of the lane's first splat
#pragma unroll
  for (int k = 0; k < kSlotPerLane; ++k) {
    sm.slot[place + k * 32] = slot[k];
    RowShape shape;
    shape.x = xr[k];
    shape.ia = 0.f;
    if (tight && (yr[k] >> 16) >= (yr[k] & 0xFFFF)) {
      const float4 co = geom[slot[k]].conic_op;
      const Footprint f = splat_footprint(co, vd.min_alpha);
      shape = row_shape(f, co, geom[slot[k]].xy, xr[k]);
    }
    float4 half[2];
    memcpy(half, &shape, sizeof(shape));
    sm.shape[0][place + k * 32] = half[0];
    sm.shape[1][place + k * 32] = half[1];
  }
  const uint32_t cap = (uint32_t)capacity;  // at most 2^31 - 1
  for (int r0 = 0; r0 < tiles_y; r0 += kMapRows) {
    const int rows = min(kMapRows, tiles_y - r0);
    const int pitch = rows | 1;
    for (int i = threadIdx.x; i < 32 * pitch; i += blockDim.x) map[i] = 0u;
    // record positions in 32 bits: nothing past the capacity is written
    for (int y = threadIdx.x; y < rows; y += blockDim.x)
      sm.dst[y] =
          (uint32_t)min(offsets[(int64_t)(vd.row_offset + r0 + y) * cpv + c], capacity);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSlotPerLane; ++k) {
      uint32_t* row = map + (w * kSlotPerLane + k) * pitch;
      const int lo = max((int)(yr[k] & 0xFFFF) - r0, 0);
      const int hi = min((int)(yr[k] >> 16) - r0, rows - 1);
      for (int y = lo; y <= hi; ++y) atomicOr(&row[y], 1u << lane);
    }
    __syncthreads();
    for (int y = w; y < rows; y += kWarps) {
      uint32_t m = map[lane * pitch + y];
      const int x = warp_inclusive_scan(__popc(m));
      const int total = __shfl_sync(kFull, x, 31);
      uint16_t* at = &sm.place[w][x - __popc(m)];
      while (m != 0u) {
        *at++ = (uint16_t)(32 * lane + __ffs(m) - 1);
        m &= m - 1u;
      }
      __syncwarp();
      const uint32_t dst = sm.dst[y];
      for (int i = lane; i < total; i += 32)
        if (dst + (uint32_t)i < cap) {
          const int p = sm.place[w][i];
          rec_slots[dst + i] = sm.slot[p];
          const float4 half[2] = {sm.shape[0][p], sm.shape[1][p]};
          RowShape shape;
          memcpy(&shape, half, sizeof(shape));
          rec_xr[dst + i] = row_columns(shape, r0 + y);
        }
      __syncwarp();  // the places are read before the next row's
    }
    if (r0 + kMapRows < tiles_y) __syncthreads();
  }
}

// ------------------------------------------------------- small images, directly
//
// With few tiles a view's tiles fit a CTA's shared memory and the lists need no
// rows in between. A CTA takes 256 depth-sorted slots, one per thread, and keeps a
// 256-bit map per tile of the ones that reach it: its counts per tile give, summed
// over the earlier chunks and scanned over the tiles, the chunk's base in every
// list, and a slot's place from there is the number of earlier bits. 4 launches
// instead of 9 to 13 (Frame::direct_lists has the times).
constexpr int kDirectSlots = kWarps * 32;

// The tiles that the thread's slot reaches, f(tile) in row order; `i` its place
// among the depth-sorted slots.
struct DirectSlot {
  uint32_t slot, yr;
  RowShape shape;
};
__device__ __forceinline__ DirectSlot direct_slot(const uint32_t* __restrict__ sorted_slots,
                                                  const uint32_t* __restrict__ sorted_keys,
                                                  const SlotGeom* __restrict__ geom, bool tight,
                                                  float min_alpha, int64_t i) {
  DirectSlot d;
  d.slot = sorted_slots[i];
  d.yr = d.shape.x = 1u;  // 1 > 0: no rows, no columns
  d.shape.ia = 0.f;
  if (sorted_keys[i] == kCulledKey) return d;
  const SlotGeom g = geom[d.slot];
  d.yr = g.rect.y;
  d.shape.x = g.rect.x;
  if (tight && (d.yr >> 16) >= (d.yr & 0xFFFF))
    d.shape = row_shape(splat_footprint(g.conic_op, min_alpha), g.conic_op, g.xy, g.rect.x);
  return d;
}
template <typename F>
__device__ __forceinline__ void for_each_reached_tile(const DirectSlot& d, int tiles_x, F&& f) {
  const int y1 = d.yr >> 16;
  for (int y = d.yr & 0xFFFF; y <= y1; ++y) {
    const uint32_t x = row_columns(d.shape, y);
    const int x1 = x >> 16;
    for (int c = x & 0xFFFF; c <= x1; ++c) f(y * tiles_x + c);
  }
}

// Each warp's bits of the chunk's map, map[kWarps][tiles].
__device__ __forceinline__ void map_tiles(const DirectSlot& d, int tiles, int tiles_x,
                                          uint32_t* map) {
  for (int i = threadIdx.x; i < kWarps * tiles; i += blockDim.x) map[i] = 0u;
  __syncthreads();
  uint32_t* mine = map + warp_id() * tiles;
  const uint32_t bit = 1u << lane_id();
  for_each_reached_tile(d, tiles_x, [&](int t) { atomicOr(&mine[t], bit); });
  __syncthreads();
}

// counts[chunk * total_tiles + tile]: slots of the chunk that reach the tile; a
// chunk counts its own view's tiles.
__global__ void __launch_bounds__(kDirectSlots)
    k_direct_counts(const uint32_t* __restrict__ sorted_slots,
                    const uint32_t* __restrict__ sorted_keys,
                    const SlotGeom* __restrict__ geom, int tight,
                    const ViewDesc* __restrict__ views, int64_t slot_stride, int cpv,
                    int total_tiles, int32_t* __restrict__ counts) {
  extern __shared__ uint32_t s_map[];
  const int v = blockIdx.x / cpv, c = blockIdx.x % cpv;
  const ViewDesc& vd = views[v];
  const int tiles = vd.tiles_x * vd.tiles_y;
  const DirectSlot d = direct_slot(sorted_slots, sorted_keys, geom, tight, vd.min_alpha,
                                   (int64_t)v * slot_stride + c * kDirectSlots + threadIdx.x);
  map_tiles(d, tiles, vd.tiles_x, s_map);
  for (int t = threadIdx.x; t < tiles; t += blockDim.x) {
    int total = 0;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) total += __popc(s_map[k * tiles + t]);
    counts[(int64_t)c * total_tiles + vd.tile_offset + t] = total;
  }
}

// The counts become each chunk's base within its tile's list, and the lists'
// lengths go to tile_counts. 32 tiles per CTA, each warp a range of the chunks.
__global__ void __launch_bounds__(kWarps * 32)
    k_direct_bases(int32_t* __restrict__ counts, int cpv, int total_tiles,
                   int32_t* __restrict__ tile_counts, int32_t* __restrict__ overflow) {
  __shared__ int s_sum[kWarps][32];
  const int w = warp_id(), lane = lane_id();
  const int tile = blockIdx.x * 32 + lane;
  const int per = (cpv + kWarps - 1) / kWarps;
  const int c0 = min(cpv, w * per), c1 = min(cpv, c0 + per);
  if (blockIdx.x == 0 && threadIdx.x == 0) *overflow = 0;
  int sum = 0;
  if (tile < total_tiles)
#pragma unroll 8
    for (int c = c0; c < c1; ++c) sum += counts[(int64_t)c * total_tiles + tile];
  s_sum[w][lane] = sum;
  __syncthreads();
  if (tile >= total_tiles) return;
  int run = 0;
  for (int k = 0; k < w; ++k) run += s_sum[k][lane];
  if (w == kWarps - 1) tile_counts[tile] = run + sum;
#pragma unroll 4
  for (int c = c0; c < c1; ++c) {
    int32_t* at = &counts[(int64_t)c * total_tiles + tile];
    const int n = *at;
    *at = run;
    run += n;
  }
}

// The lists; nothing at or past `capacity`. A view's first chunk also writes its
// tiles' ranges (a tile whose list would pass the capacity is left empty and
// raises the overflow flag).
__global__ void __launch_bounds__(kDirectSlots)
    k_direct_expand(const uint32_t* __restrict__ sorted_slots,
                    const uint32_t* __restrict__ sorted_keys,
                    const SlotGeom* __restrict__ geom, int tight,
                    const ViewDesc* __restrict__ views, int64_t slot_stride, int cpv,
                    int total_tiles, const int32_t* __restrict__ bases,
                    const int64_t* __restrict__ tile_offsets,
                    const int32_t* __restrict__ tile_counts, int64_t capacity,
                    uint32_t* __restrict__ tile_slots, int2* __restrict__ ranges,
                    int32_t* __restrict__ overflow) {
  // per tile: the map, a byte per warp counting the earlier warps' bits, the base
  extern __shared__ __align__(8) uint32_t s_map[];
  const int v = blockIdx.x / cpv, c = blockIdx.x % cpv;
  const ViewDesc& vd = views[v];
  const int tiles = vd.tiles_x * vd.tiles_y;
  uint8_t* const before = reinterpret_cast<uint8_t*>(s_map + kWarps * tiles);
  uint32_t* const base = s_map + (kWarps + 2) * tiles;
  const DirectSlot d = direct_slot(sorted_slots, sorted_keys, geom, tight, vd.min_alpha,
                                   (int64_t)v * slot_stride + c * kDirectSlots + threadIdx.x);
  map_tiles(d, tiles, vd.tiles_x, s_map);
  for (int t = threadIdx.x; t < tiles; t += blockDim.x) {
    const int64_t tile = vd.tile_offset + t;
    const int64_t first = tile_offsets[tile];
    // list positions in 32 bits: nothing past the capacity is written
    base[t] = (uint32_t)min(first + bases[(int64_t)c * total_tiles + tile], capacity);
    uint64_t packed = 0;
    int run = 0;  // at most 7 * 32 before the last warp
#pragma unroll
    for (int k = 0; k < kWarps; ++k) {
      packed |= (uint64_t)run << (8 * k);
      run += __popc(s_map[k * tiles + t]);
    }
    reinterpret_cast<uint64_t*>(before)[t] = packed;
    if (c == 0) {
      const int64_t end = first + tile_counts[tile];
      ranges[tile] = end <= capacity ? make_int2((int)first, (int)end) : make_int2(0, 0);
      if (end > capacity) atomicExch(overflow, 1);
    }
  }
  __syncthreads();
  const int w = warp_id();
  const uint32_t* mine = s_map + w * tiles;
  const unsigned lt = lanemask_lt();
  for_each_reached_tile(d, vd.tiles_x, [&](int t) {
    const uint64_t at = (uint64_t)base[t] + before[8 * t + w] + __popc(mine[t] & lt);
    if (at < (uint64_t)capacity) tile_slots[at] = d.slot;
  });
}

// ------------------------------------------------------------------ host

size_t chunk_counts_smem(int max_tiles_x) { return sizeof(int32_t) * kWarps * max_tiles_x; }
size_t chunk_expand_smem(int max_tiles_x) {
  return sizeof(uint32_t) * kMapWords * (size_t)(std::min(max_tiles_x, kMapCols) | 1);
}

size_t slot_row_expand_smem(int max_tiles_y) {
  return sizeof(RowExpandSmem) +
         sizeof(uint32_t) * 32 * (size_t)(std::min(max_tiles_y, kMapRows) | 1);
}

size_t direct_counts_smem(int tiles) { return sizeof(uint32_t) * kWarps * (size_t)tiles; }
size_t direct_expand_smem(int tiles) { return sizeof(uint32_t) * (kWarps + 3) * (size_t)tiles; }

size_t slot_row_counts_smem(int max_tiles_y) { return sizeof(int32_t) * kWarps * max_tiles_y; }

void configure_bin_kernels() {
  cudaFuncSetAttribute(k_direct_counts, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)direct_counts_smem(kMaxDirectTiles));
  cudaFuncSetAttribute(k_direct_expand, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)direct_expand_smem(kMaxDirectTiles));
  cudaFuncSetAttribute(k_chunk_counts, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)chunk_counts_smem(kMaxTilesX));
  cudaFuncSetAttribute(k_chunk_expand, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)chunk_expand_smem(kMaxTilesX));
  cudaFuncSetAttribute(k_slot_row_counts, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)slot_row_counts_smem(kMaxTilesY));
  cudaFuncSetAttribute(k_slot_row_expand, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)slot_row_expand_smem(kMaxTilesY));
}

int slot_chunks_per_view(int64_t slot_stride) { return (int)(slot_stride / kSlotChunk); }

void launch_slot_row_counts(const uint32_t* sorted_slots, const uint32_t* sorted_keys,
                            const SlotGeom* geom, const ViewDesc* views, int n_views,
                            int64_t slot_stride, int max_tiles_y, int32_t* counts,
                            cudaStream_t stream) {
  const int cpv = slot_chunks_per_view(slot_stride);
  if (n_views <= 0 || cpv <= 0) return;
  count_launch();
  k_slot_row_counts<<<(unsigned)(n_views * cpv), kWarps * 32, slot_row_counts_smem(max_tiles_y),
                      stream>>>(sorted_slots, sorted_keys, geom, views, slot_stride, cpv,
                                max_tiles_y, counts);
}

void launch_slot_row_expand(const uint32_t* sorted_slots, const uint32_t* sorted_keys,
                            const SlotGeom* geom, bool tight,
                            const ViewDesc* views, int n_views,
                            int64_t slot_stride, int max_tiles_y, const int64_t* offsets,
                            int64_t capacity, uint32_t* rec_slots, uint32_t* rec_xr,
                            cudaStream_t stream) {
  const int cpv = slot_chunks_per_view(slot_stride);
  if (n_views <= 0 || cpv <= 0) return;
  count_launch();
  k_slot_row_expand<<<(unsigned)(n_views * cpv), kWarps * 32, slot_row_expand_smem(max_tiles_y),
                      stream>>>(sorted_slots, sorted_keys, geom, tight, views,
                                slot_stride, cpv, offsets, capacity, rec_slots, rec_xr);
}

int direct_chunks_per_view(int64_t slot_stride) { return (int)(slot_stride / kDirectSlots); }

void launch_direct_counts(const uint32_t* sorted_slots, const uint32_t* sorted_keys,
                          const SlotGeom* geom, bool tight, const ViewDesc* views, int n_views,
                          int64_t slot_stride, int max_tiles, int total_tiles, int32_t* counts,
                          int32_t* tile_counts, int32_t* overflow, cudaStream_t stream) {
  const int cpv = direct_chunks_per_view(slot_stride);
  count_launch();
  k_direct_counts<<<(unsigned)(n_views * cpv), kDirectSlots, direct_counts_smem(max_tiles),
                    stream>>>(sorted_slots, sorted_keys, geom, tight, views, slot_stride, cpv,
                              total_tiles, counts);
  count_launch();
  k_direct_bases<<<(unsigned)std::max(1, (total_tiles + 31) / 32), kWarps * 32, 0, stream>>>(
      counts, cpv, total_tiles, tile_counts, overflow);
}

void launch_direct_expand(const uint32_t* sorted_slots, const uint32_t* sorted_keys,
                          const SlotGeom* geom, bool tight, const ViewDesc* views, int n_views,
                          int64_t slot_stride, int max_tiles, int total_tiles,
                          const int32_t* bases, const int64_t* tile_offsets,
                          const int32_t* tile_counts, int64_t capacity, uint32_t* tile_slots,
                          int2* ranges, int32_t* overflow, cudaStream_t stream) {
  const int cpv = direct_chunks_per_view(slot_stride);
  count_launch();
  k_direct_expand<<<(unsigned)(n_views * cpv), kDirectSlots, direct_expand_smem(max_tiles),
                    stream>>>(sorted_slots, sorted_keys, geom, tight, views, slot_stride, cpv,
                              total_tiles, bases, tile_offsets, tile_counts, capacity,
                              tile_slots, ranges, overflow);
}

int64_t max_row_chunks(int64_t records, int total_rows) { return records / kChunk + total_rows + 1; }

void launch_tile_lists(const int64_t* offsets, int cpv, const int64_t* total_records,
                       int64_t record_capacity, const uint32_t* rec_slots,
                       const uint32_t* rec_xr, const ViewDesc* views, int n_views,
                       int total_rows, int max_tiles_x, int64_t max_chunks, int4* chunks,
                       int32_t* n_chunks, int32_t* chunk_counts, int32_t* chunk_base,
                       int32_t* tile_counts, int32_t* overflow, cudaStream_t stream) {
  if (total_rows <= 0) return;
  count_launch();
  k_row_chunks<<<1, 1024, 0, stream>>>(offsets, cpv, total_records, record_capacity, total_rows,
                                       (int)max_chunks, chunks, n_chunks, overflow);
  count_launch();
  k_chunk_counts<<<(unsigned)max_chunks, kWarps * 32, chunk_counts_smem(max_tiles_x), stream>>>(
      chunks, n_chunks, rec_slots, rec_xr, views, n_views, max_tiles_x, chunk_counts);
  count_launch();
  k_row_tiles<<<total_rows, 256, 0, stream>>>(chunks, n_chunks, views, n_views, max_tiles_x,
                                              chunk_counts, chunk_base, tile_counts);
}

void launch_ranges_from_offsets(const int32_t* counts, const int64_t* offsets, int64_t n_tiles,
                                int64_t capacity, int2* ranges, int32_t* overflow,
                                cudaStream_t stream) {
  if (n_tiles <= 0) return;
  count_launch();
  k_ranges_from_offsets<<<(unsigned)((n_tiles + 255) / 256), 256, 0, stream>>>(
      counts, offsets, n_tiles, capacity, ranges, overflow);
}

void launch_chunk_expand(const int4* chunks, const int32_t* n_chunks, const uint32_t* rec_slots,
                         const uint32_t* rec_xr, const ViewDesc* views, int n_views, int max_tiles_x,
                         int64_t max_chunks, const int32_t* chunk_base,
                         const int64_t* tile_offsets, int64_t capacity, uint32_t* tile_slots,
                         cudaStream_t stream) {
  if (max_chunks <= 0) return;
  count_launch();
  k_chunk_expand<<<(unsigned)max_chunks, kWarps * 32, chunk_expand_smem(max_tiles_x), stream>>>(
      chunks, n_chunks, rec_slots, rec_xr, views, n_views, max_tiles_x, chunk_base, tile_offsets,
      capacity, tile_slots);
}

}  // namespace pxs
