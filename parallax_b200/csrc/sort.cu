// sort.cu -- scans and the depth sort for the binning path.
//
// Device-wide exclusive scans, and a stable segmented LSD radix sort of the depth
// keys of every (view, gaussian) slot with the slots as values (segmented per
// view; ties keep gaussian order), four passes of 8 bits. The first pass reads
// the keys where projection left them and counts the slots itself.
#include "common.cuh"
#include "kernels.h"

namespace pxs {
namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int kSortWarps = kSortThreads / 32;

template <typename T>
__device__ T block_exclusive_scan(T v, T* total, T* smem_warp) {
  // warp inclusive scan
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T n = __shfl_up_sync(0xffffffffu, x, o);
    if (lane_id() >= o) x += n;
  }
  if (lane_id() == 31) smem_warp[warp_id()] = x;
  __syncthreads();
  if (warp_id() == 0) {
    T w = lane_id() < (int)(blockDim.x / 32) ? smem_warp[lane_id()] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T n = __shfl_up_sync(0xffffffffu, w, o);
      if (lane_id() >= o) w += n;
    }
    smem_warp[lane_id()] = w;  // inclusive warp totals
  }
  __syncthreads();
  const T warp_prefix = warp_id() > 0 ? smem_warp[warp_id() - 1] : T(0);
  *total = smem_warp[blockDim.x / 32 - 1];
  __syncthreads();
  return warp_prefix + x - v;
}

template <typename Tin, typename T>
__global__ void __launch_bounds__(kScanThreads)
    k_scan_reduce(const Tin* __restrict__ in, int64_t n, T* __restrict__ block_sums) {
  __shared__ T warp_sums[32];
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  T sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int64_t i = base + (int64_t)k * kScanThreads + threadIdx.x;
    if (i < n) sum += (T)in[i];
  }
  T total;
  block_exclusive_scan<T>(sum, &total, warp_sums);
  if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

// Exclusive scan of one tile per block, seeded with block_offsets[block] (or 0).
template <typename Tin, typename T>
__global__ void __launch_bounds__(kScanThreads)
    k_scan_tile(const Tin* __restrict__ in, int64_t n, T* __restrict__ out,
                const T* __restrict__ block_offsets, T* __restrict__ total_out) {
  __shared__ T warp_sums[32];
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  // blocked arrangement: thread owns kScanItems consecutive items
  T vals[kScanItems];
  T sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int64_t i = base + (int64_t)threadIdx.x * kScanItems + k;
    vals[k] = i < n ? (T)in[i] : T(0);
    sum += vals[k];
  }
  T total;
  T prefix = block_exclusive_scan<T>(sum, &total, warp_sums);
  if (block_offsets != nullptr) prefix += block_offsets[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int64_t i = base + (int64_t)threadIdx.x * kScanItems + k;
    if (i < n) out[i] = prefix;
    prefix += vals[k];
  }
  if (total_out != nullptr && blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1)
    *total_out = prefix;
}

// Exclusive scan of up to kScanOneMax items by one CTA: one launch instead of
// three, in about the time of one of them.
constexpr int kScanOneThreads = 1024, kScanOneItems = 4;
constexpr int64_t kScanOneMax = 16384;

template <typename Tin, typename T>
__global__ void __launch_bounds__(kScanOneThreads)
    k_scan_one(const Tin* __restrict__ in, int n, T* __restrict__ out,
               T* __restrict__ total_out) {
  __shared__ T warp_sums[32];
  T carry = 0;
  for (int base = 0; base < n; base += kScanOneThreads * kScanOneItems) {
    const int first = base + (int)threadIdx.x * kScanOneItems;
    T vals[kScanOneItems], sum = 0, total;
#pragma unroll
    for (int k = 0; k < kScanOneItems; ++k) {
      vals[k] = first + k < n ? (T)in[first + k] : T(0);
      sum += vals[k];
    }
    T prefix = carry + block_exclusive_scan<T>(sum, &total, warp_sums);
#pragma unroll
    for (int k = 0; k < kScanOneItems; ++k) {
      if (first + k < n) out[first + k] = prefix;
      prefix += vals[k];
    }
    carry += total;
  }
  if (total_out != nullptr && threadIdx.x == 0) *total_out = carry;
}

// ------------------------------------------------------------ radix sort

constexpr int kDigits = 256, kDigitBits = 8, kPasses = 4;

// Digit counts of one tile of kItems x kSortThreads keys.
template <int kItems>
__device__ __forceinline__ void tile_histogram(const uint32_t* __restrict__ keys, int shift,
                                               uint32_t* h) {
  for (int d = threadIdx.x; d < kDigits; d += kSortThreads) h[d] = 0;
  __syncthreads();
  const int64_t begin = (int64_t)blockIdx.x * (kItems * kSortThreads);
  uint32_t key[kItems];
#pragma unroll
  for (int k = 0; k < kItems; ++k) key[k] = keys[begin + k * kSortThreads + threadIdx.x];
#pragma unroll
  for (int k = 0; k < kItems; ++k) atomicAdd(&h[(key[k] >> shift) & (kDigits - 1)], 1u);
  __syncthreads();
}

// The counts as hist[(segment * digits + digit) * blocks per segment + block], the
// order in which their exclusive scan gives each block its offsets.
__global__ void __launch_bounds__(kSortThreads)
    k_radix_upsweep(const uint32_t* __restrict__ keys, int shift, int blocks_per_segment,
                    uint32_t* __restrict__ hist) {
  __shared__ uint32_t h[kDigits];
  tile_histogram<kSortItemsPerThread>(keys, shift, h);
  const int seg = blockIdx.x / blocks_per_segment, bis = blockIdx.x % blocks_per_segment;
  for (int d = threadIdx.x; d < kDigits; d += kSortThreads)
    hist[((int64_t)seg * kDigits + d) * blocks_per_segment + bis] = h[d];
}

// For the passes that count as they go (below): the first pass's counts as
// hist[block * digits + digit], and cleared counts for the other passes.
template <int kItems>
__global__ void __launch_bounds__(kSortThreads)
    k_radix_counts(const uint32_t* __restrict__ keys, uint32_t* __restrict__ hist) {
  __shared__ uint32_t h[kDigits];
  tile_histogram<kItems>(keys, 0, h);
  const int64_t pass_size = (int64_t)gridDim.x * kDigits;
  for (int d = threadIdx.x; d < kDigits; d += kSortThreads) {
    uint32_t* at = hist + (int64_t)blockIdx.x * kDigits + d;
    at[0] = h[d];
#pragma unroll
    for (int p = 1; p < kPasses; ++p) at[p * pass_size] = 0;
  }
}

// The lanes whose digit is this lane's, by a ballot per digit bit: __match_any_sync
// takes a round per different digit, 47 against 18 us for a pass of 4M keys between
// random digits and few. Binning 2.05 -> 1.98 ms at 8 views of 1M gaussians, 111 ->
// 109 us at 152k. (The peers of all items first spare their chain, but 101
// registers: 2.01 ms.)
__device__ __forceinline__ unsigned digit_peers(uint32_t digit) {
  unsigned peers = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < kDigitBits; ++b) {
    const bool bit = (digit >> b) & 1u;
    const unsigned set = __ballot_sync(0xffffffffu, bit);
    peers &= bit ? set : ~set;
  }
  return peers;
}

// Stable scatter of one block tile by one digit. Items are warp-striped (warp w
// owns kItems * 32 consecutive ones, item k of a lane at k*32 + lane) and ranked
// among their digit's peers, then offset by earlier warps. The tile is
// reordered by digit in shared memory and written out digit run by digit run,
// so consecutive threads write consecutive addresses. vals_in null: the values
// are the items' places.
//
// Where the block's digit runs begin: `offsets` is the scan of k_radix_upsweep's
// counts, or (kCounting) the counts themselves by block, which each block sums for
// itself, and each item written also counts towards its tile of the next pass
// (`next`, null in the last). That spares two launches a pass and is for few
// enough blocks (depth_sort).
template <int kItems, bool kCounting>
__global__ void __launch_bounds__(kSortThreads)
    k_radix_downsweep(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                      uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out,
                      int shift, int blocks_per_segment, const uint32_t* __restrict__ offsets,
                      uint32_t* __restrict__ next) {
  constexpr int kTileItems = kItems * kSortThreads;
  constexpr int kStageWords = kTileItems > kSortWarps * kDigits ? kTileItems : kSortWarps * kDigits;
  // per-warp digit counters; reused as the staging buffer once ranks are known
  __shared__ uint32_t counts[kStageWords];
  __shared__ uint32_t block_offset[kDigits];
  __shared__ uint32_t digit_start[kDigits];
  __shared__ uint32_t warp_sums[32];
  // of each digit, by fourth block: in the segment's blocks, in the earlier ones
  __shared__ __align__(16) uint32_t s_whole[kCounting ? 4 : 1][kCounting ? kDigits : 4];
  __shared__ __align__(16) uint32_t s_before[kCounting ? 4 : 1][kCounting ? kDigits : 4];
  static_assert(kSortThreads == kDigits, "a digit per thread");
  const int t = threadIdx.x;
  const int seg = blockIdx.x / blocks_per_segment, bis = blockIdx.x % blocks_per_segment;
  const int64_t begin = (int64_t)blockIdx.x * kTileItems;
  const int warp = warp_id(), lane = lane_id();
  const unsigned lt = lanemask_lt();
  uint32_t key[kItems], val[kItems], rank[kItems];
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const int64_t i = begin + warp * (kItems * 32) + k * 32 + lane;
    key[k] = keys_in[i];
    val[k] = vals_in != nullptr ? vals_in[i] : (uint32_t)i;
  }
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) counts[w * kDigits + t] = 0;
  if (kCounting) {
    // a quarter of the threads per fourth block, four digits per thread: the
    // segment's counts in a few rounds of 16-byte loads (one digit per thread
    // took a round per eight blocks, most of the kernel at 74 blocks)
    const uint4* rows = reinterpret_cast<const uint4*>(
        offsets + (int64_t)seg * blocks_per_segment * kDigits);
    const int phase = t >> 6, quad = t & 63;
    uint4 whole = make_uint4(0, 0, 0, 0), before = whole;
#pragma unroll 8
    for (int b = phase; b < blocks_per_segment; b += 4) {
      const uint4 n = rows[b * (kDigits / 4) + quad];
      whole.x += n.x;
      whole.y += n.y;
      whole.z += n.z;
      whole.w += n.w;
      if (b < bis) {
        before.x += n.x;
        before.y += n.y;
        before.z += n.z;
        before.w += n.w;
      }
    }
    reinterpret_cast<uint4*>(s_whole[phase])[quad] = whole;
    reinterpret_cast<uint4*>(s_before[phase])[quad] = before;
  } else {
    block_offset[t] = offsets[((int64_t)seg * kDigits + t) * blocks_per_segment + bis];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const uint32_t d = (key[k] >> shift) & (kDigits - 1);
    const unsigned peers = digit_peers(d);
    const uint32_t base = counts[warp * kDigits + d];
    __syncwarp();
    if (lane == __ffs(peers) - 1) counts[warp * kDigits + d] = base + __popc(peers);
    __syncwarp();
    rank[k] = base + __popc(peers & lt);
  }
  __syncthreads();
  // digit t: exclusive prefix over warps in place, then the block-local start of
  // each digit by a scan in digit order
  uint32_t run = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) {
    const uint32_t c = counts[w * kDigits + t];
    counts[w * kDigits + t] = run;
    run += c;
  }
  uint32_t block_total;
  digit_start[t] = block_exclusive_scan<uint32_t>(run, &block_total, warp_sums);
  if constexpr (kCounting) {
    const uint32_t whole = s_whole[0][t] + s_whole[1][t] + s_whole[2][t] + s_whole[3][t];
    const uint32_t before = s_before[0][t] + s_before[1][t] + s_before[2][t] + s_before[3][t];
    block_offset[t] = (uint32_t)seg * blocks_per_segment * kTileItems + before +
                      block_exclusive_scan<uint32_t>(whole, &block_total, warp_sums);
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const uint32_t d = (key[k] >> shift) & (kDigits - 1);
    rank[k] += digit_start[d] + counts[warp * kDigits + d];  // the place in the tile
  }
  __syncthreads();  // counts is now free: stage the keys by digit
#pragma unroll
  for (int k = 0; k < kItems; ++k) counts[rank[k]] = key[k];
  __syncthreads();
  uint32_t to[kItems];
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const int i = k * kSortThreads + t;
    const uint32_t kk = counts[i];
    const uint32_t d = (kk >> shift) & (kDigits - 1);
    to[k] = block_offset[d] + ((uint32_t)i - digit_start[d]);
    keys_out[to[k]] = kk;
    if (kCounting && next != nullptr)
      atomicAdd(&next[(int64_t)(to[k] / kTileItems) * kDigits +
                      ((kk >> (shift + kDigitBits)) & (kDigits - 1))],
                1u);
  }
  __syncthreads();  // stage the values the same way
#pragma unroll
  for (int k = 0; k < kItems; ++k) counts[rank[k]] = val[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kItems; ++k) vals_out[to[k]] = counts[k * kSortThreads + t];
}

}  // namespace

// --------------------------------------------------------------- host side

template <typename Tin, typename T>
static void scan_impl(const Tin* in, T* out, int64_t n, T* total, ScanScratch& scratch, int level,
                      cudaStream_t stream) {
  const int64_t blocks = (n + kScanTile - 1) / kScanTile;
  if (blocks <= 1) {
    count_launch();
    k_scan_tile<Tin, T><<<1, kScanThreads, 0, stream>>>(in, n, out, nullptr, total);
    return;
  }
  if (n <= kScanOneMax) {
    count_launch();
    k_scan_one<Tin, T><<<1, kScanOneThreads, 0, stream>>>(in, (int)n, out, total);
    return;
  }
  T* sums = reinterpret_cast<T*>(scratch.level[level]);
  T* sums_scanned = reinterpret_cast<T*>(scratch.level[level]) + blocks;
  count_launch();
  k_scan_reduce<Tin, T><<<(unsigned)blocks, kScanThreads, 0, stream>>>(in, n, sums);
  scan_impl<T, T>(sums, sums_scanned, blocks, total, scratch, level + 1, stream);
  count_launch();
  k_scan_tile<Tin, T><<<(unsigned)blocks, kScanThreads, 0, stream>>>(in, n, out, sums_scanned,
                                                                      nullptr);
}

size_t scan_scratch_bytes(int64_t n, int level) {
  const int64_t blocks = (n + kScanTile - 1) / kScanTile;
  if (blocks <= 1) return 0;
  return (size_t)blocks * 2 * sizeof(int64_t) + scan_scratch_bytes(blocks, level + 1);
}

void scan_scratch_assign(ScanScratch& s, char* base, int64_t n) {
  int level = 0;
  int64_t m = n;
  while (level < ScanScratch::kLevels) {
    const int64_t blocks = (m + kScanTile - 1) / kScanTile;
    if (blocks <= 1) break;
    s.level[level] = base;
    base += blocks * 2 * sizeof(int64_t);
    m = blocks;
    ++level;
  }
}

void exclusive_scan_i32_to_i64(const int32_t* in, int64_t* out, int64_t n, int64_t* total,
                               ScanScratch& scratch, cudaStream_t stream) {
  if (n <= 0) {
    cudaMemsetAsync(total, 0, sizeof(int64_t), stream);
    return;
  }
  scan_impl<int32_t, int64_t>(in, out, n, total, scratch, 0, stream);
}

void exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t n, ScanScratch& scratch,
                        cudaStream_t stream) {
  if (n <= 0) return;
  scan_impl<uint32_t, uint32_t>(in, out, n, nullptr, scratch, 0, stream);
}

namespace {

// Items per thread of the counting passes, 0 where they do not pay: their blocks
// each sum every block's counts of their view and count each item with a global
// atomic, but a sort is 5 launches instead of 12 to 20, and small tiles spread a
// small cloud over the SMs. The binning stage in us, with and without: 33 / 52 (4k
// slots), 45 / 62 (20k), 64 / 91 (3 x 40k), 70 / 87 (60k), 109 / 129 (152k), 141 /
// 154 (300k), 191 / 194 (600k); past the lines 244 / 237 (900k), and 597 / 475 for
// 6M slots of 40 small views.
int counting_items(int64_t segment_len, int64_t n) {
  if (n > (int64_t)1 << 20 || segment_len > (int64_t)5 << 17) return 0;
  return segment_len <= (int64_t)1 << 16 ? 4 : segment_len <= (int64_t)1 << 18 ? 8 : 16;
}

template <int kItems>
void counting_sort(const uint32_t* keys, int64_t n, int64_t segment_len, uint32_t* keys_a,
                   uint32_t* vals_a, uint32_t* keys_b, uint32_t* vals_b, uint32_t* hist,
                   cudaStream_t stream) {
  const int tile = kItems * kSortThreads;
  const int blocks = (int)(n / tile), per_segment = (int)(segment_len / tile);
  const int64_t pass_size = (int64_t)blocks * kDigits;
  count_launch();
  k_radix_counts<kItems><<<blocks, kSortThreads, 0, stream>>>(keys, hist);
  const uint32_t *ki = keys, *vi = nullptr;
  for (int p = 0; p < kPasses; ++p) {
    uint32_t *ko = p % 2 ? keys_b : keys_a, *vo = p % 2 ? vals_b : vals_a;
    count_launch();
    k_radix_downsweep<kItems, true><<<blocks, kSortThreads, 0, stream>>>(
        ki, vi, ko, vo, p * kDigitBits, per_segment, hist + p * pass_size,
        p + 1 < kPasses ? hist + (p + 1) * pass_size : nullptr);
    ki = ko;
    vi = vo;
  }
}

}  // namespace

size_t depth_sort_hist_entries(int64_t n, int64_t segment_len) {
  const int items = counting_items(segment_len, n);
  return items > 0 ? (size_t)(n / (items * kSortThreads)) * kDigits * kPasses
                   : (size_t)(n / kSortTile) * kDigits;
}

// The counting passes scan no counts.
size_t depth_sort_scanned_entries(int64_t n, int64_t segment_len) {
  return counting_items(segment_len, n) > 0 ? 0 : depth_sort_hist_entries(n, segment_len);
}

void depth_sort(const uint32_t* keys, int64_t n, int64_t segment_len, uint32_t* keys_a,
                uint32_t* vals_a, uint32_t* keys_b, uint32_t* vals_b, uint32_t* hist,
                uint32_t* hist_scanned, ScanScratch& scratch, cudaStream_t stream) {
  static_assert(kPasses % 2 == 0, "the result lies in the b buffers");
  if (n <= 0) return;
  const int items = counting_items(segment_len, n);
  if (items == 4) {
    counting_sort<4>(keys, n, segment_len, keys_a, vals_a, keys_b, vals_b, hist, stream);
  } else if (items == 8) {
    counting_sort<8>(keys, n, segment_len, keys_a, vals_a, keys_b, vals_b, hist, stream);
  } else if (items == 16) {
    counting_sort<16>(keys, n, segment_len, keys_a, vals_a, keys_b, vals_b, hist, stream);
  } else {
    const int blocks = (int)(n / kSortTile), per_segment = (int)(segment_len / kSortTile);
    const uint32_t *ki = keys, *vi = nullptr;
    for (int p = 0; p < kPasses; ++p) {
      uint32_t *ko = p % 2 ? keys_b : keys_a, *vo = p % 2 ? vals_b : vals_a;
      count_launch();
      k_radix_upsweep<<<blocks, kSortThreads, 0, stream>>>(ki, p * kDigitBits, per_segment, hist);
      exclusive_scan_u32(hist, hist_scanned, (int64_t)blocks * kDigits, scratch, stream);
      count_launch();
      k_radix_downsweep<kSortItemsPerThread, false><<<blocks, kSortThreads, 0, stream>>>(
          ki, vi, ko, vo, p * kDigitBits, per_segment, hist_scanned, nullptr);
      ki = ko;
      vi = vo;
    }
  }
}

}  // namespace pxs
