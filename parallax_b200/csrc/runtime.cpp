// runtime.cpp -- the per-batch rasterisation frame: buffers and stage launches.
#include "runtime.h"

#include <algorithm>
#include <cmath>

namespace pxs {

int g_fail_allocation_after = 0;
int64_t g_device_allocations = 0;
int64_t g_kernel_launches = 0;

void check_cuda(cudaError_t err, const char* what) {
  if (err != cudaSuccess) {
    cudaGetLastError();
    throw Error(PXS_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(err));
  }
}

// ssimKernel (SplatRaster.cpp:587-600), with the same libm expf as the reference.
void ssim_kernel_weights(float out[11]) {
  float total = 0.f;
  for (int i = -5; i <= 5; ++i) {
    const float v = std::exp(-0.5f * static_cast<float>(i * i) / (1.5f * 1.5f));
    out[i + 5] = v;
    total += v;
  }
  for (int i = 0; i < 11; ++i) out[i] /= total;
}

void downscaled_size(int width, int height, int target_width, int* out_width, int* out_height) {
  if (width <= 0 || height <= 0 || target_width <= 0 || width <= target_width) {
    *out_width = width;
    *out_height = height;
    return;
  }
  *out_width = target_width;
  *out_height = std::max(1, static_cast<int>(std::lround(static_cast<double>(height) *
                                                          target_width / width)));
}

ViewBatch make_batch(const pxs_camera* cameras, int n_views, const pxs_raster_options& options,
                     int cloud_sh_degree) {
  ViewBatch b;
  b.views.resize(static_cast<size_t>(n_views));
  int tile_offset = 0, row_offset = 0;
  int64_t pixel_offset = 0;
  for (int v = 0; v < n_views; ++v) {
    ViewDesc& d = b.views[static_cast<size_t>(v)];
    std::memset(&d, 0, sizeof(d));
    d.cam = cameras[v];
    if (d.cam.width < 0 || d.cam.height < 0) throw Error(PXS_ERR_INVALID, "negative image size");
    for (int c = 0; c < 3; ++c) d.background[c] = options.background[c];
    d.sh_degree = std::min(options.sh_degree, cloud_sh_degree);
    d.tiles_x = (d.cam.width + kTile - 1) / kTile;
    d.tiles_y = (d.cam.height + kTile - 1) / kTile;
    if (d.tiles_x > kMaxTilesX || d.tiles_y > kMaxTilesY)
      throw Error(PXS_ERR_INVALID, "image too large (at most 2048 tiles across and down)");
    d.tile_offset = tile_offset;
    d.row_offset = row_offset;
    d.pixel_offset = pixel_offset;
    d.target_offset = pixel_offset;
    d.min_alpha = options.min_alpha;
    d.transmittance_cutoff = options.transmittance_cutoff;
    d.screen_dilation = options.screen_dilation;
    tile_offset += d.tiles_x * d.tiles_y;
    row_offset += d.tiles_y;
    b.max_tiles_x = std::max(b.max_tiles_x, d.tiles_x);
    b.max_tiles_y = std::max(b.max_tiles_y, d.tiles_y);
    b.max_tiles = std::max(b.max_tiles, d.tiles_x * d.tiles_y);
    pixel_offset += static_cast<int64_t>(d.cam.width) * d.cam.height;
  }
  std::vector<int> widths, heights, counts;  // of the different sizes
  for (const ViewDesc& d : b.views) {
    size_t k = 0;
    while (k < counts.size() && (widths[k] != d.cam.width || heights[k] != d.cam.height)) ++k;
    if (k == counts.size()) {
      widths.push_back(d.cam.width);
      heights.push_back(d.cam.height);
      counts.push_back(0);
    }
    ++counts[k];
  }
  b.loss = loss_plan(widths.data(), heights.data(), counts.data(),
                     static_cast<int>(counts.size()));
  for (ViewDesc& d : b.views) {
    d.loss_tile_offset = static_cast<int32_t>(b.loss_blocks);
    d.l1_block_offset = static_cast<int32_t>(b.l1_blocks);
    b.loss_blocks += loss_blocks(d.cam.width, d.cam.height, b.loss);
    b.l1_blocks += loss_blocks(d.cam.width, d.cam.height, LossPlan{});
  }
  b.total_pixels = pixel_offset;
  b.total_tiles = tile_offset;
  b.total_rows = row_offset;
  return b;
}

void Frame::ensure_scan_scratch(int64_t n) {
  if (n <= scan_capacity_) return;
  const size_t bytes = scan_scratch_bytes(n) + 64;
  char* base = scan_scratch.reserve(bytes);
  scan_ = ScanScratch();
  scan_scratch_assign(scan_, base, n);
  scan_capacity_ = n;
}

void Frame::prepare(const ViewBatch& b, int n, int s, cudaStream_t stream) {
  if (!configured_) {
    configure_loss_kernel();
    configure_bin_kernels();
    configure_param_grads_kernel();
    PXS_CUDA(cudaGetLastError());
    configured_ = true;
  }
  batch = b;
  N = n;
  S = s;
  V = static_cast<int>(b.views.size());
  int widest = 1;  // the largest gaussian range of a view
  for (ViewDesc& d : batch.views) {
    if (!batch.own_ranges) {
      d.gauss_offset = 0;
      d.gauss_count = N;
    } else if (d.gauss_offset < 0 || d.gauss_count < 0 ||
               static_cast<int64_t>(d.gauss_offset) + d.gauss_count > N) {
      throw Error(PXS_ERR_INVALID, "a view's gaussian range lies outside the cloud");
    }
    widest = std::max(widest, d.gauss_count);
  }
  slot_stride = round_up(widest, kSortTile);
  const size_t slots = static_cast<size_t>(V) * static_cast<size_t>(slot_stride);
  d_views.reserve(static_cast<size_t>(std::max(V, 1)));
  if (V > 0)
    PXS_CUDA(cudaMemcpyAsync(d_views.get(), batch.views.data(), sizeof(ViewDesc) * V,
                             cudaMemcpyHostToDevice, stream));
  geom.reserve(slots);
  color.reserve(slots);
  depth_key.reserve(slots);
  sort_keys.reserve(slots);
  sort_vals.reserve(slots);
  sort_keys_alt.reserve(slots);
  sort_vals_alt.reserve(slots);
  const size_t row_chunks =
      direct_lists()
          ? static_cast<size_t>(std::max(batch.total_tiles, 1)) * direct_chunks_per_view(slot_stride)
          : static_cast<size_t>(std::max(batch.total_rows, 1)) * slot_chunks_per_view(slot_stride);
  row_chunk_counts.reserve(row_chunks);
  if (!direct_lists()) row_chunk_offsets.reserve(row_chunks);
  d_total_pairs.reserve(1);
  screen.reserve(slots);
  overflow.reserve(1);
  const size_t pixels = static_cast<size_t>(std::max<int64_t>(batch.total_pixels, 1));
  rgb.reserve(pixels * 3);
  dL.reserve(pixels * 3);
  transmittance.reserve(pixels);
  last.reserve(pixels);
  ranges.reserve(static_cast<size_t>(std::max(batch.total_tiles, 1)));
  tile_order.reserve(static_cast<size_t>(std::max(batch.total_tiles, 1)));
  order_work.reserve(64);
  tickets.reserve(2);
  order_ready = false;
  tile_counts.reserve(static_cast<size_t>(std::max(batch.total_tiles, 1)));
  tile_offsets.reserve(static_cast<size_t>(std::max(batch.total_tiles, 1)));
  n_chunks.reserve(1);
  d_total_records.reserve(1);
  loss_sums.reserve(static_cast<size_t>(2 * std::max(V, 1) + 1));
  loss_per_view.reserve(static_cast<size_t>(std::max(V, 1)));
  loss_total.reserve(1);
  hist.reserve(depth_sort_hist_entries(static_cast<int64_t>(slots), slot_stride));
  hist_scanned.reserve(depth_sort_scanned_entries(static_cast<int64_t>(slots), slot_stride));
  ensure_scan_scratch(std::max<int64_t>(std::max<int64_t>(static_cast<int64_t>(slots),
                                                          static_cast<int64_t>(hist.capacity())),
                                        static_cast<int64_t>(
                                            std::max<size_t>(row_chunks, batch.total_tiles))));
  // the chunk table depends on the rows as well as on the record capacity; size
  // it here, before any stream capture of the binning stage
  if (record_capacity > 0) ensure_chunks();
}

StepShape Frame::shape() const {
  return {N,
          S,
          V,
          slot_stride,
          batch.own_ranges,
          batch.total_pixels,
          batch.total_tiles,
          batch.total_rows,
          batch.max_tiles,
          batch.max_tiles_x,
          batch.max_tiles_y,
          batch.loss.form,
          batch.loss.rows,
          batch.loss_blocks,
          batch.l1_blocks,
          pair_capacity,
          record_capacity,
          max_chunks,
          direct_lists()};
}

void Frame::reserve_pairs(int64_t capacity) {
  if (capacity > INT32_MAX) throw Error(PXS_ERR_CAPACITY, "more than 2^31 tile pairs");
  if (capacity <= pair_capacity && tile_slots.get() != nullptr) return;
  const size_t cap = static_cast<size_t>(std::max<int64_t>(capacity, 1));
  tile_slots.reserve(cap);
  block_bits.reserve(cap);
  pair_capacity = static_cast<int64_t>(cap);
}

void Frame::reserve_records(int64_t capacity) {
  if (capacity > INT32_MAX) throw Error(PXS_ERR_CAPACITY, "more than 2^31 tile-row records");
  if (capacity <= record_capacity && rec_vals.get() != nullptr) return;
  const size_t cap = static_cast<size_t>(std::max<int64_t>(capacity, 1));
  rec_vals.reserve(cap);
  rec_xr.reserve(cap);
  record_capacity = static_cast<int64_t>(cap);
  ensure_chunks();
}

void Frame::ensure_chunks() {
  const int64_t need = max_row_chunks(std::max<int64_t>(record_capacity, 1), batch.total_rows);
  const size_t per = static_cast<size_t>(std::max(batch.max_tiles_x, 1));
  if (need > max_chunks || chunk_counts.capacity() < static_cast<size_t>(need) * per) {
    chunks.reserve(static_cast<size_t>(need));
    chunk_counts.reserve(static_cast<size_t>(need) * per);
    chunk_base.reserve(static_cast<size_t>(need) * per);
    max_chunks = need;
  }
}

void Frame::project(const float* params, cudaStream_t stream, bool want_debug,
                    bool whole_lists) {
  whole_lists_ = whole_lists;
  ProjectedSoA out;
  out.geom = geom.get();
  out.color = color.get();
  out.depth_key = depth_key.get();
  out.debug_cov = nullptr;
  if (want_debug) out.debug_cov = debug_cov.reserve(static_cast<size_t>(V) * slot_stride);
  launch_project(params, N, S, slot_stride, d_views.get(), V, out, !whole_lists,
                 batch.own_ranges, stream);
  PXS_CUDA(cudaGetLastError());
}

// The direct lists keep a map over a view's tiles in shared memory, and clear and
// read it once per 256 slots: their time grows with tiles times slots, that of the
// lists by rows with the records. The binning stage in us, directly / by rows: 37 /
// 58 (4k slots, 64 tiles), 47 / 68 (20k, 300), 68 / 91 (3 views of 38k, 1080), 76 /
// 93 (60k, 1938), 86 / 105 (150k, 1200), 168 / 221 (8 views of 150k, 300 tiles: 1.4M
// counts); past the line 131 / 119 (200k, 1900), 171 / 156 (400k, 1200), 272 / 197
// (8 of 100k, 1900), and 228 / 213 (800k, 300) for the slots alone.
bool Frame::direct_lists() const {
  return batch.max_tiles <= kMaxDirectTiles && slot_stride <= (1 << 18) &&
         static_cast<int64_t>(batch.total_tiles) * direct_chunks_per_view(slot_stride) <=
             1450000;
}

int64_t Frame::bin(bool host_sync, cudaStream_t stream) {
  order_ready = false;  // new tile lists
  const int64_t slots = static_cast<int64_t>(V) * slot_stride;
  if (slots == 0) {
    last_pair_count = 0;
    return 0;
  }
  // 1. every slot near to far within its view (stable: equal depths by index)
  depth_sort(depth_key.get(), slots, slot_stride, sort_keys_alt.get(), sort_vals_alt.get(),
             sort_keys.get(), sort_vals.get(), hist.get(), hist_scanned.get(), scan_, stream);
  const uint32_t* const k = sort_keys.get();  // kCulledKey for a culled slot
  uint32_t* const v = sort_vals.get();
  sorted_slots = v;
  if (batch.total_tiles == 0) {  // no view has a pixel: no lists
    PXS_CUDA(cudaMemsetAsync(d_total_pairs.get(), 0, sizeof(int64_t), stream));
    PXS_CUDA(cudaMemsetAsync(overflow.get(), 0, sizeof(int32_t), stream));
    last_pair_count = last_record_count = 0;
    sorted_pair_vals = tile_slots.get();
    PXS_CUDA(cudaGetLastError());
    return host_sync ? 0 : -1;
  }
  if (direct_lists()) {
    launch_direct_counts(v, k, geom.get(), !whole_lists_, d_views.get(), V, slot_stride,
                         batch.max_tiles, batch.total_tiles, row_chunk_counts.get(),
                         tile_counts.get(), overflow.get(), stream);
    exclusive_scan_i32_to_i64(tile_counts.get(), tile_offsets.get(), batch.total_tiles,
                              d_total_pairs.get(), scan_, stream);
    PXS_CUDA(cudaGetLastError());
    last_record_count = 0;
    if (host_sync) {
      PXS_CUDA(cudaMemcpyAsync(&last_pair_count, d_total_pairs.get(), sizeof(int64_t),
                               cudaMemcpyDeviceToHost, stream));
      PXS_CUDA(cudaStreamSynchronize(stream));
      if (last_pair_count > pair_capacity)
        reserve_pairs(last_pair_count + last_pair_count / 8 + 1024);
    }
    if (tile_slots.get() == nullptr) {
      if (!host_sync)
        throw Error(PXS_ERR_INVALID, "pair buffers must be reserved before an unsynchronised bin");
      reserve_pairs(1024);
    }
    launch_direct_expand(v, k, geom.get(), !whole_lists_, d_views.get(), V, slot_stride,
                         batch.max_tiles, batch.total_tiles, row_chunk_counts.get(),
                         tile_offsets.get(), tile_counts.get(), pair_capacity, tile_slots.get(),
                         ranges.get(), overflow.get(), stream);
    sorted_pair_vals = tile_slots.get();
    PXS_CUDA(cudaGetLastError());
    return host_sync ? last_pair_count : -1;
  }
  // 2. one record per covered tile row, grouped by row and near to far within
  //    a row: per (view, slot chunk) row counts, their scan in (row, chunk)
  //    order, then each chunk writes its records at its bases
  const int cpv = slot_chunks_per_view(slot_stride);
  const int64_t n_row_chunks = static_cast<int64_t>(batch.total_rows) * cpv;
  launch_slot_row_counts(v, k, geom.get(), d_views.get(), V, slot_stride,
                         batch.max_tiles_y, row_chunk_counts.get(), stream);
  exclusive_scan_i32_to_i64(row_chunk_counts.get(), row_chunk_offsets.get(), n_row_chunks,
                            d_total_records.get(), scan_, stream);
  PXS_CUDA(cudaGetLastError());
  if (host_sync) {
    PXS_CUDA(cudaMemcpyAsync(&last_record_count, d_total_records.get(), sizeof(int64_t),
                             cudaMemcpyDeviceToHost, stream));
    PXS_CUDA(cudaStreamSynchronize(stream));
    if (last_record_count > record_capacity)
      reserve_records(last_record_count + last_record_count / 8 + 1024);
  } else if (rec_vals.get() == nullptr || tile_slots.get() == nullptr) {
    throw Error(PXS_ERR_INVALID, "pair buffers must be reserved before an unsynchronised bin");
  }
  PXS_CUDA(cudaMemsetAsync(overflow.get(), 0, sizeof(int32_t), stream));
  launch_slot_row_expand(v, k, geom.get(), !whole_lists_, d_views.get(), V, slot_stride,
                         batch.max_tiles_y, row_chunk_offsets.get(), record_capacity,
                         rec_vals.get(), rec_xr.get(), stream);
  const uint32_t* rv = rec_vals.get();
  // 4. tile lengths from chunked rows, their offsets, then the lists themselves
  ensure_chunks();
  launch_tile_lists(row_chunk_offsets.get(), cpv, d_total_records.get(), record_capacity, rv,
                    rec_xr.get(), d_views.get(), V, batch.total_rows, batch.max_tiles_x,
                    max_chunks, chunks.get(), n_chunks.get(), chunk_counts.get(),
                    chunk_base.get(), tile_counts.get(), overflow.get(), stream);
  exclusive_scan_i32_to_i64(tile_counts.get(), tile_offsets.get(), batch.total_tiles,
                            d_total_pairs.get(), scan_, stream);
  PXS_CUDA(cudaGetLastError());
  int64_t K = -1;
  if (host_sync) {
    PXS_CUDA(cudaMemcpyAsync(&last_pair_count, d_total_pairs.get(), sizeof(int64_t),
                             cudaMemcpyDeviceToHost, stream));
    PXS_CUDA(cudaStreamSynchronize(stream));
    K = last_pair_count;
    if (K > pair_capacity) reserve_pairs(K + K / 8 + 1024);
  }
  launch_ranges_from_offsets(tile_counts.get(), tile_offsets.get(), batch.total_tiles,
                             pair_capacity, ranges.get(), overflow.get(), stream);
  launch_chunk_expand(chunks.get(), n_chunks.get(), rv, rec_xr.get(), d_views.get(), V,
                      batch.max_tiles_x, max_chunks, chunk_base.get(), tile_offsets.get(),
                      pair_capacity, tile_slots.get(), stream);
  sorted_pair_vals = tile_slots.get();
  PXS_CUDA(cudaGetLastError());
  return K;
}

// The heaviest-first tile order of the current lists, when a schedule wants it.
const int* Frame::ordered_tiles(int schedule, cudaStream_t stream) {
  if (schedule == 0) return nullptr;
  if (!order_ready) {
    launch_tile_order(ranges.get(), batch.total_tiles, tile_order.get(), order_work.get(),
                      stream);
    PXS_CUDA(cudaGetLastError());
    order_ready = true;
  }
  return tile_order.get();
}

void Frame::forward(cudaStream_t stream, unsigned long long* counts) {
  const int* order = counts ? nullptr : ordered_tiles(raster_config().forward_schedule, stream);
  have_block_bits =
      launch_forward(ranges.get(), sorted_pair_vals, geom.get(), color.get(),
                     d_views.get(), V, batch.total_tiles, rgb.get(), transmittance.get(),
                     last.get(), stream, counts, block_bits.get(), order, tickets.get());
  PXS_CUDA(cudaGetLastError());
}

Frame::~Frame() {
  if (copy_stream_) {
    cudaStreamSynchronize(copy_stream_);
    cudaStreamDestroy(copy_stream_);
  }
  for (cudaEvent_t e : band_done_)
    if (e) cudaEventDestroy(e);
  if (copied_) cudaEventDestroy(copied_);
}

cudaStream_t Frame::copy_stream() {
  if (copied_ == nullptr) PXS_CUDA(cudaEventCreateWithFlags(&copied_, cudaEventDisableTiming));
  if (copy_stream_ == nullptr)
    PXS_CUDA(cudaStreamCreateWithFlags(&copy_stream_, cudaStreamNonBlocking));
  return copy_stream_;
}

void Frame::begin_copies(cudaStream_t stream) {
  cudaStream_t copies = copy_stream();
  PXS_CUDA(cudaEventRecord(copied_, stream));
  PXS_CUDA(cudaStreamWaitEvent(copies, copied_, 0));
}

void Frame::join_copies(cudaStream_t stream) {
  PXS_CUDA(cudaEventRecord(copied_, copy_stream_));
  PXS_CUDA(cudaStreamWaitEvent(stream, copied_, 0));
}

// Whether the driver can copy to `p` directly (page-locked or device memory).
static bool page_locked(const void* p) {
  cudaPointerAttributes attributes;
  if (cudaPointerGetAttributes(&attributes, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return attributes.type != cudaMemoryTypeUnregistered;
}

// A band is at least the tiles that the device composites at once (8 CTAs on
// each of 148 SMs): with fewer the SMs would idle at every band's end. What the
// copies take (31 MB of a 1600x1200 image at 52 GB/s: 590 us) hides the
// compositing but for the first band's: a pinned 1600x1200 render of 300k
// gaussians 1009 -> 910 us. A copy to pageable memory is staged by the host, which
// fills and drains that pipeline for every band (20 to 50 us each): 20k gaussians at
// 1600x1200, with the transmittance, took 1.79 ms in one band and 2.12 in eight, but
// 12 Mpixels 8.01 and 7.75 ms, so there a band is also at least 1.25 Mpixels.
void Frame::forward_to_host(float* rgb_out, float* transmittance_out, cudaStream_t stream) {
  constexpr int kBandTiles = 148 * 8;
  const RasterConfig& rc = raster_config();
  const int tiles_x = batch.max_tiles_x, tiles_y = batch.max_tiles_y;
  int rows = tiles_y;
  if (V == 1 && rc.forward_px == 2 && rc.forward_schedule == 0 && tiles_x > 0)
    rows = std::max((kBandTiles + tiles_x - 1) / tiles_x, (tiles_y + kMaxBands - 1) / kMaxBands);
  if (rows < tiles_y && !(page_locked(rgb_out) && (transmittance_out == nullptr ||
                                                   page_locked(transmittance_out)))) {
    constexpr int kBandPixels = 5 << 18;
    const int bands = static_cast<int>(std::max<int64_t>(batch.total_pixels / kBandPixels, 1));
    rows = std::max(rows, (tiles_y + bands - 1) / bands);
  }
  const size_t pixels = static_cast<size_t>(batch.total_pixels);
  if (rows >= tiles_y || pixels == 0) {
    forward(stream);
    if (pixels == 0) return;
    PXS_CUDA(cudaMemcpyAsync(rgb_out, rgb.get(), pixels * 3 * sizeof(float),
                             cudaMemcpyDeviceToHost, stream));
    if (transmittance_out != nullptr)
      PXS_CUDA(cudaMemcpyAsync(transmittance_out, transmittance.get(), pixels * sizeof(float),
                               cudaMemcpyDeviceToHost, stream));
    return;
  }
  // every band is launched before the first copy: a copy to pageable memory
  // holds the host until it is done
  cudaStream_t copies = copy_stream();
  const int bands = (tiles_y + rows - 1) / rows;
  for (int b = 0; b < bands; ++b) {
    const int first = b * rows * tiles_x;
    const int count = std::min(rows, tiles_y - b * rows) * tiles_x;
    have_block_bits =
        launch_forward(ranges.get(), sorted_pair_vals, geom.get(), color.get(), d_views.get(), V,
                       count, rgb.get(), transmittance.get(), last.get(), stream, nullptr,
                       block_bits.get(), nullptr, tickets.get(), first);
    PXS_CUDA(cudaGetLastError());
    if (band_done_[b] == nullptr)
      PXS_CUDA(cudaEventCreateWithFlags(&band_done_[b], cudaEventDisableTiming));
    PXS_CUDA(cudaEventRecord(band_done_[b], stream));
  }
  const size_t width = static_cast<size_t>(batch.views[0].cam.width);
  for (int b = 0; b < bands; ++b) {
    const size_t p0 = static_cast<size_t>(b) * rows * kTile * width;
    const size_t p1 = std::min(pixels, p0 + static_cast<size_t>(rows) * kTile * width);
    PXS_CUDA(cudaStreamWaitEvent(copies, band_done_[b], 0));
    PXS_CUDA(cudaMemcpyAsync(rgb_out + 3 * p0, rgb.get() + 3 * p0, (p1 - p0) * 3 * sizeof(float),
                             cudaMemcpyDeviceToHost, copies));
    if (transmittance_out != nullptr)
      PXS_CUDA(cudaMemcpyAsync(transmittance_out + p0, transmittance.get() + p0,
                               (p1 - p0) * sizeof(float), cudaMemcpyDeviceToHost, copies));
  }
  join_copies(stream);
}

void Frame::loss(const float* target, float ssim_weight, int mode, float* grad_out,
                 cudaStream_t stream) {
  LossParams lp;
  ssim_kernel_weights(lp.kernel);
  lp.ssim_weight = ssim_weight;
  lp.mode = mode;
  const bool ssim = mode == 1 || ssim_weight > 0.f;
  launch_loss(rgb.get(), target, d_views.get(), V, ssim ? batch.loss_blocks : batch.l1_blocks,
              ssim ? batch.loss : LossPlan{}, lp, grad_out, loss_sums.get(), loss_per_view.get(),
              loss_total.get(), stream);
  PXS_CUDA(cudaGetLastError());
}

void Frame::backward(const float* dL_drgb, cudaStream_t stream) {
  const size_t slots = static_cast<size_t>(V) * static_cast<size_t>(slot_stride);
  PXS_CUDA(cudaMemsetAsync(screen.get(), 0, sizeof(ScreenGrad) * slots, stream));
  const int* order = ordered_tiles(raster_config().backward_schedule, stream);
  launch_backward(ranges.get(), sorted_pair_vals, geom.get(), color.get(),
                  d_views.get(), V, batch.total_tiles, transmittance.get(), last.get(), dL_drgb,
                  screen.get(), stream, have_block_bits ? block_bits.get() : nullptr, order,
                  tickets.get() + 1);
  PXS_CUDA(cudaGetLastError());
}

void Frame::param_grads(const float* params, float* grads, float* screen_gradient,
                        int32_t* visible_count, cudaStream_t stream) {
  launch_param_grads(params, N, S, slot_stride, d_views.get(), V, depth_key.get(), geom.get(),
                     color.get(), screen.get(), grads, screen_gradient, visible_count, stream);
  PXS_CUDA(cudaGetLastError());
}

}  // namespace pxs
