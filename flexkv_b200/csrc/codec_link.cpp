#include "codec_link.h"

#include <algorithm>

#include "kernels/kv_compress.h"
#include "kernels/kv_quant.h"

namespace fkv {

namespace {
class DeviceScope {
 public:
  explicit DeviceScope(int device) {
    if (cudaGetDevice(&before_) != cudaSuccess) before_ = -1;
    cudaSetDevice(device);
  }
  ~DeviceScope() { if (before_ >= 0) cudaSetDevice(before_); }

 private:
  int before_ = -1;
};
}  // namespace

namespace {
// Slot bytes of the last piece of a restore: smaller ones come in copies too short for the link.
constexpr int64_t kRowRampBytes = 12 << 20;
}  // namespace

CodecLink::CodecLink(int device, int num_layers, int kv_dim, int64_t chunk_slot, int64_t staging_bytes)
    : device_(device), num_layers_(num_layers), chunk_slot_(chunk_slot), staging_bytes_(staging_bytes) {
  DeviceScope on(device_);
  // in place before the first op; refused memory leaves the ops with the kernel
  const int64_t block = chunk_slot * kv_dim * num_layers;
  if (block > 0) ce_staging_prepare(staging_, std::max<int64_t>(1, staging_bytes_ / block), block);
}

CodecLink::~CodecLink() {
  DeviceScope on(device_);
  if (staging_.copy_stream) cudaStreamSynchronize(staging_.copy_stream);
  ce_staging_free(staging_);
  (void)cudaGetLastError();
}

bool CodecLink::plan(const KvCopyParams& p, int64_t min_bytes, int64_t ramp_bytes, CeStagePlan& out) {
  if (p.num_pairs * p.c_block_stride < min_bytes) return false;
  if (!ce_host_blocks_abut(p, num_layers_, chunk_slot_) || staging_.block_bytes != p.c_block_stride) return false;
  const int64_t min_run = std::max<int64_t>(1, (CePolicy().min_bytes_per_copy + p.c_block_stride - 1) / p.c_block_stride);
  return ce_plan_staged(p, const_cast<int64_t*>(p.gpu_blocks), const_cast<int64_t*>(p.cpu_blocks), min_run,
                        staging_.blocks, out, ramp_bytes);
}

cudaError_t CodecLink::quant_fp8(const KvCopyParams& p, int num_ctas, cudaStream_t stream) {
  CeStagePlan pl;
  if (!plan(p, kMinQuantBytes, kCeRampBytes, pl)) return launch_kv_quant_fp8(p, num_ctas, stream);
  ++staged_ops_;
  return ce_copy_staged(
      p, pl, staging_,
      [num_ctas](const KvCopyParams& q, int64_t, cudaStream_t s) { return launch_kv_quant_fp8(q, num_ctas, s); }, stream);
}

namespace {

// Copies of one piece of packed blocks: rows at a constant pitch, as wide as the largest tile among them.
struct RowCopy {
  int64_t offset, pitch, width, rows;
};

// The copies that bring the tiles of `piece` in, judged by its size-table rows; false when the kernel does better.
bool plan_rows(const KvCopyParams& p, const uint32_t* sizes, const CeHostRun& piece, std::vector<RowCopy>& out) {
  const int64_t elems = p.chunk_bytes / 2;
  const int tiles = (int)compress_tiles_per_chunk(elems);
  const int classes = p.kv_dim * tiles;
  const int64_t rows = piece.len * p.num_layers;
  std::vector<uint32_t> width((size_t)classes, 0);
  int64_t used = 0;
  const uint32_t* sz = sizes + piece.cpu_block * p.num_layers * classes;
  for (int64_t r = 0; r < rows; ++r)
    for (int k = 0; k < classes; ++k, ++sz) {
      const int64_t left = elems - (int64_t)(k % tiles) * kCompressTileElems;
      const uint32_t cap = 16u + 2u * (uint32_t)std::min<int64_t>(left, kCompressTileElems);
      if (*sz < 32 || *sz > cap || (*sz & 15u)) return false;      // the kernel reports it
      width[(size_t)k] = std::max(width[(size_t)k], *sz);
      used += *sz;
    }
  // rows of whole 128-byte lines: 55.3 GB/s against 54.1 (11 KiB rows). Every slot is a multiple of 128 bytes.
  for (uint32_t& w : width) w = (w + 127u) & ~127u;
  out.clear();
  int64_t apart = 0;
  uint32_t widest = 0;
  for (uint32_t w : width) { apart += rows * w; widest = std::max(widest, w); }
  // A copy costs 3.5 us beside its bytes, as much as 190 KB of them: one copy of all tiles where they are of one size
  // and at one pitch, else one for each class.
  constexpr int64_t kCopyCostBytes = 190 << 10;
  const int64_t layer_slot = p.c_layer_stride, pitch = p.c_kv_stride / tiles;
  const bool even = tiles == 1 || elems % kCompressTileElems == 0;    // every tile slot of the same size
  int64_t moved;
  if (even && rows * classes * (int64_t)widest - apart < (classes - 1) * kCopyCostBytes) {
    out.push_back(RowCopy{0, pitch, widest, rows * classes});
    moved = rows * classes * (int64_t)widest + kCopyCostBytes;
  } else {
    for (int k = 0; k < classes; ++k)
      out.push_back(RowCopy{(k / tiles) * p.c_kv_stride + (int64_t)(k % tiles) * kCompressTileSlot, layer_slot,
                            width[(size_t)k], rows});
    moved = apart + classes * kCopyCostBytes;
  }
  // 54.5 GB/s in long copies against the kernel's 51 for the used bytes alone. Below 2 MB (40 us) the difference is
  // less than what changing to the kernel and back costs.
  return moved < used + std::max<int64_t>(used / 16, 2 << 20);
}

}  // namespace

cudaError_t CodecLink::compress_bf16(const KvCopyParams& p, uint32_t* size_table, int layers_total, int num_ctas,
                                     int staged_ctas, cudaStream_t stream) {
  CeStagePlan pl;
  // chunks that the codec refuses (no multiple of 1024 values) are refused before a copy is planned for them
  if (!p.h2d || size_table == nullptr || p.chunk_bytes < kMinRowChunk || p.chunk_bytes % 2048 != 0 || layers_total != num_layers_ ||
      !plan(p, kMinRowBytes, kRowRampBytes, pl))
    return launch_kv_compress_bf16(p, size_table, layers_total, num_ctas, stream);
  ++staged_ops_;
  const int64_t row_entries = (int64_t)p.num_layers * p.kv_dim * compress_tiles_per_chunk(p.chunk_bytes / 2);
  std::vector<RowCopy> rows;
  const uint8_t* host = reinterpret_cast<const uint8_t*>(p.cpu_base);
  CeLinkCopy link;
  link.worth = [&](const CeHostRun& piece) { return plan_rows(p, size_table, piece, rows); };
  link.copy = [&](const CeHostRun& piece, uint8_t* staged, cudaStream_t s) -> cudaError_t {
    const uint8_t* from = host + piece.cpu_block * p.c_block_stride;
    for (const RowCopy& r : rows) {
      const cudaError_t e = cudaMemcpy2DAsync(staged + r.offset, (size_t)r.pitch, from + r.offset, (size_t)r.pitch,
                                              (size_t)r.width, (size_t)r.rows, cudaMemcpyHostToDevice, s);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  };
  return ce_copy_staged(
      p, pl, staging_,
      [&](const KvCopyParams& q, int64_t host_block, cudaStream_t s) {
        const bool staged = q.cpu_base != p.cpu_base;
        return launch_kv_compress_bf16(q, size_table + host_block * row_entries, layers_total,
                                       staged ? staged_ctas : num_ctas, s);
      },
      stream, &link);
}

}  // namespace fkv
