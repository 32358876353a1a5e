// GPU<->host moves of a packed host pool, on the copy engines where the host blocks allow it.
//
// The codec kernels read or write the host pool themselves, so their traffic crosses the link as SM-issued requests:
// 52.5 GB/s out, 51 in, and 37 each way with both directions busy (B200). Where the op's host blocks come in rows the
// kernel packs into a device staging buffer instead (or unpacks out of it) and a copy engine moves the packed blocks
// at 56.5 / 55, or 48 each way: the staged route of ce_copy.h with a codec kernel in the place of the plain gather.
// The packed bytes are the same either way. Blocks that stand alone, pools shared by several ranks of a launch and
// hosts without memory for the staging buffers stay with the kernel.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

#include "ce_copy.h"

namespace fkv {

// One GPU, one direction. quant_fp8() or compress_bf16() is called by one thread at a time.
class CodecLink {
 public:
  // Ops of fewer host bytes stay with the kernel, whose start and end are shorter. B200, us, kernel -> staged: fp8 out
  // 483 (25 MB) -> 483, 944 (50 MB) -> 910, 5025 (268 MB) -> 4707; lossless in, llama3-8b pages 885 (66 MB of slots)
  // -> 873, 3451 (258 MB) -> 3305, 6858 -> 6538, deepseek-v3 pages 893 (64 MB) -> 931, 1751 (127 MB) -> 1750,
  // 3430 (254 MB) -> 3382.
  static constexpr int64_t kMinQuantBytes = 48 << 20, kMinRowBytes = 128 << 20;
  // Rows of smaller chunks (bf16 bytes) are too short for a copy engine: 48.2 GB/s at 2048 values, the kernel 50.4.
  static constexpr int64_t kMinRowChunk = 8192;

  // `chunk_slot`: bytes a packed (layer, kv, block) chunk takes in the host pool; `staging_bytes` of each of the two
  // staging buffers.
  CodecLink(int device, int num_layers, int kv_dim, int64_t chunk_slot, int64_t staging_bytes = kCeStageBytes);
  ~CodecLink();
  CodecLink(const CodecLink&) = delete;
  CodecLink& operator=(const CodecLink&) = delete;

  // Block-scaled fp8, as launch_kv_quant_fp8. `p.gpu_blocks` and `p.cpu_blocks` are host memory that the kernel can
  // read; their pairs may be reordered. They and the status words are in use until `stream` has passed the op.
  cudaError_t quant_fp8(const KvCopyParams& p, int num_ctas, cudaStream_t stream);
  // The lossless codec, as launch_kv_compress_bf16; `size_table` is host memory that the kernel can read. Restores are
  // staged: only the used bytes of the tile slots cross, as rows of a 2-D copy, each class of tiles (K or V, tile of
  // the chunk) as wide as its largest tile in the piece. Offloads stay with the kernel: the sizes are not known before
  // a piece is packed, and rows of 11 KiB go out at 51.7 GB/s where the kernel reaches 52.5.
  // `staged_ctas` takes the place of `num_ctas` where the kernel unpacks out of the staging buffer.
  cudaError_t compress_bf16(const KvCopyParams& p, uint32_t* size_table, int layers_total, int num_ctas,
                            int staged_ctas, cudaStream_t stream);
  uint64_t staged_ops() const { return staged_ops_; }

 private:
  bool plan(const KvCopyParams& p, int64_t min_bytes, int64_t ramp_bytes, CeStagePlan& out);

  int device_, num_layers_;
  int64_t chunk_slot_, staging_bytes_;
  CeStaging staging_;
  uint64_t staged_ops_ = 0;
};

}  // namespace fkv
