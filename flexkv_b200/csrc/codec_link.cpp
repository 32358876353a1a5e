#include "codec_link.h"

#include <algorithm>

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

CodecLink::CodecLink(int device, int num_layers, int kv_dim, int64_t chunk_slot)
    : device_(device), num_layers_(num_layers), chunk_slot_(chunk_slot) {
  DeviceScope on(device_);
  // in place before the first op; refused memory leaves the ops with the kernel
  ce_staging_prepare(staging_, 0, chunk_slot * kv_dim * num_layers);
}

CodecLink::~CodecLink() {
  DeviceScope on(device_);
  if (staging_.copy_stream) cudaStreamSynchronize(staging_.copy_stream);
  ce_staging_free(staging_);
  (void)cudaGetLastError();
}

bool CodecLink::plan(const KvCopyParams& p, CeStagePlan& out) {
  if (!ce_host_blocks_abut(p, num_layers_, chunk_slot_) || !ce_staging_prepare(staging_, 0, p.c_block_stride)) return false;
  const int64_t min_run = std::max<int64_t>(1, (CePolicy().min_bytes_per_copy + p.c_block_stride - 1) / p.c_block_stride);
  return ce_plan_staged(p, const_cast<int64_t*>(p.gpu_blocks), const_cast<int64_t*>(p.cpu_blocks), min_run,
                        staging_.blocks, out);
}

cudaError_t CodecLink::quant_fp8(const KvCopyParams& p, int num_ctas, cudaStream_t stream) {
  CeStagePlan pl;
  if (!plan(p, pl)) return launch_kv_quant_fp8(p, num_ctas, stream);
  ++staged_ops_;
  return ce_copy_staged(
      p, pl, staging_,
      [num_ctas](const KvCopyParams& q, int64_t, cudaStream_t s) { return launch_kv_quant_fp8(q, num_ctas, s); }, stream);
}

}  // namespace fkv
