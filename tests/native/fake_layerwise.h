// What layerwise restores need beside fake_cuda.h.
#pragma once
#include "fake_cuda.h"
#include "layerwise_group.h"

extern "C" {
cudaError_t cudaGetDriverEntryPoint(const char*, void**, unsigned long long, cudaDriverEntryPointQueryResult*) {
  return cudaErrorNotSupported;
}
cudaError_t cudaLaunchHostFunc(cudaStream_t s, cudaHostFn_t fn, void* arg) {
  fake::push(s, [=] { fn(arg); });
  return cudaSuccess;
}
}
namespace fkv {
cudaError_t launch_kv_compress_bf16(const KvCopyParams&, uint32_t*, int, int, cudaStream_t) { return cudaErrorNotSupported; }
int64_t SsdIoEngine::transfer(uint8_t*, const int64_t*, const int64_t*, int64_t n, bool, const SsdLayout&, int, int,
                              uint8_t*) { return n; }
}  // namespace fkv
