// The CUDA runtime calls of the transfer code, executed on the CPU as late as a GPU may: what is queued on a stream runs
// when that stream is waited for, and not before. Kernels are host_kv_copy(). A chosen launch can fail.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <mutex>

#include "kernels/kv_copy.h"

namespace fake {

struct Mark {                  // the place of an event's last record
  cudaStream_t stream = nullptr;
  uint64_t id = 0;
};
struct Op {
  uint64_t id;
  std::function<void()> run;   // empty: wait for `until`
  Mark until;
};

inline std::recursive_mutex mu;
inline uint64_t next_id = 1;
inline std::map<cudaStream_t, std::deque<Op>> streams;
inline std::map<cudaEvent_t, Mark> marks;
inline std::atomic<int> launches{0}, fail_launch{-1};   // the launch of this number fails
inline std::atomic<size_t> device_bytes{0};             // asked for with cudaMalloc so far
inline std::function<void(const fkv::KvCopyParams&)> on_launch;   // on the launching thread, before a launch

inline void drain(cudaStream_t s, uint64_t upto) {
  auto& q = streams[s];
  while (!q.empty() && q.front().id <= upto) {
    Op op = std::move(q.front());
    q.pop_front();
    if (op.run) op.run();
    else if (op.until.id) drain(op.until.stream, op.until.id);
  }
}
inline void push(cudaStream_t s, std::function<void()> f, Mark until = {}) {
  std::lock_guard<std::recursive_mutex> g(mu);
  streams[s].push_back(Op{next_id++, std::move(f), until});
}
inline size_t in_flight() {
  std::lock_guard<std::recursive_mutex> g(mu);
  size_t n = 0;
  for (auto& s : streams)
    for (auto& op : s.second) n += op.run ? 1 : 0;
  return n;
}
inline std::atomic<uintptr_t> next_handle{0x1000};

}  // namespace fake

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) { *lo = *hi = 0; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
  fake::device_bytes += n;
  *p = std::malloc(n ? n : 1);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::malloc(n ? n : 1); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  fake::push(st, [=] { std::memcpy(d, s, n); });
  return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t st) {
  fake::push(st, [=] {
    for (size_t i = 0; i < h; ++i) std::memcpy((char*)d + i * dp, (const char*)s + i * sp, w);
  });
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(fake::next_handle++);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> g(fake::mu);
  fake::drain(s, UINT64_MAX);
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  std::lock_guard<std::recursive_mutex> g(fake::mu);
  for (auto& s : fake::streams) fake::drain(s.first, UINT64_MAX);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = reinterpret_cast<cudaEvent_t>(fake::next_handle++);
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::lock_guard<std::recursive_mutex> g(fake::mu);
  fake::marks[e] = fake::Mark{s, fake::next_id - 1};
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::lock_guard<std::recursive_mutex> g(fake::mu);
  const fake::Mark m = fake::marks[e];
  if (m.id) fake::drain(m.stream, m.id);
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) { return cudaEventSynchronize(e); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  std::lock_guard<std::recursive_mutex> g(fake::mu);
  fake::push(s, nullptr, fake::marks[e]);
  return cudaSuccess;
}
}

namespace fkv {

cudaError_t kv_copy_load_kernels() { return cudaSuccess; }
cudaError_t launch_kv_copy(const KvCopyParams& p, const KvCopyLaunch&, cudaStream_t s) {
  if (fake::on_launch) fake::on_launch(p);
  if (fake::launches++ == fake::fail_launch) return cudaErrorLaunchOutOfResources;
  fake::push(s, [p] {
    if (const int err = host_kv_copy(p, 1))
      for (int b = 0; b < kStatusWords; ++b)
        if (err & (1 << b)) p.status[b] = 1;
    if (p.done_counter)
      for (int l = p.layer_start; l < p.layer_start + p.num_layers; ++l) p.dev_flags[l] = p.host_flags[l] = p.epoch;
  });
  return cudaSuccess;
}
cudaError_t launch_kv_copy_refshape(const KvCopyParams& p, int, cudaStream_t s) { return launch_kv_copy(p, {}, s); }

}  // namespace fkv
