#include "kv_quant.h"

#include <cfloat>

#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "ptx_sm100.cuh"

namespace fkv {
namespace {

// A CTA of 256 threads runs tile pipelines of T threads each, two CTAs to an SM. Against the host the link bounds it.
// Within HBM (packing into the staging buffer of the copy-engine route) the latency of the arithmetic does. Eight lanes
// hold a group, 16 values each, so that four groups share a warp and a maximum takes three shuffles instead of five.
// Packing within HBM, GB/s of bf16 on B200, 48 / 148 CTAs: a warp per group 144 / 438 (128 threads), eight lanes per
// group 226 / 680, 256 threads and quant2 below 371 / 1097; unpacking 504 / 1481 -> 685 / 1973. The short tile of a
// small chunk (one or two KV heads per rank) takes 32 values per thread as a full one does, in a pipeline of its own.
constexpr int kCtaThreads = 256;
constexpr int kLanesPerGroup = 8;
constexpr uint64_t kWaitBudgetNs = 2000000000ull;

template <int T>
struct Pipe {
  static constexpr int kTileElems = 32 * T;  // T = 256: 16 KiB of bf16 in, 8 KiB + 256 B out
  static constexpr int kGroups = kCtaThreads / T;
};

template <bool PACK, int T>
struct __align__(16) Smem {
  static constexpr int kTileElems = Pipe<T>::kTileElems;
  // host reads need more tiles in flight than HBM reads
  static constexpr int kInStages = PACK ? 4 : 6;
  // pack: in = bf16 tile; unpack: in = e4m3 payload followed by its scales
  uint8_t in[kInStages][PACK ? kTileElems * 2 : kTileElems + kTileElems / kQuantGroup * 4];
  uint8_t out[2][kTileElems * 2];
  float out_scales[2][kTileElems / kQuantGroup];
};

// barrier among the threads of one pipeline (hardware barrier 1 + pipeline; 0 is __syncthreads')
template <int T>
__device__ __forceinline__ void pipe_sync(int pipe) {
  asm volatile("bar.sync %0, %1;" ::"r"(pipe + 1), "n"(T) : "memory");
}

// The scale of a group with this largest magnitude. Below FLT_MIN it would be flushed to zero (the build flushes
// subnormals) and its reciprocal would be infinite: zeros would become NaN codes, all else the largest code.
__device__ __forceinline__ float group_scale(float amax) {
  return amax > 0.f ? fmaxf(__fdiv_rn(amax, 448.f), FLT_MIN) : 1.f;
}

// largest value among the lanes that hold a group
__device__ __forceinline__ float group_max(float v) {
#pragma unroll
  for (int o = kLanesPerGroup / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ float2 bf16x2_floats(uint32_t w) {
  const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&w);
  return make_float2(__low2float(h), __high2float(h));
}

// The e4m3 codes of fdiv_rn(x, scale) for a pair of values. `lo` and `hi` are 1 / scale made smaller and larger by
// 2^-20, far more than the rounding of the reciprocal and of a product: the quotient lies between x * lo and x * hi,
// rounding to e4m3 is monotone, so where both have the same code the quotient has it too and no division is needed
// (one pair in some 5000 is divided). That needs a finite 1 / scale, which group_scale() sees to; zero, infinite and
// NaN values and an infinite scale then give the same in both forms.
__device__ __forceinline__ uint32_t quant2(float2 x, float scale, float lo, float hi) {
  const uint32_t a = __nv_cvt_float2_to_fp8x2(make_float2(__fmul_rn(x.x, lo), __fmul_rn(x.y, lo)), __NV_SATFINITE, __NV_E4M3);
  const uint32_t b = __nv_cvt_float2_to_fp8x2(make_float2(__fmul_rn(x.x, hi), __fmul_rn(x.y, hi)), __NV_SATFINITE, __NV_E4M3);
  if (a == b) return a;
  return __nv_cvt_float2_to_fp8x2(make_float2(__fdiv_rn(x.x, scale), __fdiv_rn(x.y, scale)), __NV_SATFINITE, __NV_E4M3);
}

// eight values -> their codes
__device__ __forceinline__ uint2 quant8(const float2 (&x)[4], float scale, float lo, float hi) {
  uint32_t q[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = quant2(x[i], scale, lo, hi);
  return make_uint2(q[0] | (q[1] << 16), q[2] | (q[3] << 16));
}

// two e4m3 codes -> two bf16 values
__device__ __forceinline__ uint32_t dequant2(uint32_t q, float scale) {
  const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(q & 0xffffu), __NV_E4M3);
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
  __nv_bfloat162 o = __floats2bfloat162_rn(__fmul_rn(f.x, scale), __fmul_rn(f.y, scale));
  return *reinterpret_cast<uint32_t*>(&o);
}

template <bool PACK, int T>
__global__ void __launch_bounds__(kCtaThreads, 2) kv_quant_fp8_kernel(const __grid_constant__ KvCopyParams p,
                                                                      int tiles_per_chunk) {
  constexpr int kInStages = Smem<PACK, T>::kInStages, kTileElems = Pipe<T>::kTileElems, kGroups = Pipe<T>::kGroups;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  struct State {
    uint64_t full[kInStages];
    uint64_t dst[kInStages];       // destination of the tile's payload
    uint64_t dst2[kInStages];      // pack: destination of the tile's scales
    int32_t elems[kInStages];      // 0 = skipped tile
    int abort;
  };
  __shared__ __align__(8) State state[kGroups];
  const int pipe = threadIdx.x / T, tid = threadIdx.x % T, warp = tid >> 5, lane = tid & 31;
  Smem<PACK, T>& sm = reinterpret_cast<Smem<PACK, T>*>(smem_raw)[pipe];
  uint64_t* const full = state[pipe].full;
  uint64_t* const s_dst = state[pipe].dst;
  uint64_t* const s_dst2 = state[pipe].dst2;
  int32_t* const s_elems = state[pipe].elems;
  int& s_abort = state[pipe].abort;
  const int64_t vcta = (int64_t)blockIdx.x * kGroups + pipe, vgrid = (int64_t)gridDim.x * kGroups;

  if (tid == 0) {
    for (int s = 0; s < kInStages; ++s) ptx::mbar_init(&full[s], 1);
    s_abort = 0;
    ptx::fence_mbar_init();
  }
  pipe_sync<T>(pipe);

  const int64_t chunk_elems = p.chunk_bytes / 2;
  const int32_t span = p.num_layers * p.kv_dim * tiles_per_chunk;
  const int64_t total = (int64_t)span * p.num_pairs;
  // every pipeline owns one contiguous run of tiles: consecutive tiles share their block ids (fetched
  // once per pair, possibly over PCIe) and their size-table neighbourhood
  const int64_t per_pipe = (total + vgrid - 1) / vgrid;
  const int64_t first = vcta * per_pipe, step = 1;
  const int64_t n_mine = first < total ? (total - first < per_pipe ? total - first : per_pipe) : 0;
  // thread 0 keeps the ids of the pair it is working on and asks for the next pair's early
  int32_t id_pair = -1;
  int64_t id_g = 0, id_c = 0, nx_g = 0, nx_c = 0;
  auto pair_ids = [&](int32_t pair, int64_t& g, int64_t& c) {
    if (pair != id_pair) {
      if (pair == id_pair + 1 && id_pair >= 0) { id_g = nx_g; id_c = nx_c; }
      else { id_g = __ldg(p.gpu_blocks + pair); id_c = __ldg(p.cpu_blocks + pair); }
      id_pair = pair;
      if (pair + 1 < p.num_pairs) { nx_g = __ldg(p.gpu_blocks + pair + 1); nx_c = __ldg(p.cpu_blocks + pair + 1); }
    }
    g = id_g; c = id_c;
  };
  int err = 0;
  uint32_t phases = 0;   // every thread tracks the parity of each stage's next completion

  // thread 0: address generation and all bulk copies
  auto issue_load = [&](int64_t it) {
    const int st = (int)(it % kInStages);
    const int64_t t = first + it * step;
    const int32_t pair = (int32_t)(t / span), r = (int32_t)(t % span);
    const int s_ = r % tiles_per_chunk, q = r / tiles_per_chunk;
    const int kv = q % p.kv_dim, layer = p.layer_start + q / p.kv_dim;
    int64_t gblk, cblk;
    pair_ids(pair, gblk, cblk);
    bool ok = true;
    if (p.gpu_num_blocks > 0 && (gblk < 0 || gblk >= p.gpu_num_blocks)) { err |= KV_ERR_GPU_BLOCK_RANGE; ok = false; }
    if (p.cpu_num_blocks > 0 && (cblk < 0 || cblk >= p.cpu_num_blocks)) { err |= KV_ERR_CPU_BLOCK_RANGE; ok = false; }
    const int64_t e0 = (int64_t)s_ * kTileElems;
    const int64_t left = chunk_elems - e0;
    const int32_t elems = (int32_t)(left < kTileElems ? left : kTileElems);
    const uint64_t g = kv_gpu_tensor(p, layer * p.idx_layer_mul + kv * p.idx_kv_mul) + layer * p.g_layer_stride +
                       kv * p.g_kv_stride + gblk * p.g_block_stride + p.g_off + e0 * 2;
    const uint64_t c = p.cpu_base + layer * p.c_layer_stride + kv * p.c_kv_stride + cblk * p.c_block_stride + p.c_off;
    const uint64_t c_payload = c + e0, c_scales = c + chunk_elems + (e0 / kQuantGroup) * 4;
    if (!ok) {
      s_elems[st] = 0;
      ptx::mbar_arrive(&full[st]);
      return;
    }
    s_elems[st] = elems;
    if (PACK) {
      s_dst[st] = c_payload;
      s_dst2[st] = c_scales;
      ptx::mbar_expect_tx(&full[st], (uint32_t)elems * 2);
      ptx::bulk_g2s(sm.in[st], reinterpret_cast<const void*>(g), (uint32_t)elems * 2, &full[st]);
    } else {
      s_dst[st] = g;
      const uint32_t sc_bytes = (uint32_t)(elems / kQuantGroup) * 4;
      ptx::mbar_expect_tx(&full[st], (uint32_t)elems + sc_bytes);
      ptx::bulk_g2s(sm.in[st], reinterpret_cast<const void*>(c_payload), (uint32_t)elems, &full[st]);
      ptx::bulk_g2s(sm.in[st] + kTileElems, reinterpret_cast<const void*>(c_scales), sc_bytes, &full[st]);
    }
  };

  if (tid == 0)
    for (int64_t it = 0; it < n_mine && it < kInStages - 1; ++it) issue_load(it);

  for (int64_t it = 0; it < n_mine; ++it) {
    const int st = (int)(it % kInStages), ob = (int)(it & 1);
    if (tid == 0) {
      // stage (it-1) % kInStages was drained by everyone before the barrier that ended iteration it-1
      if (it + kInStages - 1 < n_mine) issue_load(it + kInStages - 1);
      if (it >= 2) ptx::bulk_wait_read<1>();   // the store of tile it-2 has finished reading out[ob]
    }
    pipe_sync<T>(pipe);
    if (!ptx::mbar_wait_bounded(&full[st], (phases >> st) & 1u, kWaitBudgetNs)) s_abort = 1;
    phases ^= 1u << st;
    pipe_sync<T>(pipe);
    if (*reinterpret_cast<volatile int*>(&s_abort)) break;      // the pipeline leaves together
    const int elems = s_elems[st];
    const int groups = elems / kQuantGroup;      // a multiple of 4: a warp's four groups are there or not together
    const int l8 = lane % kLanesPerGroup;        // this lane's values: 8 * l8 .. + 7 of either half of its group
    for (int gidx = warp * 4 + lane / kLanesPerGroup; gidx < groups; gidx += T / kLanesPerGroup) {
      if (PACK) {
        const uint4* src = reinterpret_cast<const uint4*>(sm.in[st]) + gidx * (kQuantGroup / 8) + l8;
        const uint4 a = src[0], b = src[kLanesPerGroup];
        const float2 xa[4] = {bf16x2_floats(a.x), bf16x2_floats(a.y), bf16x2_floats(a.z), bf16x2_floats(a.w)};
        const float2 xb[4] = {bf16x2_floats(b.x), bf16x2_floats(b.y), bf16x2_floats(b.z), bf16x2_floats(b.w)};
        float m = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          m = fmaxf(m, fmaxf(fmaxf(fabsf(xa[i].x), fabsf(xa[i].y)), fmaxf(fabsf(xb[i].x), fabsf(xb[i].y))));
        const float amax = group_max(m);
        const float scale = group_scale(amax);
        const float inv = __frcp_rn(scale), lo = inv * (1.f - 0x1p-20f), hi = inv * (1.f + 0x1p-20f);
        uint2* dst = reinterpret_cast<uint2*>(sm.out[ob]) + gidx * (kQuantGroup / 8) + l8;
        dst[0] = quant8(xa, scale, lo, hi);
        dst[kLanesPerGroup] = quant8(xb, scale, lo, hi);
        if (l8 == 0) sm.out_scales[ob][gidx] = scale;
      } else {
        const uint2* src = reinterpret_cast<const uint2*>(sm.in[st]) + gidx * (kQuantGroup / 8) + l8;
        const uint2 a = src[0], b = src[kLanesPerGroup];
        const float scale = reinterpret_cast<const float*>(sm.in[st] + kTileElems)[gidx];
        uint4* dst = reinterpret_cast<uint4*>(sm.out[ob]) + gidx * (kQuantGroup / 8) + l8;
        dst[0] = make_uint4(dequant2(a.x, scale), dequant2(a.x >> 16, scale), dequant2(a.y, scale),
                            dequant2(a.y >> 16, scale));
        dst[kLanesPerGroup] = make_uint4(dequant2(b.x, scale), dequant2(b.x >> 16, scale), dequant2(b.y, scale),
                                         dequant2(b.y >> 16, scale));
      }
    }
    ptx::fence_proxy_async_smem();   // generic-proxy writes to out[] before the bulk store reads them
    pipe_sync<T>(pipe);
    if (tid == 0) {
      if (elems > 0) {
        if (PACK) {
          ptx::bulk_s2g(reinterpret_cast<void*>(s_dst[st]), sm.out[ob], (uint32_t)elems);
          ptx::bulk_s2g(reinterpret_cast<void*>(s_dst2[st]), sm.out_scales[ob], (uint32_t)groups * 4);
        } else {
          ptx::bulk_s2g(reinterpret_cast<void*>(s_dst[st]), sm.out[ob], (uint32_t)elems * 2);
        }
      }
      ptx::bulk_commit();
    }
  }
  if (tid == 0) {
    ptx::bulk_wait<0>();
    if (s_abort) err |= KV_ERR_WAIT_EXPIRED;
    if (err && p.status)
      for (int b = 0; b < kStatusWords; ++b)
        if (err & (1 << b)) reinterpret_cast<volatile int32_t*>(p.status)[b] = 1;
  }
}

template <bool PACK, int T>
constexpr int pipe_smem() { return (int)sizeof(Smem<PACK, T>) * Pipe<T>::kGroups; }

template <bool PACK, int T>
cudaError_t load_pipe() {
  return cudaFuncSetAttribute(kv_quant_fp8_kernel<PACK, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              pipe_smem<PACK, T>());
}

template <bool PACK, int T>
cudaError_t launch_pipe(const KvCopyParams& p, int num_ctas, cudaStream_t stream) {
  const cudaError_t e = load_pipe<PACK, T>();
  if (e != cudaSuccess) return e;
  const int tiles_per_chunk = (int)((p.chunk_bytes / 2 + Pipe<T>::kTileElems - 1) / Pipe<T>::kTileElems);
  const int64_t total = (int64_t)p.num_pairs * p.num_layers * p.kv_dim * tiles_per_chunk;
  const int64_t need = (total + Pipe<T>::kGroups - 1) / Pipe<T>::kGroups;
  const int64_t ctas = num_ctas > 0 ? num_ctas : 32;
  kv_quant_fp8_kernel<PACK, T><<<(unsigned)(ctas < need ? ctas : need), kCtaThreads, pipe_smem<PACK, T>(), stream>>>(
      p, tiles_per_chunk);
  return cudaGetLastError();
}

}  // namespace

cudaError_t kv_quant_load_kernels() {
  cudaError_t e = load_pipe<false, 256>();
  if (e == cudaSuccess) e = load_pipe<true, 256>();
  if (e == cudaSuccess) e = load_pipe<false, 128>();
  if (e == cudaSuccess) e = load_pipe<true, 128>();
  if (e == cudaSuccess) e = load_pipe<false, 64>();
  if (e == cudaSuccess) e = load_pipe<true, 64>();
  return e;
}

cudaError_t launch_kv_quant_fp8(const KvCopyParams& p, int num_ctas, cudaStream_t stream) {
  if (p.num_pairs <= 0 || p.num_layers <= 0 || p.kv_dim <= 0 || p.chunk_bytes <= 0) return cudaSuccess;
  const int64_t chunk_elems = p.chunk_bytes / 2;
  if ((p.chunk_bytes & 1) || chunk_elems % 512 != 0 || !kv_copy_tma_eligible(p)) return cudaErrorInvalidValue;
  if (chunk_elems <= Pipe<64>::kTileElems)
    return p.h2d ? launch_pipe<false, 64>(p, num_ctas, stream) : launch_pipe<true, 64>(p, num_ctas, stream);
  if (chunk_elems <= Pipe<128>::kTileElems)
    return p.h2d ? launch_pipe<false, 128>(p, num_ctas, stream) : launch_pipe<true, 128>(p, num_ctas, stream);
  return p.h2d ? launch_pipe<false, 256>(p, num_ctas, stream) : launch_pipe<true, 256>(p, num_ctas, stream);
}

}  // namespace fkv
