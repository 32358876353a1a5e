// Paged KV gather/scatter kernels (see kv_copy.h for the addressing model).
//
// Engine 0 — bulk-copy pipeline. A persistent CTA runs W independent one-warp pipelines, each with its own ring
// of shared-memory stages driven through the TMA unit: lane 0 issues a 1-D bulk load (global -> shared,
// completion on an mbarrier) for tiles up to LOOKAHEAD ahead, and as each tile lands issues the matching bulk
// store (shared -> global). Either side may be mapped host memory, so the same pipeline does GPU->host and
// host->GPU with no SM load/store instructions on the data and no registers holding payload. The addresses of
// the next 32 tiles are computed by the 32 lanes at once and handed to lane 0 through shared memory.
//
// What bounds it: against the host, the link, from two to four CTAs on; between two places in HBM, the bytes a CTA
// can keep in flight (192 KiB, about 48 GB/s per CTA). Before, one warp per CTA computed the addresses tile by tile
// and took 0.8 us per tile whatever its size. Measured on B200, GB/s before -> now, 8 CTAs:
//   4 KiB chunks GPU->host 40 -> 52.5, host->GPU 41 -> 51.3 (16 CTAs 52.4 -> 52.5 / 39 -> 51.3); 1 KiB 10 -> 52.5
//   within HBM: 4 KiB chunks 40 -> 378, 32 KiB 160 -> 391; 64 CTAs 300 -> 2470 and 1180 -> 2570
//   one op of 2 MiB in 32 KiB chunks: GPU->host 54 -> 50 us
//
// Engine 1 — SIMT vector copy, warp per tile, 16/8/4/1-byte lanes with an
// 8-deep unrolled load batch. It serves chunks whose size or alignment rules
// out 16-byte bulk copies (the reference needs an 8-byte path for the same
// reason: csrc/transfer.cu:34-92) and is the cross-check for engine 0.
#include "kv_copy.h"
#include "kv_signal.cuh"
#include "ptx_sm100.cuh"

namespace fkv {
namespace {

constexpr uint64_t kWaitBudgetNs = 2000000000ull;  // 2 s per bulk-copy wait
constexpr uint64_t kSignalBudgetNs = 60000000000ull;  // signaller warp: longer than any restore, still finite

struct TileAddr {
  uint64_t gpu;
  uint64_t cpu;
  uint32_t bytes;  // 0 = skip (bad block id)
};

// Position of a tile inside the launch. Tiles are enumerated pair-major
// (pair, layer, kv, sub-tile: one host block's bytes are visited contiguously)
// or, for per-layer signalling, layer-major (layer, pair, kv, sub-tile).
struct TilePos {
  int32_t pair, layer, kv, s;
};

__device__ __forceinline__ TilePos decode_tile(const KvCopyParams& p, int32_t major, int32_t r, int tiles_per_chunk) {
  TilePos t;
  t.s = r % tiles_per_chunk;
  const int32_t q = r / tiles_per_chunk;
  if (p.layer_major) {
    t.layer = p.layer_start + major;
    t.kv = q % p.kv_dim;
    t.pair = q / p.kv_dim;
  } else {
    t.pair = major;
    t.kv = q % p.kv_dim;
    t.layer = p.layer_start + q / p.kv_dim;
  }
  return t;
}

__device__ __forceinline__ TileAddr tile_addr(const KvCopyParams& p, const TilePos& t, int64_t gblk, int64_t cblk,
                                              int tile_bytes) {
  TileAddr a;
  const int64_t off = (int64_t)t.s * tile_bytes;
  const int64_t left = p.chunk_bytes - off;
  a.bytes = (uint32_t)(left < tile_bytes ? left : tile_bytes);
  a.gpu = kv_gpu_tensor(p, t.layer * p.idx_layer_mul + t.kv * p.idx_kv_mul) + t.layer * p.g_layer_stride +
          t.kv * p.g_kv_stride + gblk * p.g_block_stride + p.g_off + off;
  const uint64_t cbase = p.c_use_table ? kv_c_tensor(p, t.layer * p.c_idx_layer_mul + t.kv * p.c_idx_kv_mul) : p.cpu_base;
  a.cpu = cbase + t.layer * p.c_layer_stride + t.kv * p.c_kv_stride + cblk * p.c_block_stride + p.c_off + off;
  return a;
}

__device__ __forceinline__ bool ids_in_range(const KvCopyParams& p, int64_t g, int64_t c, int& err) {
  bool ok = true;
  if (p.gpu_num_blocks > 0 && (g < 0 || g >= p.gpu_num_blocks)) { err |= KV_ERR_GPU_BLOCK_RANGE; ok = false; }
  if (p.cpu_num_blocks > 0 && (c < 0 || c >= p.cpu_num_blocks)) { err |= KV_ERR_CPU_BLOCK_RANGE; ok = false; }
  return ok;
}

// Descriptors of the tiles a pipeline is working on: written by all lanes 32 tiles at a time, read by lane 0, which is
// done with a batch LOOKAHEAD tiles into the next one. What is overwritten is four batches old, so two warp barriers
// (one follows the writes of every batch) lie between its last read and the write. With room for two batches a
// barrier of its own would be needed at the end of each; it cost a tenth of the time of 4 KiB chunks within HBM
// (340 -> 374 us for 187 blocks of an 80-layer, one-head cache, 8 CTAs of a B200).
constexpr int kDescRing = 128;
struct TileDesc {
  uint64_t src, dst;
  uint32_t bytes;   // 0 = skipped
  int32_t major;    // layer-major launches: layer (relative) of the tile
};

// Layer-major launches run one more warp per CTA whose only job is the per-layer publication: fences, the
// counter atomic and the system-scope flag store issued by a copy warp itself would wait for that warp's loads
// in flight and drain the pipeline at every layer boundary. The copy warps only wait for their bulk stores and
// post "layers [0, n) done" to a shared-memory mailbox each; the CTA has finished what all of them have.
template <int W, int STAGES, int LOOKAHEAD>
__global__ void __launch_bounds__(32 * (W + 1), 1)
kv_copy_bulk_kernel(const __grid_constant__ KvCopyParams p, int tile_bytes, int tiles_per_chunk) {
  static_assert(LOOKAHEAD >= 1 && LOOKAHEAD < STAGES, "lookahead must leave one stage for stores");
  static_assert(STAGES <= 32, "stage phases are kept in one 32-bit mask");
  static_assert(LOOKAHEAD <= 32 && kDescRing >= 96, "a barrier between the last read of a descriptor and the next write");
  extern __shared__ __align__(128) uint8_t ring_all[];
  __shared__ __align__(8) uint64_t full_all[W][STAGES];
  __shared__ TileDesc desc_all[W][kDescRing];
  __shared__ int s_layers_done[W];      // mailboxes: this warp finished (stores included) layers [0, n)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    for (int w = 0; w < W; ++w) {
#pragma unroll
      for (int s = 0; s < STAGES; ++s) ptx::mbar_init(&full_all[w][s], 1);
      s_layers_done[w] = 0;
    }
    ptx::fence_mbar_init();
  }
  __syncthreads();
  const bool signalling = p.layer_major && p.done_counter != nullptr;
  if (warp == W) {
    // ---- signaller warp (present only on layer-major launches with signalling)
    if (lane != 0 || !signalling) return;
    int sig = 0;
    const uint64_t t0 = ptx::globaltimer_ns();
    while (sig < p.num_layers) {
      int d = p.num_layers;
#pragma unroll
      for (int w = 0; w < W; ++w) d = min(d, *reinterpret_cast<volatile int*>(&s_layers_done[w]));
      if (d > sig) {
        __threadfence_block();            // acquire side of the mailboxes
        signal_layers(p, sig, d);
        sig = d;
      } else {
        if (ptx::globaltimer_ns() - t0 > kSignalBudgetNs) {   // the copy warps always post the last layer; belt and braces
          if (p.status) report_status(p.status, KV_ERR_WAIT_EXPIRED);
          return;
        }
        __nanosleep(64);
      }
    }
    return;
  }
  uint8_t* const ring = ring_all + (size_t)warp * STAGES * tile_bytes;
  uint64_t* const full = full_all[warp];
  TileDesc* const desc = desc_all[warp];

  // span = tiles per major unit (a pair, or a layer when layer-major); counts per pipeline fit 32 bits
  const int32_t n_major = p.layer_major ? p.num_layers : p.num_pairs;
  const int32_t span = (p.layer_major ? p.num_pairs : p.num_layers) * p.kv_dim * tiles_per_chunk;
  const int64_t total = (int64_t)span * n_major;
  // consecutive tiles go to different CTAs first, so that a small op uses all of them
  const int64_t first = (int64_t)warp * gridDim.x + blockIdx.x, step = (int64_t)gridDim.x * W;
  const int32_t n_mine = first < total ? (int32_t)((total - first + step - 1) / step) : 0;
  // this lane decodes tiles lane, lane + 32, ... of the pipeline; (major, r) advances without divisions
  const int64_t step32 = step * 32;
  const int32_t step_q = (int32_t)(step32 / span), step_r = (int32_t)(step32 % span);
  const int64_t t_lane = first + lane * step;
  int32_t major = (int32_t)(t_lane / span), r = (int32_t)(t_lane % span);
  TilePos pos{0, 0, 0, 0};
  int64_t gblk = 0, cblk = 0;
  // block ids may live in host memory: those of the next batch are requested while this one is being moved
  auto fetch = [&](int32_t idx) {
    if (idx >= n_mine) return;
    pos = decode_tile(p, major, r, tiles_per_chunk);
    gblk = __ldg(p.gpu_blocks + pos.pair);
    cblk = __ldg(p.cpu_blocks + pos.pair);
  };
  fetch(lane);

  int err = 0;
  int dead = 0;          // set after an expired wait: stop issuing, drain, leave
  uint32_t phases = 0;   // lane 0: parity of the next completion of each stage's barrier
  int ld_st = 0, st_st = 0;   // lane 0: stage of the next load / of the next store
  int32_t signalled = 0; // lane 0, layer-major: layers [0, signalled) already posted by this warp

  const int32_t n_steps = n_mine > 0 ? n_mine + LOOKAHEAD : 0;
  for (int32_t base = 0; base < n_steps; base += 32) {
    if (base + lane < n_mine) {
      TileDesc d{0, 0, 0, major};
      if (ids_in_range(p, gblk, cblk, err)) {
        const TileAddr a = tile_addr(p, pos, gblk, cblk, tile_bytes);
        d.src = p.h2d ? a.cpu : a.gpu;
        d.dst = p.h2d ? a.gpu : a.cpu;
        d.bytes = a.bytes;
      }
      desc[(base + lane) & (kDescRing - 1)] = d;
      major += step_q;
      r += step_r;
      if (r >= span) { r -= span; ++major; }
      fetch(base + 32 + lane);
    }
    __syncwarp();
    if (lane == 0) {
      const int32_t end = min(base + 32, n_steps);
      for (int32_t it = base; it < end; ++it) {
        const int32_t j = it - LOOKAHEAD;
        if (j >= 0) {
          const TileDesc& d = desc[j & (kDescRing - 1)];
          if (signalling && d.major > signalled) {
            // first store of a later layer: everything this warp owned in the earlier layers is committed;
            // drain those stores (the loads in flight are unaffected) and post the layers
            ptx::bulk_wait<0>();
            __threadfence_block();
            *reinterpret_cast<volatile int*>(&s_layers_done[warp]) = d.major;
            signalled = d.major;
          }
          if (d.bytes) {
            if (!ptx::mbar_wait_bounded(&full[st_st], (phases >> st_st) & 1u, kWaitBudgetNs)) {
              dead = 1;
              break;
            }
            phases ^= 1u << st_st;
            ptx::bulk_s2g(reinterpret_cast<void*>(d.dst), ring + (size_t)st_st * tile_bytes, d.bytes);
          }
          ptx::bulk_commit();  // one group per tile (possibly empty) keeps the wait arithmetic uniform
          if (++st_st == STAGES) st_st = 0;
        }
        if (it < n_mine) {
          const TileDesc& d = desc[it & (kDescRing - 1)];
          // the stage was last used by tile it-STAGES; all but the newest
          // STAGES-LOOKAHEAD store groups must have finished reading smem
          if (it >= STAGES) ptx::bulk_wait_read<STAGES - LOOKAHEAD>();
          if (d.bytes) {
            ptx::mbar_expect_tx(&full[ld_st], d.bytes);
            ptx::bulk_g2s(ring + (size_t)ld_st * tile_bytes, reinterpret_cast<const void*>(d.src), d.bytes,
                          &full[ld_st]);
          }
          if (++ld_st == STAGES) ld_st = 0;
        }
      }
    }
    dead = __shfl_sync(0xffffffffu, dead, 0);
    if (dead) break;
  }
  err = (int)__reduce_or_sync(0xffffffffu, (unsigned)err);
  if (lane == 0) {
    if (dead) err |= KV_ERR_WAIT_EXPIRED;
    ptx::bulk_wait<0>();
    if (err && p.status) report_status(p.status, err);
    if (p.layer_major) {
      __threadfence_block();
      *reinterpret_cast<volatile int*>(&s_layers_done[warp]) = p.num_layers;   // every exit path ends here
    } else {
      signal_done(p, gridDim.x * W);
    }
  }
}

// ---------------------------------------------------------------- SIMT engine

template <typename V> struct VecIO;
template <> struct VecIO<uint4> {
  static __device__ __forceinline__ uint4 ld(const void* p) { return ptx::ld_nc_v4(p); }
  static __device__ __forceinline__ void st(void* p, const uint4& v) { ptx::st_cg_v4(p, v); }
};
template <> struct VecIO<uint2> {
  static __device__ __forceinline__ uint2 ld(const void* p) { return ptx::ld_nc_v2(p); }
  static __device__ __forceinline__ void st(void* p, const uint2& v) { ptx::st_cg_v2(p, v); }
};
template <> struct VecIO<uint32_t> {
  static __device__ __forceinline__ uint32_t ld(const void* p) { return ptx::ld_nc_u32(p); }
  static __device__ __forceinline__ void st(void* p, const uint32_t& v) { ptx::st_cg_u32(p, v); }
};
template <> struct VecIO<uint8_t> {
  static __device__ __forceinline__ uint8_t ld(const void* p) { return *reinterpret_cast<const volatile uint8_t*>(p); }
  static __device__ __forceinline__ void st(void* p, const uint8_t& v) { *reinterpret_cast<volatile uint8_t*>(p) = v; }
};

template <typename V>
__global__ void __launch_bounds__(512)
kv_copy_simt_kernel(const __grid_constant__ KvCopyParams p, int tile_bytes, int tiles_per_chunk) {
  constexpr int UNROLL = 8;
  const int lane = threadIdx.x & 31;
  const int warps_per_cta = blockDim.x >> 5;
  const int64_t warp0 = (int64_t)blockIdx.x * warps_per_cta + (threadIdx.x >> 5);
  const int64_t nwarps = (int64_t)gridDim.x * warps_per_cta;
  const int32_t n_major = p.layer_major ? p.num_layers : p.num_pairs;
  const int32_t span = (p.layer_major ? p.num_pairs : p.num_layers) * p.kv_dim * tiles_per_chunk;
  const int64_t total = (int64_t)span * n_major;
  int err = 0;
  for (int64_t t = warp0; t < total; t += nwarps) {
    const TilePos pos = decode_tile(p, (int32_t)(t / span), (int32_t)(t % span), tiles_per_chunk);
    const int64_t gblk = __ldg(p.gpu_blocks + pos.pair);
    const int64_t cblk = __ldg(p.cpu_blocks + pos.pair);
    if (!ids_in_range(p, gblk, cblk, err)) continue;
    const TileAddr a = tile_addr(p, pos, gblk, cblk, tile_bytes);
    const uint8_t* src = reinterpret_cast<const uint8_t*>(p.h2d ? a.cpu : a.gpu);
    uint8_t* dst = reinterpret_cast<uint8_t*>(p.h2d ? a.gpu : a.cpu);
    const int nvec = (int)(a.bytes / sizeof(V));
    int i = lane;
    for (; i + 32 * (UNROLL - 1) < nvec; i += 32 * UNROLL) {
      V v[UNROLL];
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) v[u] = VecIO<V>::ld(src + (size_t)(i + 32 * u) * sizeof(V));
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) VecIO<V>::st(dst + (size_t)(i + 32 * u) * sizeof(V), v[u]);
    }
    for (; i < nvec; i += 32) VecIO<V>::st(dst + (size_t)i * sizeof(V), VecIO<V>::ld(src + (size_t)i * sizeof(V)));
  }
  if (err && p.status && lane == 0) report_status(p.status, err);
  if (p.done_counter) {
    __syncthreads();
    if (threadIdx.x == 0) signal_done(p);
  }
}

// ---------------------------------------------------------------- baseline shape
// One warp per (layer, pair); inside, a loop over kv planes with 16-byte lanes.
__global__ void __launch_bounds__(1024) kv_copy_refshape_kernel(const __grid_constant__ KvCopyParams p) {
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const int64_t total = (int64_t)p.num_layers * p.num_pairs;
  const int nvec = (int)(p.chunk_bytes / 16);
  for (int64_t w = warp0; w < total; w += nwarps) {
    const int layer = p.layer_start + (int)(w / p.num_pairs);
    const int64_t pair = w % p.num_pairs;
    const int64_t gblk = p.gpu_blocks[pair];
    const int64_t cblk = p.cpu_blocks[pair];
    for (int kv = 0; kv < p.kv_dim; ++kv) {
      const uint64_t g = kv_gpu_tensor(p, layer * p.idx_layer_mul + kv * p.idx_kv_mul) + layer * p.g_layer_stride +
                         kv * p.g_kv_stride + gblk * p.g_block_stride + p.g_off;
      const uint64_t c =
          p.cpu_base + layer * p.c_layer_stride + kv * p.c_kv_stride + cblk * p.c_block_stride + p.c_off;
      const uint8_t* src = reinterpret_cast<const uint8_t*>(p.h2d ? c : g);
      uint8_t* dst = reinterpret_cast<uint8_t*>(p.h2d ? g : c);
      for (int i = lane; i < nvec; i += 32) ptx::st_cg_v4(dst + (size_t)i * 16, ptx::ld_nc_v4(src + (size_t)i * 16));
    }
  }
}

// Dynamic shared memory that every instance may ask for: its rings at the largest tile it serves. One figure for
// all, so that threads launching ops of different tile sizes cannot lower it under one another.
constexpr int kRingBytes = 192 << 10;

template <int W, int STAGES, int LA>
cudaError_t load_bulk() {
  // idempotent and cheap; avoids per-device bookkeeping
  return cudaFuncSetAttribute(kv_copy_bulk_kernel<W, STAGES, LA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              kRingBytes);
}

template <int W, int STAGES, int LA>
cudaError_t launch_bulk(const KvCopyParams& p, int ctas, int tile_bytes, int tiles_per_chunk, cudaStream_t s) {
  cudaError_t e = load_bulk<W, STAGES, LA>();
  if (e != cudaSuccess) return e;
  const int warps = W + (p.layer_major && p.done_counter != nullptr ? 1 : 0);   // last warp = layer signaller
  kv_copy_bulk_kernel<W, STAGES, LA><<<ctas, 32 * warps, W * STAGES * tile_bytes, s>>>(p, tile_bytes, tiles_per_chunk);
  return cudaGetLastError();
}

inline bool all_multiple(const KvCopyParams& p, int64_t m) {
  auto ok = [m](int64_t v) { return (v % m) == 0; };
  bool r = ok(p.chunk_bytes) && ok(p.g_layer_stride) && ok(p.g_kv_stride) && ok(p.g_block_stride) && ok(p.g_off) &&
           ok((int64_t)(p.cpu_base % (uint64_t)m)) && ok(p.c_layer_stride) && ok(p.c_kv_stride) &&
           ok(p.c_block_stride) && ok(p.c_off);
  const int nptr = p.idx_layer_mul == 0 && p.idx_kv_mul == 0
                       ? 1
                       : (p.layer_start + p.num_layers - 1) * p.idx_layer_mul + (p.kv_dim - 1) * p.idx_kv_mul + 1;
  for (int i = 0; i < nptr && i < p.num_gpu_ptrs; ++i) r = r && (kv_gpu_tensor(p, i) % (uint64_t)m) == 0;
  if (p.c_use_table) {
    const int nc = p.c_idx_layer_mul == 0 && p.c_idx_kv_mul == 0
                       ? 1
                       : (p.layer_start + p.num_layers - 1) * p.c_idx_layer_mul + (p.kv_dim - 1) * p.c_idx_kv_mul + 1;
    for (int i = 0; i < nc && i < p.num_c_ptrs; ++i) r = r && (kv_c_tensor(p, i) % (uint64_t)m) == 0;
  }
  return r;
}

}  // namespace

cudaError_t kv_copy_load_kernels() {
  cudaError_t e = load_bulk<4, 12, 11>();
  if (e == cudaSuccess) e = load_bulk<4, 12, 6>();
  if (e == cudaSuccess) e = load_bulk<4, 6, 5>();
  if (e == cudaSuccess) e = load_bulk<4, 6, 3>();
  if (e == cudaSuccess) e = load_bulk<4, 3, 2>();
  if (e == cudaSuccess) e = load_bulk<2, 3, 2>();
  return e;
}

bool kv_copy_tma_eligible(const KvCopyParams& p) { return kv_copy_tables_ok(p) && all_multiple(p, 16); }

cudaError_t launch_kv_copy(const KvCopyParams& p, const KvCopyLaunch& cfg, cudaStream_t stream) {
  if (p.num_pairs <= 0 || p.num_layers <= 0 || p.kv_dim <= 0 || p.chunk_bytes <= 0) return cudaSuccess;
  if (!kv_copy_tables_ok(p)) return cudaErrorInvalidValue;
  int tile = cfg.tile_bytes > 0 ? cfg.tile_bytes : 16384;
  int engine = cfg.engine;
  if (engine == 0 && !all_multiple(p, 16)) engine = 1;
  if (engine == 0) {
    tile = (tile / 16) * 16;
    if (tile < 1024) tile = 1024;
    if (tile > 32768) tile = 32768;
    if ((int64_t)tile > p.chunk_bytes) tile = (int)p.chunk_bytes;
    const int tiles_per_chunk = (int)((p.chunk_bytes + tile - 1) / tile);
    const int64_t total = (int64_t)p.num_pairs * p.num_layers * p.kv_dim * tiles_per_chunk;
    int ctas = cfg.num_ctas > 0 ? cfg.num_ctas : 16;
    if ((int64_t)ctas > total) ctas = (int)total;
    // Pipelines per CTA and the depth of their rings: together they hold at most 192 KiB of the 227 KiB a CTA may
    // have, whatever the tile. Host reads need bytes in flight to cover the PCIe round trip, so host->GPU keeps
    // every stage but one loading; GPU->host leaves half of a deep ring to queued posted writes.
    if (p.h2d) {
      if (tile <= 4096) return launch_bulk<4, 12, 11>(p, ctas, tile, tiles_per_chunk, stream);
      if (tile <= 8192) return launch_bulk<4, 6, 5>(p, ctas, tile, tiles_per_chunk, stream);
      if (tile <= 16384) return launch_bulk<4, 3, 2>(p, ctas, tile, tiles_per_chunk, stream);
      return launch_bulk<2, 3, 2>(p, ctas, tile, tiles_per_chunk, stream);
    }
    if (tile <= 4096) return launch_bulk<4, 12, 6>(p, ctas, tile, tiles_per_chunk, stream);
    if (tile <= 8192) return launch_bulk<4, 6, 3>(p, ctas, tile, tiles_per_chunk, stream);
    if (tile <= 16384) return launch_bulk<4, 3, 2>(p, ctas, tile, tiles_per_chunk, stream);
    return launch_bulk<2, 3, 2>(p, ctas, tile, tiles_per_chunk, stream);
  }
  // SIMT engine
  if (tile > p.chunk_bytes) tile = (int)p.chunk_bytes;
  int vec = all_multiple(p, 16) ? 16 : all_multiple(p, 8) ? 8 : all_multiple(p, 4) ? 4 : 1;
  tile = (tile / vec) * vec;
  if (tile <= 0) tile = vec;
  const int tiles_per_chunk = (int)((p.chunk_bytes + tile - 1) / tile);
  const int64_t total = (int64_t)p.num_pairs * p.num_layers * p.kv_dim * tiles_per_chunk;
  int ctas = cfg.num_ctas > 0 ? cfg.num_ctas : 16;
  const int64_t need = (total + 15) / 16;
  if ((int64_t)ctas > need) ctas = (int)need;
  switch (vec) {
    case 16: kv_copy_simt_kernel<uint4><<<ctas, 512, 0, stream>>>(p, tile, tiles_per_chunk); break;
    case 8: kv_copy_simt_kernel<uint2><<<ctas, 512, 0, stream>>>(p, tile, tiles_per_chunk); break;
    case 4: kv_copy_simt_kernel<uint32_t><<<ctas, 512, 0, stream>>>(p, tile, tiles_per_chunk); break;
    default: kv_copy_simt_kernel<uint8_t><<<ctas, 512, 0, stream>>>(p, tile, tiles_per_chunk); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_kv_copy_refshape(const KvCopyParams& p, int num_ctas, cudaStream_t stream) {
  if (p.num_pairs <= 0 || p.num_layers <= 0) return cudaSuccess;
  if (!kv_copy_tables_ok(p) || !all_multiple(p, 16)) return cudaErrorInvalidValue;
  kv_copy_refshape_kernel<<<num_ctas > 0 ? num_ctas : 4, 1024, 0, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace fkv
