// Copy-engine path for GPU<->host block moves.
//
// The DMA engines move long contiguous spans a few percent faster than SM-issued
// traffic on PCIe (no SM time at all), but cost one driver call per span. An op is
// therefore analysed into maximal runs of consecutive (gpu, cpu) block-id pairs and
// routed: whole-run single copies when the block is laid out identically on both
// sides, one pitched 2-D copy per (run, layer, kv) when only the chunk is contiguous,
// and the persistent TMA kernel when the runs are too short to amortise the calls.
// Same role as the reference's adaptive copy-engine dispatcher (csrc/ce_transfer.cu:37-104,
// path list csrc/ce_transfer.h:42-49). A fourth route covers the common case of scattered GPU pages whose
// host blocks were allocated in a row (a fresh pool, or blocks recycled sequence by sequence): the copy
// kernel gathers the pages into a double-buffered device staging area in host block format, at HBM speed, and
// the DMA engine moves each staged piece to the contiguous host span with one large copy (and the reverse for
// restores), the reference's GATHER_DIRECT idea (csrc/ce_transfer.cu:643-812). Host blocks that are scattered
// too stay on the kernel: per-block driver copies of 2 MiB reach 50.6 / 49.5 GB/s on B200 with any number of
// streams, below the kernel's 52.8 / 51.5, and a host-side scatter would spend CPU cores and memory bandwidth.
#pragma once
#include <cstdint>
#include <functional>
#include <vector>

#include <cuda_runtime.h>

#include "kernels/kv_copy.h"

namespace fkv {

struct CeRun {
  int64_t gpu_block, cpu_block, len;
};

struct CeAnalysis {
  std::vector<CeRun> runs;
  int64_t num_blocks = 0;
  int64_t longest = 0;
  int status = 0;  // KvCopyStatus range bits for ids that were dropped
};

enum class CePath : int {
  KERNEL = 0,        // leave the op to the copy kernel
  CONTIG_BLOCKS = 1, // one cudaMemcpyAsync per run (identical block geometry on both sides)
  SEGMENT_2D = 2,    // one cudaMemcpy2DAsync per (run, layer, kv)
  GATHER_STAGED = 3, // kernel gather into device staging + one large copy per piece of a host run
};

struct CePolicy {
  int64_t max_copies = 4096;         // driver calls per op above which the kernel wins
  // measured on B200 (2 MiB blocks, 32 KiB chunks): 16 MiB per driver copy gives 54.6 GB/s against the
  // kernel's 52.0; 2 MiB per copy gives 50.5, below the kernel
  int64_t min_bytes_per_copy = 8 << 20;
};

// `gpu_blocks`/`cpu_blocks` must be host-readable. Out-of-range ids are skipped and
// recorded in `status`.
CeAnalysis ce_analyze(const int64_t* gpu_blocks, const int64_t* cpu_blocks, int64_t n, int64_t gpu_num_blocks,
                      int64_t cpu_num_blocks);
CePath ce_choose(const CeAnalysis& a, const KvCopyParams& p, const CePolicy& pol);
int64_t ce_num_copies(const CeAnalysis& a, const KvCopyParams& p, CePath path);
// Issues the copies on `stream`; returns the first CUDA error.
cudaError_t ce_copy(const KvCopyParams& p, const CeAnalysis& a, CePath path, cudaStream_t stream);

// ---- staged route -------------------------------------------------------------------------------------------
// A run of consecutive host blocks over consecutive pairs of the op.
struct CeHostRun {
  int64_t first;      // index of the run's first pair in the op's id arrays
  int64_t cpu_block;  // its first host block
  int64_t len;
};

// How an op is split: pairs [0, staged) cross the link in pieces, one large copy each; the others, whose host
// blocks stand alone, stay with the kernel.
struct CeStagePlan {
  std::vector<CeHostRun> pieces;   // in the order they are moved; none longer than a staging buffer
  int64_t staged = 0;
};

constexpr int kCeStageBufs = 2;
// Bytes of one staging buffer unless a caller asks for a number of blocks. B200, contiguous copies back to back,
// GB/s GPU->host / host->GPU: pieces of 4 MiB 54.1 / 52.5, 16 MiB 56.2 / 54.8, 64 MiB 56.6 / 55.4, one of 1 GiB
// 57.0 / 55.6.
constexpr int64_t kCeStageBytes = 32 << 20;
// An op moves kernel-first until its first piece is gathered (and kernel-last for a restore), so that piece is small
// and the following ones double.
constexpr int64_t kCeRampBytes = 4 << 20;
// Bytes that the runs must hold before an op is split between copy engine and kernel: about 8 % of their time is
// won, and the second launch and the events cost some 20 us.
constexpr int64_t kCeMixedMinBytes = 32 << 20;

// Device staging of one GPU (owned by the caller's per-rank state, freed by ce_staging_free).
struct CeStaging {
  uint8_t* buf[kCeStageBufs] = {};
  int64_t* iota = nullptr;            // device array 0, 1, 2, ...: the staged block ids
  cudaEvent_t kernel_done[kCeStageBufs] = {}, copy_done[kCeStageBufs] = {};
  cudaStream_t copy_stream = nullptr;
  int64_t blocks = 0, block_bytes = 0;
  bool used[kCeStageBufs] = {};
  bool refused = false;               // there was no memory for it: not asked for again
};
// Makes room for `blocks` blocks per buffer (0: kCeStageBytes' worth) on the current device. False when the
// device has no memory for it; the op then stays with the kernel.
bool ce_staging_prepare(CeStaging& st, int64_t blocks, int64_t block_bytes);
void ce_staging_free(CeStaging& st);

// True when the host side of `p` is whole blocks of [layer][kv][chunk_slot] that abut, so that consecutive block ids
// are one span of memory.
bool ce_host_blocks_abut(const KvCopyParams& p, int total_layers, int64_t chunk_slot);

// Plans the staged route for an op whose host blocks abut. Runs of at least `min_run` consecutive host blocks become
// pieces of at most `max_piece` blocks; where they leave other pairs over, the id arrays are REORDERED in place (runs
// first) and the op is only split when the runs hold at least kCeMixedMinBytes. False, with the arrays as they were,
// when the op belongs to the kernel: an id out of range, no run long enough.
bool ce_plan_staged(const KvCopyParams& p, int64_t* gpu_blocks, int64_t* cpu_blocks, int64_t min_run,
                    int64_t max_piece, CeStagePlan& plan, int64_t ramp_bytes = kCeRampBytes);

// Launches the kernel of a piece or of the pairs that stay with it. For a piece, `q` addresses the staging buffer as
// the host side (block ids 0, 1, ...) and `host_block` is the host block that id 0 stands for; otherwise it is 0.
using CeStageKernel = std::function<cudaError_t(const KvCopyParams& q, int64_t host_block, cudaStream_t stream)>;
// Moves a staged piece to or from the host where that is not one contiguous copy of its blocks. `worth` is asked
// before anything is queued for the piece; a piece that it declines is left to the kernel.
struct CeLinkCopy {
  std::function<bool(const CeHostRun& piece)> worth;
  std::function<cudaError_t(const CeHostRun& piece, uint8_t* staged, cudaStream_t stream)> copy;
};
// Moves the op: pieces through the staging buffers, gather or scatter kernel on `stream`, large copies on the
// staging's own stream, both buffers in flight; the other pairs by the kernel, on `stream`, beside the last copies
// (offload) or the first ones (restore). When it returns, everything has been queued and `stream` waits for the last
// copy; when it fails, part of the op may have been moved and nothing of it is in flight any more. `p` carries the id
// arrays as planned.
cudaError_t ce_copy_staged(const KvCopyParams& p, const CeStagePlan& plan, CeStaging& st, const CeStageKernel& kernel,
                           cudaStream_t stream, const CeLinkCopy* link = nullptr);

}  // namespace fkv
