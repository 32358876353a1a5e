#include "kv_hash.h"

namespace fkv {
namespace {

constexpr uint64_t P1 = 0x9E3779B185EBCA87ULL;
constexpr uint64_t P2 = 0xC2B2AE3D27D4EB4FULL;
constexpr uint64_t P3 = 0x165667B19E3779F9ULL;
constexpr uint64_t P4 = 0x85EBCA77C2B2AE63ULL;
constexpr uint64_t P5 = 0x27D4EB2F165667C5ULL;

__device__ __forceinline__ uint64_t rotl(uint64_t x, int r) { return (x << r) | (x >> (64 - r)); }
__device__ __forceinline__ uint64_t xround(uint64_t acc, uint64_t in) { return rotl(acc + in * P2, 31) * P1; }
__device__ __forceinline__ uint64_t xmerge(uint64_t h, uint64_t v) { return (h ^ xround(0, v)) * P1 + P4; }
__device__ __forceinline__ uint64_t avalanche(uint64_t h) {
  h ^= h >> 33; h *= P2; h ^= h >> 29; h *= P3; h ^= h >> 32;
  return h;
}

// The input of a sequence is a stream of 64-bit words w[0], w[1], ... (namespace prefix, then tokens). XXH64
// consumes it in stripes of four words; word k of a stripe feeds accumulator k. A digest after `n` words: the n/4
// complete stripes are in the accumulators, the last n%4 words are the "tail" and are folded in sequentially.
//
// What bounds it: acc = rotl(acc + w*P2, 31) * P1 cannot be reassociated, so a sequence is one chain of
// (words / 4) dependent rounds whatever the width of the machine. Everything else is taken off that chain: warp 0
// of a CTA does nothing but the chain (one lane per accumulator), reading ready-made w*P2 from shared memory and
// leaving the accumulators after every stripe there; the other warps fetch and multiply the next segment and turn
// the accumulators of the previous one into digests. Segments are double-buffered, one barrier each.
// Measured on B200 with the Python wrapper, before (four lanes did fetch, chain and digests in turn, inputs were
// concatenated and three offset tables uploaded) -> now: 64 x 4096 tokens, 16 per block, GPU 351 -> 30 us, whole
// call 343 -> 63 us; one 32K prompt 1764 -> 181 us; 64 x 4096 with one token per block 2710 -> 89 us; 8192 x 1024
// tokens (flat form, eight sequences per CTA) 20.6 -> 14.6 ms, most of it concatenation.
constexpr int kHashThreads = 128;
constexpr int kHashHelpers = kHashThreads - 32;
constexpr int kSegStripes = 256;      // stripes per segment and CTA, over its G sequences: 2 x 8 KiB in, 2 x 8 KiB out

struct HashParams {
  // exactly one of the two forms: `offsets` set = flat arrays, null = the list below
  const int64_t* tokens;
  const int64_t* offsets;
  const int64_t* out_offsets;
  const int64_t* ns;                  // prefix values in memory; null = ns8
  uint64_t* out;
  int64_t num_seqs;
  int64_t ns_len;
  int32_t tpb;
  const int64_t* list_tokens[kHashListSeqs];
  int32_t list_len[kHashListSeqs];
  uint64_t list_out[kHashListSeqs];   // first key of the sequence in `out`
  uint8_t ns8[kHashListNs];
};

// G sequences per CTA.
template <int G>
__global__ void __launch_bounds__(kHashThreads) kv_block_hashes_kernel(const __grid_constant__ HashParams p) {
  constexpr int SEG = kSegStripes / G;                 // stripes of one sequence per segment
  constexpr int SEGW = SEG * 4;                        // words
  __shared__ uint64_t s_in[2][G * SEGW];               // word * P2
  __shared__ uint64_t s_acc[2][G * SEGW];              // the four accumulators after each stripe
  __shared__ const int64_t* s_tok[G];
  __shared__ uint64_t* s_out[G];
  __shared__ int64_t s_stripes[G], s_blocks[G];
  __shared__ unsigned long long s_segs;
  const int tid = threadIdx.x;
  if (tid == 0) s_segs = 0;
  __syncthreads();
  if (tid < G) {
    const int64_t seq = (int64_t)blockIdx.x * G + tid;
    int64_t ntok = 0;
    s_tok[tid] = nullptr;
    s_out[tid] = nullptr;
    if (seq < p.num_seqs) {
      if (p.offsets) {
        const int64_t t0 = p.offsets[seq];
        ntok = p.offsets[seq + 1] - t0;
        s_tok[tid] = p.tokens + t0;
        s_out[tid] = p.out + p.out_offsets[seq];
      } else {
        ntok = p.list_len[seq];
        s_tok[tid] = p.list_tokens[seq];
        s_out[tid] = p.out + p.list_out[seq];
      }
    }
    const HashExtent x = hash_extent(ntok, p.ns_len, p.tpb);
    s_blocks[tid] = x.blocks;
    s_stripes[tid] = x.stripes;
    if (x.blocks > 0) atomicMax(&s_segs, (unsigned long long)max((int64_t)1, (x.stripes + SEG - 1) / SEG));
  }
  __syncthreads();
  const int32_t segs = (int32_t)s_segs;                // of 1024 words or 128: 2^31 of them are beyond any memory
  auto word = [&](int g, int64_t i) -> uint64_t {      // i-th word of the stream of sequence g
    if (i >= p.ns_len) return (uint64_t)__ldg(s_tok[g] + (i - p.ns_len));
    return p.ns ? (uint64_t)p.ns[i] : (uint64_t)p.ns8[i];
  };
  auto fetch = [&](int seg, int t, int threads) {
    for (int i = t; i < G * SEGW; i += threads) {
      const int g = i / SEGW;
      const int64_t w = (int64_t)seg * SEGW + i % SEGW;
      if (w < s_stripes[g] * 4) s_in[seg & 1][i] = word(g, w) * P2;
    }
  };
  // number of blocks whose digest covers at most `stripes` complete stripes
  auto blocks_upto = [&](int64_t stripes) -> int64_t {
    const int64_t words = 4 * stripes + 3 - p.ns_len;  // the longest stream with that many stripes, prefix taken off
    return words <= 0 ? 0 : words / p.tpb;
  };
  auto digest = [&](int seg, int t, int threads) {
    for (int g = 0; g < G; ++g) {
      const int64_t hi = min(s_blocks[g], blocks_upto((int64_t)(seg + 1) * SEG));
      for (int64_t b = (seg == 0 ? 0 : blocks_upto((int64_t)seg * SEG)) + t; b < hi; b += threads) {
        const int64_t n = p.ns_len + (b + 1) * p.tpb;  // words covered by this digest
        const int64_t stripes = n >> 2;
        uint64_t h = P5;                               // seed 0
        if (stripes > 0) {
          const uint64_t* v = &s_acc[seg & 1][g * SEGW + (int)(stripes - 1 - (int64_t)seg * SEG) * 4];
          const uint64_t v0 = v[0], v1 = v[1], v2 = v[2], v3 = v[3];
          h = rotl(v0, 1) + rotl(v1, 7) + rotl(v2, 12) + rotl(v3, 18);
          h = xmerge(h, v0); h = xmerge(h, v1); h = xmerge(h, v2); h = xmerge(h, v3);
        }
        h += (uint64_t)n * 8;
        for (int64_t i = 4 * stripes; i < n; ++i) {    // at most three trailing words
          h ^= xround(0, word(g, i));
          h = rotl(h, 27) * P1 + P4;
        }
        s_out[g][b] = avalanche(h);
      }
    }
  };
  if (segs > 0) fetch(0, tid, kHashThreads);
  __syncthreads();
  const int q = tid & 3, cg = tid >> 2;                // chain lanes: accumulator q of sequence cg
  uint64_t acc = q == 0 ? P1 + P2 : (q == 1 ? P2 : (q == 2 ? 0 : 0 - P1));
  for (int seg = 0; seg <= segs; ++seg) {
    if (tid < 32) {
      if (seg < segs && cg < G) {
        const uint64_t* in = &s_in[seg & 1][cg * SEGW + q];
        uint64_t* st = &s_acc[seg & 1][cg * SEGW + q];
        const int cnt = (int)min((int64_t)SEG, s_stripes[cg] - (int64_t)seg * SEG);
        int s = 0;
        for (; s + 8 <= cnt; s += 8) {
          uint64_t x[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) x[u] = in[(s + u) * 4];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            acc = rotl(acc + x[u], 31) * P1;
            st[(s + u) * 4] = acc;
          }
        }
        for (; s < cnt; ++s) {
          acc = rotl(acc + in[s * 4], 31) * P1;
          st[s * 4] = acc;
        }
      }
    } else {
      if (seg + 1 < segs) fetch(seg + 1, tid - 32, kHashHelpers);
      if (seg > 0) digest(seg - 1, tid - 32, kHashHelpers);
    }
    __syncthreads();
  }
}

// One sequence per CTA while all of them fit the GPU at once (6 CTAs of 33 KiB per SM x 148): the chain of each
// then runs at its own latency. Beyond that eight share a CTA, whose chain warp uses all of its lanes.
cudaError_t launch(const HashParams& p, cudaStream_t stream) {
  if (p.num_seqs <= 888)
    kv_block_hashes_kernel<1><<<(unsigned)p.num_seqs, kHashThreads, 0, stream>>>(p);
  else
    kv_block_hashes_kernel<8><<<(unsigned)((p.num_seqs + 7) / 8), kHashThreads, 0, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_kv_block_hashes(const int64_t* tokens, const int64_t* offsets, int64_t num_seqs, int tokens_per_block,
                                   const int64_t* ns_prefix, int64_t ns_len, uint64_t* out, const int64_t* out_offsets,
                                   cudaStream_t stream) {
  if (num_seqs <= 0) return cudaSuccess;
  if (tokens_per_block <= 0 || ns_len < 0 || (ns_len > 0 && ns_prefix == nullptr))
    return cudaErrorInvalidValue;
  HashParams p{};
  p.tokens = tokens;
  p.offsets = offsets;
  p.out_offsets = out_offsets;
  p.ns = ns_prefix;
  p.out = out;
  p.num_seqs = num_seqs;
  p.tpb = tokens_per_block;
  p.ns_len = ns_len;
  return launch(p, stream);
}

cudaError_t launch_kv_block_hashes_list(const int64_t* const* tokens, const int64_t* lens, int num_seqs,
                                        int tokens_per_block, const uint8_t* ns, int ns_len, uint64_t* out,
                                        cudaStream_t stream) {
  if (num_seqs <= 0) return cudaSuccess;
  if (tokens_per_block <= 0 || ns_len < 0 || ns_len > kHashListNs || num_seqs > kHashListSeqs)
    return cudaErrorInvalidValue;
  HashParams p{};
  p.out = out;
  p.num_seqs = num_seqs;
  p.tpb = tokens_per_block;
  p.ns_len = ns_len;
  for (int i = 0; i < ns_len; ++i) p.ns8[i] = ns[i];
  uint64_t keys = 0;
  for (int i = 0; i < num_seqs; ++i) {
    if (lens[i] < 0 || lens[i] > INT32_MAX) return cudaErrorInvalidValue;
    p.list_tokens[i] = tokens[i];
    p.list_len[i] = (int32_t)lens[i];
    p.list_out[i] = keys;
    keys += (uint64_t)hash_extent(lens[i], ns_len, tokens_per_block).blocks;
  }
  return launch(p, stream);
}

}  // namespace fkv
