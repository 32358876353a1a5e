// Batched block-key generation on the GPU: cumulative streaming XXH64 (seed 0) over int64
// token ids, one digest per block, bit-identical to the host hasher (hasher.h; reference
// behaviour csrc/hash.cpp:47-66). For callers whose token ids already live on the device
// (an engine that keeps its prompts in HBM) or that hash thousands of long sequences at once;
// for a single request the host hasher (about 12 us per 8K tokens) is faster than any launch.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

namespace fkv {

// What a sequence of `ntok` tokens behind a prefix of `ns_len` words comes to: keys, and the complete stripes of four
// words that its last key covers. 64 bits: with one token per block 2^31 tokens are 16 GiB.
struct HashExtent {
  int64_t blocks, stripes;
};
__host__ __device__ constexpr HashExtent hash_extent(int64_t ntok, int64_t ns_len, int64_t tokens_per_block) {
  const int64_t blocks = ntok / tokens_per_block;
  return {blocks, blocks > 0 ? (ns_len + blocks * tokens_per_block) >> 2 : 0};
}

// tokens: all sequences back to back; offsets[n+1] (in tokens) and out_offsets[n+1] (in blocks)
// are device- or mapped-host-readable. ns_prefix (ns_len int64 values, may be null) is fed
// before every sequence.
cudaError_t launch_kv_block_hashes(const int64_t* tokens, const int64_t* offsets, int64_t num_seqs, int tokens_per_block,
                                   const int64_t* ns_prefix, int64_t ns_len, uint64_t* out, const int64_t* out_offsets,
                                   cudaStream_t stream);

constexpr int kHashListSeqs = 128;   // sequences whose addresses travel in the launch parameters
constexpr int kHashListNs = 256;     // namespace bytes that do

// The same for at most kHashListSeqs sequences that lie anywhere on the device: no concatenation and no offset
// tables to upload. tokens[i] / lens[i]: device address and length of sequence i (lengths below 2^31); the keys of
// sequence i follow those of sequence i-1 in `out`. ns: at most kHashListNs prefix values, each one byte.
cudaError_t launch_kv_block_hashes_list(const int64_t* const* tokens, const int64_t* lens, int num_seqs,
                                        int tokens_per_block, const uint8_t* ns, int ns_len, uint64_t* out,
                                        cudaStream_t stream);

}  // namespace fkv
