// An op whose launch fails half way leaves nothing in flight: neither kernels that read its block ids nor copies that
// still move blocks, whatever the stream.
#include "fake_cuda.h"

#include <cstdio>
#include <vector>

#include "transfer_group.h"

using namespace fkv;

#define CHECK(c)                                                       \
  do {                                                                 \
    if (!(c)) { std::printf("%s:%d: %s\n", __FILE__, __LINE__, #c); return 1; } \
  } while (0)

constexpr int kLayers = 2, kBlocks = 64;
constexpr int64_t kChunk = 64 << 10, kBlock = kLayers * 2 * kChunk;   // 256 KiB: a run of 32 blocks is 8 MiB

struct Rig {
  std::vector<uint8_t> gpu[kLayers], host;
  std::unique_ptr<TransferGroup> group;

  Rig() : host((size_t)(kBlocks * kBlock)) {
    GpuSide g;
    for (auto& t : gpu) {
      t.resize((size_t)(kBlocks * 2 * kChunk));
      g.ptrs.push_back(reinterpret_cast<uint64_t>(t.data()));
    }
    g.kv_stride = kBlocks * kChunk;
    g.block_stride = kChunk;
    g.num_blocks = kBlocks;
    GroupOptions o;
    o.num_layers = kLayers;
    o.chunk_bytes = kChunk;
    o.h2d.engine = o.d2h.engine = kEngineAuto;
    o.ring_slots = 1;
    o.max_blocks_per_op = kBlocks;
    o.ce_staging_blocks = 8;
    group.reset(new TransferGroup({g}, {reinterpret_cast<uint64_t>(host.data()), 2 * kChunk, kChunk, kBlock, kBlocks}, o));
  }
  ~Rig() { fake::fail_launch = -1; }
};

// pages in reverse, host blocks in a row: the staged route, pieces of at most 8 blocks
static std::vector<int64_t> pages(int n, int first) {
  std::vector<int64_t> v;
  for (int i = 0; i < n; ++i) v.push_back(first + n - 1 - i);
  return v;
}
static std::vector<int64_t> row(int n) {
  std::vector<int64_t> v;
  for (int i = 0; i < n; ++i) v.push_back(i);
  return v;
}

// `submitted`: through the rank's thread, else on the calling thread
static int failed_op(bool h2d, bool submitted, int failing_launch) {
  Rig rig;
  std::memset(rig.host.data(), 7, rig.host.size());
  const auto g = pages(32, 0), c = row(32);
  fake::launches = 0;
  fake::fail_launch = failing_launch;
  auto op = [&](const std::vector<int64_t>& gpu) {
    if (!submitted) return rig.group->transfer(gpu.data(), c.data(), 32, h2d, 0, kLayers);
    return rig.group->wait(rig.group->submit(gpu.data(), c.data(), 32, h2d, 0, kLayers));
  };
  CHECK(op(g).status < 0);
  CHECK(fake::launches == failing_launch + 1 && rig.group->staged_ops() == 1);
  CHECK(fake::in_flight() == 0);
  // the next op has the failed one's ring slot: no kernel may read the new ids for the old op
  fake::fail_launch = -1;
  const auto g2 = pages(32, 32);
  for (auto& t : rig.gpu) std::memset(t.data(), 0, t.size());
  CHECK(op(g2).status == 0);
  if (h2d)
    for (int l = 0; l < kLayers; ++l)
      for (int64_t k = 0; k < 2; ++k)
        for (int64_t b = 0; b < kBlocks; ++b)
          CHECK(rig.gpu[l][(size_t)((k * kBlocks + b) * kChunk)] == (b < 32 ? 0 : 7));
  return 0;
}

int main() {
  for (int h2d = 0; h2d < 2; ++h2d)
    for (int submitted = 0; submitted < 2; ++submitted)
      for (int at = 0; at < 4; ++at)
        if (failed_op(h2d != 0, submitted != 0, at)) return 1;
  std::printf("OK\n");
  return 0;
}
