// A layerwise restore that fails half way leaves nothing in flight when its waiters are released.
#include "fake_cuda.h"
#include "fake_layerwise.h"

#include <cstdio>
#include <vector>

using namespace fkv;

#define CHECK(c)                                                       \
  do {                                                                 \
    if (!(c)) { std::printf("%s:%d: %s\n", __FILE__, __LINE__, #c); return 1; } \
  } while (0)

constexpr int kLayers = 3, kBlocks = 64;
constexpr int64_t kChunk = 64 << 10, kRow = 2 * kChunk, kBlock = kLayers * kRow;   // 8 MiB a layer

// form: 0 = rows by the copy engines, 1 = a launch per layer, 2 = layers made of members
static int failed_restore(int form, NotifyMode notify, int failing_launch) {
  std::vector<uint8_t> gpu[kLayers], host((size_t)(kBlocks * kBlock), 7);
  GpuSide g;
  for (auto& t : gpu) {
    t.resize((size_t)(kBlocks * kRow));
    g.ptrs.push_back(reinterpret_cast<uint64_t>(t.data()));
  }
  g.kv_stride = kBlocks * kChunk;
  g.block_stride = kChunk;
  g.num_blocks = kBlocks;
  const HostSide h{reinterpret_cast<uint64_t>(host.data()), kRow, kChunk, kBlock, kBlocks};
  LayerwiseOptions o;
  o.group.num_layers = kLayers;
  o.group.chunk_bytes = kChunk;
  o.group.h2d.engine = form == 0 ? kEngineAuto : kEngineTma;
  o.group.max_blocks_per_op = kBlocks;
  o.notify = notify;
  o.layers_per_batch = form == 0 ? -1 : 1;
  std::unique_ptr<LayerwiseGroup> group;
  if (form == 2) {
    std::vector<std::vector<LayerMember>> members;
    for (int l = 0; l < kLayers; ++l) members.push_back({LayerMember{0, l}});
    group.reset(new LayerwiseGroup({LayerwiseMemberGroup{{g}, h, o.group}}, members, h, o));
  } else {
    group.reset(new LayerwiseGroup({g}, h, o));
  }
  std::vector<int64_t> pages, row;
  for (int i = 0; i < kBlocks; ++i) {
    pages.push_back(kBlocks - 1 - i);
    row.push_back(i);
  }
  fake::launches = 0;
  fake::fail_launch = failing_launch;
  const LayerwiseResult r = group->restore(pages.data(), row.data(), kBlocks, 0, nullptr, nullptr, nullptr, nullptr, 0);
  fake::fail_launch = -1;
  CHECK(r.status < 0 && fake::launches == failing_launch + 1);
  CHECK(fake::in_flight() == 0);
  const uint32_t* flags = reinterpret_cast<const uint32_t*>(group->host_flags_ptr(0, 0));
  for (int l = 0; l < kLayers; ++l) CHECK(flags[l] == r.epoch);
  CHECK(group->counter_status(0) == r.status);
  return 0;
}

int main() {
  for (int form = 0; form < 3; ++form)
    for (NotifyMode m : {NotifyMode::HOSTFUNC, NotifyMode::POLLING, NotifyMode::FLAG})
      for (int at = 0; at < kLayers; ++at)
        if (failed_restore(form, m, at)) {
          std::printf("form %d, mode %d, launch %d\n", form, (int)m, at);
          return 1;
        }
  std::printf("OK\n");
  return 0;
}
