// Several threads on one transfer group, blocking calls and submitted ops mixed.
#include "fake_cuda.h"

#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <thread>
#include <vector>

#include "transfer_group.h"

using namespace fkv;

#define CHECK(c)                                                       \
  do {                                                                 \
    if (!(c)) { std::printf("%s:%d: %s\n", __FILE__, __LINE__, #c); return 1; } \
  } while (0)

constexpr int kBlocks = 256;
constexpr int64_t kChunk = 1024, kBlock = 2 * kChunk;

struct Rig {
  std::vector<uint8_t> gpu, host;
  std::unique_ptr<TransferGroup> group;
  Rig() : gpu((size_t)(kBlocks * kBlock)), host((size_t)(kBlocks * kBlock)) {
    GpuSide g;
    g.ptrs.push_back(reinterpret_cast<uint64_t>(gpu.data()));
    g.kv_stride = kBlocks * kChunk;
    g.block_stride = kChunk;
    g.num_blocks = kBlocks;
    GroupOptions o;
    o.chunk_bytes = kChunk;
    o.max_blocks_per_op = kBlocks;
    o.ring_slots = 16;
    group.reset(new TransferGroup({g}, {reinterpret_cast<uint64_t>(host.data()), kBlock, kChunk, kBlock, kBlocks}, o));
  }
  ~Rig() { fake::on_launch = nullptr; }
};

// While one op is being launched others arrive: they are launched in the order they came in, and ahead of one another
// as far as the group allows (four ops).
static int order_and_overlap(bool first_submitted) {
  Rig rig;
  std::mutex mu;
  std::condition_variable cv;
  bool started = false, go = false;
  std::vector<int64_t> order;
  size_t ahead = 0;
  fake::on_launch = [&](const KvCopyParams& p) {
    std::unique_lock<std::mutex> lk(mu);
    order.push_back(p.gpu_blocks[0]);
    ahead = std::max(ahead, fake::in_flight());
    started = true;
    cv.notify_all();
    cv.wait(lk, [&] { return go; });
  };
  auto op = [&](int64_t b, bool submitted) {
    if (submitted) rig.group->wait(rig.group->submit(&b, &b, 1, true, 0, 1));
    else rig.group->transfer(&b, &b, 1, true, 0, 1);
  };
  std::vector<std::thread> threads;
  threads.emplace_back(op, 0, first_submitted);
  { std::unique_lock<std::mutex> lk(mu); cv.wait(lk, [&] { return started; }); }
  for (int64_t b = 1; b <= 4; ++b) {
    threads.emplace_back(op, b, b == 2);
    std::this_thread::sleep_for(std::chrono::milliseconds(100));
  }
  { std::lock_guard<std::mutex> g(mu); go = true; }
  cv.notify_all();
  for (auto& t : threads) t.join();
  CHECK((order == std::vector<int64_t>{0, 1, 2, 3, 4}));
  CHECK(ahead == 3);
  return 0;
}

// Every op moves its own blocks there and back; a mix-up of ids, slots or status words shows in the bytes.
static int many_threads() {
  Rig rig;
  for (size_t i = 0; i < rig.host.size(); ++i) rig.host[i] = (uint8_t)(i / kChunk * 7 + 1);
  const std::vector<uint8_t> want = rig.host;
  std::atomic<int> bad{0};
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&, t] {
      for (int round = 0; round < 200; ++round) {
        std::vector<int64_t> ids;
        for (int i = 0; i < 1 + (round + t) % 32; ++i) ids.push_back(t * 32 + i);
        for (bool h2d : {true, false}) {
          const int64_t n = (int64_t)ids.size();
          const OpResult r = (round + t) % 3 ? rig.group->transfer(ids.data(), ids.data(), n, h2d, 0, 1)
                                             : rig.group->wait(rig.group->submit(ids.data(), ids.data(), n, h2d, 0, 1));
          if (r.status) ++bad;
          if (h2d)
            for (int64_t b : ids) std::memset(rig.host.data() + b * kBlock, 0, (size_t)kBlock);
        }
        const int64_t wrong = kBlocks;      // out of range: reported by this op alone
        if (rig.group->transfer(&wrong, &ids[0], 1, true, 0, 1).status != KV_ERR_GPU_BLOCK_RANGE) ++bad;
      }
    });
  for (auto& t : threads) t.join();
  CHECK(bad == 0);
  CHECK(rig.host == want);
  return 0;
}

int main() {
  if (order_and_overlap(false) || order_and_overlap(true) || many_threads()) return 1;
  std::printf("OK\n");
  return 0;
}
