// Staging buffers are taken by the groups that can use them, and by no other.
#include "fake_cuda.h"
#include "fake_layerwise.h"

#include <cstdio>

using namespace fkv;

struct Shape {
  int64_t chunk, blocks;
  bool abut = true;
  int engine = kEngineAuto, layers_per_batch = -1;
};

constexpr int kLayers = 2;
constexpr size_t kStaging = (size_t)kCeStageBufs * kCeStageBytes;

static GroupOptions options(const Shape& s) {
  GroupOptions o;
  o.num_layers = kLayers;
  o.chunk_bytes = s.chunk;
  o.h2d.engine = o.d2h.engine = s.engine;
  o.max_blocks_per_op = 4096;
  return o;
}
static GpuSide gpu() {
  GpuSide g;
  g.ptrs = {0x1000, 0x2000};
  return g;
}
static HostSide host(const Shape& s) {
  const int64_t kv = s.abut ? s.chunk : 2 * s.chunk;      // otherwise one of two ranks' slices
  return {0x100000, 2 * kv, kv, 2 * kLayers * kv, s.blocks};
}

static bool transfer_stages(const Shape& s) {
  fake::device_bytes = 0;
  TransferGroup g({gpu()}, host(s), options(s));
  return fake::device_bytes >= kStaging / 2;
}
static bool layerwise_stages(const Shape& s) {
  LayerwiseOptions o;
  o.group = options(s);
  o.layers_per_batch = s.layers_per_batch;
  fake::device_bytes = 0;
  LayerwiseGroup g({gpu()}, host(s), o);
  return fake::device_bytes >= kStaging / 2;
}

int main() {
  struct Case { Shape s; bool transfer, layerwise; };
  const int64_t K = 1 << 10;
  const Case cases[] = {
      {{32 * K, 4096}, true, true},
      {{32 * K, 4096, true, kEngineTma}, false, false},
      {{32 * K, 4096, true, kEngineAuto, 1}, true, false},   // one launch per layer asked for
      {{4 * K, 4096}, true, false},                          // rows of 8 KiB
      {{8 * K, 4096}, true, true},                           // rows of 16 KiB
      {{32 * K, 95}, true, false},                           // 5.94 MiB a layer in the whole pool
      {{32 * K, 96}, true, true},                            // 6 MiB
      {{32 * K, 63}, false, false},                          // no run of 8 MiB in it
      {{32 * K, 64}, true, false},
      {{32 * K, 4096, false}, false, false},
  };
  for (const Case& c : cases)
    if (transfer_stages(c.s) != c.transfer || layerwise_stages(c.s) != c.layerwise) {
      std::printf("chunk %lld, %lld blocks, engine %d\n", (long long)c.s.chunk, (long long)c.s.blocks, c.s.engine);
      return 1;
    }
  std::printf("OK\n");
  return 0;
}
