"""The worker of packed host pools without a GPU: streams, events and the codec only record what is asked of them."""
import contextlib
import types

import numpy as np
import pytest
import torch

from flexkv_b200.transfer.workers import QuantGpuHostWorker


class Stream:
    def __init__(self, dev, log):
        self.dev, self.log, self.cuda_stream = dev, log, dev

    def synchronize(self):
        self.log.append(("sync", self.dev))


class Event:
    """Time passes by one millisecond with every launch."""

    def __init__(self, clock, log):
        self.clock, self.log, self.at = clock, log, None

    def record(self, stream):
        self.at = self.clock[0]

    def synchronize(self):
        self.log.append(("event", self.at))

    def elapsed_time(self, later):
        return float(later.at - self.at)


def _worker(devices, run, shared=False):
    """A worker over one rank per entry of ``devices``; ``run(rank)`` stands for the codec's launch."""
    log, clock = [], [0]
    w = QuantGpuHostWorker.__new__(QuantGpuHostWorker)
    w.h2d, w.shared, w.name = True, shared, "h2d-test"
    w._torch = types.SimpleNamespace(empty=torch.empty, int64=torch.int64,
                                     cuda=types.SimpleNamespace(device=lambda d: contextlib.nullcontext(),
                                                                Event=lambda enable_timing: Event(clock, log)))
    w.regs = [types.SimpleNamespace(device_id=d, num_layers=1, kv_dim=2, chunk_bytes=1024, ptrs=[1], idx_layer_mul=1,
                                    idx_kv_mul=0, layer_stride=0, kv_stride=0, block_stride=1024, num_blocks=64)
              for d in devices]
    w.host = types.SimpleNamespace(base=0, block_bytes=4096, num_blocks=64)
    w.layer_stride = w.kv_stride = w.tp_stride = 1024
    w.num_ctas = 8
    w.streams = {d: Stream(d, log) for d in devices}
    w._ids = torch.zeros((2, 64), dtype=torch.int64)
    w.status = {d: torch.zeros(8, dtype=torch.int32) for d in devices}
    w._words = {d: t.numpy() for d, t in w.status.items()}
    w._events = [(Event(clock, log), Event(clock, log)) for _ in devices]

    class Strategy:
        def run(self, params, rank, num_ctas, stream):
            log.append(("launch", rank))
            clock[0] += run(rank, w)
    w.strategy = Strategy()
    return w, log


def _op(n=5):
    return types.SimpleNamespace(src_block_ids=np.arange(n), dst_block_ids=np.arange(n), num_layers=-1, layer_start=0)


def test_a_rank_that_cannot_launch_waits_for_the_others():
    """The ranks share the id buffers: what the first ones queued must be done with them before the next op."""
    def run(rank, w):
        w._words[rank][3] = 1                    # a kernel that did run reports something
        if rank == 2:
            raise RuntimeError("launch failed")
        return 1
    w, log = _worker([0, 1, 2], run)
    with pytest.raises(RuntimeError):
        w.execute(_op())
    assert {e for e in log if e[0] == "sync"} == {("sync", 0), ("sync", 1), ("sync", 2)}
    assert not any(words.any() for words in w._words.values())

@pytest.mark.parametrize("devices", [[0], [0, 1], [0, 0, 0]])
def test_time_of_an_op_is_that_of_its_slowest_rank(devices):
    took = [7, 3, 2]
    w, _ = _worker(devices, lambda rank, w: took[rank])
    out = w.execute(_op())
    assert out.success and out.gpu_ms == 7.0
