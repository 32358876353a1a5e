"""What ``gpu_block_hashes`` hands to the kernel, without a GPU: CPU tensors that pass for CUDA tensors, a stream and a
native module that only record what they are asked for, in order."""
import types

import pytest
import torch

from flexkv_b200.ops import kv_hash

CONVERSIONS = {"to", "contiguous", "cat", "clone"}


class Recorded(torch.Tensor):
    """A tensor that says it is on GPU ``index`` and writes down the copies made of it."""
    log = []
    index = 0

    @property
    def is_cuda(self):
        return self.index >= 0

    @property
    def device(self):
        return torch.device("cuda", self.index) if self.index >= 0 else torch.device("cpu")

    def get_device(self):
        return self.index

    def record_stream(self, stream):
        self.log.append(("keep", self.data_ptr()))

    @classmethod
    def __torch_function__(cls, func, types_, args=(), kwargs=None):
        if func.__name__ in CONVERSIONS:
            cls.log.append(("convert", func.__name__))
        return super().__torch_function__(func, types_, args, kwargs or {})


class OnOtherGpu(Recorded):
    index = 1


class OnHost(Recorded):
    index = -1


class Stream:
    cuda_stream = 7

    def __init__(self, log):
        self.log = log

    def wait_stream(self, other):
        self.log.append(("wait", None))


@pytest.fixture
def rig(monkeypatch):
    log = []
    monkeypatch.setattr(Recorded, "log", log)

    class Native:
        HASH_LIST_SEQS, HASH_LIST_NS = kv_hash._native.C.HASH_LIST_SEQS, kv_hash._native.C.HASH_LIST_NS

        def kv_block_hashes_list(self, tokens, lens, *rest):
            log.append(("launch", list(tokens)))

        def kv_block_hashes(self, tokens, *rest):
            log.append(("launch", [tokens]))

    monkeypatch.setattr(kv_hash, "_native", types.SimpleNamespace(C=Native()))
    current = Stream(log)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: current)
    for name in ("empty", "tensor"):
        real = getattr(torch, name)
        monkeypatch.setattr(torch, name, lambda *a, _real=real, device=None, **kw: _real(*a, **kw).as_subclass(Recorded))
    return types.SimpleNamespace(log=log, side=Stream(log))


def _seqs(n, kind=Recorded, dtype=torch.int64):
    return [torch.arange(40, dtype=dtype).as_subclass(kind) for _ in range(n)]


@pytest.mark.parametrize("stranger", [OnHost, OnOtherGpu])
@pytest.mark.parametrize("count", [2, 200])
def test_sequences_elsewhere_are_refused_before_any_launch(rig, stranger, count):
    """The kernel reads the addresses it is given: one in host memory or on another GPU must not reach it."""
    seqs = _seqs(count)
    seqs[count // 2] = _seqs(1, stranger)[0]
    with pytest.raises(ValueError):
        kv_hash.gpu_block_hashes(seqs, 16)
    with pytest.raises(ValueError):
        kv_hash.gpu_block_hashes(_seqs(1, OnHost), 16, stream=rig.side)
    assert not [e for e in rig.log if e[0] == "launch"]


@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
@pytest.mark.parametrize("count", [3, 200])
def test_a_side_stream_waits_for_the_conversions(rig, count, dtype):
    """Conversions, concatenations and uploads run on the current stream; the other stream is told to wait for it after
    the last of them and before the launch."""
    seqs = _seqs(count, dtype=dtype)
    seqs[1] = seqs[1][::2]
    kv_hash.gpu_block_hashes(seqs, 16, stream=rig.side)
    what = [e[0] for e in rig.log]
    last = max(i for i, w in enumerate(what) if w == "convert")
    assert last < what.index("wait") < what.index("launch") and what.count("wait") == 1


@pytest.mark.parametrize("count,in_place", [(1, True), (3, False), (200, False)])
def test_a_side_stream_reads_copies(rig, count, in_place):
    """Several sequences are copied in the order of the current stream, so that the caller may go on to overwrite them
    there while the keys are computed on the other stream."""
    seqs = _seqs(count)
    mine = {t.data_ptr() for t in seqs}
    kv_hash.gpu_block_hashes(seqs, 16, stream=rig.side)
    read = [e[1] for e in rig.log if e[0] == "launch"][0]
    assert all((p in mine) == in_place for p in read)
    assert set(read) <= {e[1] for e in rig.log if e[0] == "keep"}


def test_the_current_stream_reads_in_place(rig):
    seqs = _seqs(4)
    kv_hash.gpu_block_hashes(seqs, 16)
    assert rig.log == [("launch", [t.data_ptr() for t in seqs])]


@pytest.mark.parametrize("ntok", [0, 15, 16, 4099, 2**31 - 1, 2**31, 2**33 + 5])
@pytest.mark.parametrize("tpb,ns_len", [(1, 0), (16, 7), (64, 300)])
def test_extent_of_a_sequence(ntok, tpb, ns_len):
    """Keys and stripes of a sequence, as the kernel splits its work: both go beyond 32 bits with short blocks."""
    blocks = ntok // tpb
    assert kv_hash._native.C.hash_extent(ntok, ns_len, tpb) == (blocks, (ns_len + blocks * tpb) // 4 if blocks else 0)
