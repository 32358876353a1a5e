"""The engine that each GPU<->host path asks the native side for, without a GPU: the native constructors only record
their arguments."""
import types

import pytest

from flexkv_b200 import _native
from flexkv_b200.common.storage import KVCacheLayoutType
from flexkv_b200.transfer import layerwise, workers
from flexkv_b200.transfer.compression import strategy

MB = 1 << 20
REAL = _native.C


class Built(Exception):
    pass


def _storage(num_blocks=64, block_bytes=2 * MB):
    """One registered GPU of 4 layers with K and V planes of 256 KiB a block, and a block-first host pool."""
    reg = types.SimpleNamespace(num_layers=4, kv_dim=2, chunk_bytes=block_bytes // 8, device_id=0,
                                as_native=lambda: {})
    host = types.SimpleNamespace(base=0x7F0000000000, num_blocks=num_blocks, block_bytes=block_bytes,
                                 layer_stride=block_bytes // 4, kv_stride=block_bytes // 8, chunk_bytes=block_bytes // 8,
                                 quant="none", layout=types.SimpleNamespace(is_multi_group=False,
                                                                            type=KVCacheLayoutType.BLOCKFIRST))
    return types.SimpleNamespace(gpu_regs={"k": {0: reg}}, host=host, pp_stage_offset=lambda r: 0)


MODEL = types.SimpleNamespace(use_mla=False, num_kv_heads=8, effective_tp_size=1)


@pytest.fixture
def native(monkeypatch):
    def record(gpus, host, opts):
        raise Built(opts)
    monkeypatch.setattr(_native, "C", types.SimpleNamespace(TransferGroup=record, LayerwiseGroup=record))
    monkeypatch.delenv("FLEXKV_HOST_REGISTER_CHUNK_BYTES", raising=False)
    monkeypatch.delenv("FLEXKV_CUDAHOST_CHUNK_SIZE_GB", raising=False)


class Key(str):
    pp_rank = 0


@pytest.mark.parametrize("engine,chunk,want", [("auto", None, 3), ("ce", None, 2), ("tma", None, 0), ("simt", None, 1),
                                               ("auto", 32 * MB, 0), ("ce", 32 * MB, 0), ("simt", 32 * MB, 1),
                                               ("auto", 128 * MB, 3), ("auto", 128 * MB - 4096, 0)])
def test_pool_registered_in_parts_is_left_to_the_kernels(native, monkeypatch, engine, chunk, want):
    """A driver copy that straddles two registrations fails. The pool here holds 128 MiB: one part of that size is one
    registration."""
    monkeypatch.setattr(workers.GLOBAL_CONFIG_FROM_ENV, "transfer_engine", engine)
    if chunk is not None:
        monkeypatch.setenv("FLEXKV_HOST_REGISTER_CHUNK_BYTES", str(chunk))
    st, key = _storage(), Key("k")
    with pytest.raises(Built) as raw:
        workers.build_transfer_group(st, MODEL, key)
    with pytest.raises(Built) as layered:
        layerwise.build_layerwise_group(st, MODEL, key, notify_mode="polling")
    for opts in (raw.value.args[0], layered.value.args[0]):
        assert opts["h2d"]["engine"] == opts["d2h"]["engine"] == want
    cfg = workers.host_launch_cfg(workers.GLOBAL_CONFIG_FROM_ENV, True, st.host)
    assert cfg["engine"] == want


@pytest.mark.parametrize("name,h2d,blocks,block_bytes,n_ranks,slice_of,want", [
    ("fp8", True, 64, 2 * MB, 1, 1, True), ("fp8", False, 64, 2 * MB, 1, 1, True),
    ("fp8", True, 23, 2 * MB, 1, 1, False),                    # a pool of 46 MiB: no op reaches the 48 MiB
    ("fp8", True, 64, 2 * MB, 2, 1, False), ("fp8", True, 64, 2 * MB, 1, 2, False),
    ("xp", True, 64, 2 * MB, 1, 1, True), ("xp", False, 64, 2 * MB, 1, 1, False),
    ("xp", True, 63, 2 * MB, 1, 1, False),                     # 126 of 128 MiB
    ("xp", True, 4096, 64 << 10, 1, 1, True), ("xp", True, 4096, 32 << 10, 1, 1, False)])       # 8 and 4 KiB chunks
def test_codec_routers_are_made_where_they_can_be_used(native, name, h2d, blocks, block_bytes, n_ranks, slice_of, want):
    """A router holds staging buffers on the GPU from its start."""
    made = []

    class CodecLink:
        MIN_QUANT_BYTES, MIN_ROW_BYTES, MIN_ROW_CHUNK = (getattr(REAL.CodecLink, k) for k in (
            "MIN_QUANT_BYTES", "MIN_ROW_BYTES", "MIN_ROW_CHUNK"))

        def __init__(self, *args):
            made.append(args)

    _native.C.CodecLink = CodecLink
    st = _storage(blocks, block_bytes)
    reg = st.gpu_regs["k"][0]
    worker = types.SimpleNamespace(regs=[reg] * n_ranks, copy_engines=True, h2d=h2d, host=st.host,
                                   kv_stride=st.host.kv_stride // slice_of)
    s = strategy.Fp8BlockScaleStrategy() if name == "fp8" else strategy.ExponentPackStrategy(object(), object())
    s.attach(worker)
    assert bool(made) == (s._link is not None) == want
    worker.copy_engines = False
    s.attach(worker)
    assert s._link is None
