"""The engine that each GPU<->host path asks the native side for, without a GPU: the native constructors only record
their arguments."""
import types

import pytest

from flexkv_b200 import _native
from flexkv_b200.common.storage import KVCacheLayoutType
from flexkv_b200.transfer import layerwise, workers
from flexkv_b200.transfer.compression import strategy

MB = 1 << 20


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
    worker = types.SimpleNamespace(regs=[st.gpu_regs[key][0]], copy_engines=cfg["engine"] >= 2, kv_stride=MB // 4)
    if not worker.copy_engines:
        assert strategy.codec_link(worker, 32 * MB) is None
