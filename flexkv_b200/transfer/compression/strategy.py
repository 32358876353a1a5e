"""Codec strategies used by the GPU<->host workers.

A strategy is attached once to a worker (``attach``) and then launches one fused
pack-or-unpack kernel per rank and op (``run``). Reference plug-in point:
flexkv/transfer/compression/common/strategy.py:13-51 (``CompressionStrategy.attach/run``,
``NullCompressionStrategy``); the nvCOMP ANS strategy of the reference
(compression/ans/ans_strategy.py) is replaced by own kernels that read GPU pages and write
packed tiles, either into the host pool itself or into the staging buffer of a copy-engine move.
"""
from __future__ import annotations

from typing import Any, Dict

from ... import _native
from ...storage.storage_engine import host_register_chunk_bytes


def codec_link(worker: Any, staging_bytes: int, min_op_bytes: int = 0, min_chunk: int = 0):
    """The native router of a worker's ops between kernel and copy engines, or None where every op belongs to the
    kernel: an engine of the user's choice (FLEXKV_TRANSFER_ENGINE), a host pool registered in parts, which a driver
    copy must not straddle, several ranks behind one op (they read the same id arrays) or one rank's slice of a wider
    block (which is not one span), chunks below ``min_chunk`` bytes, or a pool that cannot hold an op of
    ``min_op_bytes``. The router takes twice ``staging_bytes`` of GPU memory for its lifetime."""
    if len(worker.regs) != 1 or not worker.copy_engines or host_register_chunk_bytes():
        return None
    reg, host = worker.regs[0], worker.host
    if worker.kv_stride * reg.kv_dim * reg.num_layers != host.block_bytes or reg.chunk_bytes < min_chunk or \
            host.num_blocks * host.block_bytes < min_op_bytes:
        return None
    return _native.C.CodecLink(reg.device_id, reg.num_layers, reg.kv_dim, worker.kv_stride, staging_bytes)


class CompressionStrategy:
    """Interface. ``params`` is the addressing dict of one rank's launch (same keys as
    the plain copy kernel); ``stream`` is a raw CUDA stream handle."""
    name = "abstract"
    lossless = True

    def attach(self, worker: Any) -> None:
        self.worker = worker

    def detach(self) -> None:
        """Gives back what ``attach`` took; no run is in flight."""

    def host_chunk_bytes(self, chunk_elems: int, itemsize: int) -> int:
        raise NotImplementedError

    def run(self, params: Dict[str, Any], rank_index: int, num_ctas: int, stream: int) -> None:
        raise NotImplementedError

    @property
    def needs_size_table(self) -> bool:
        return False


class NullCompressionStrategy(CompressionStrategy):
    """Raw bytes through the plain copy kernel (used when every codec is refused)."""
    name = "none"

    def host_chunk_bytes(self, chunk_elems: int, itemsize: int) -> int:
        return chunk_elems * itemsize

    def run(self, params, rank_index, num_ctas, stream) -> None:
        _native.C.kv_copy(params, num_ctas, int(params.get("tile_bytes", 16384)), 0, stream)


class Fp8BlockScaleStrategy(CompressionStrategy):
    """bf16/fp16 -> fp8 e4m3 with one fp32 scale per 128 values (lossy, 0.53x bytes)."""
    name = "fp8_e4m3"
    lossless = False
    GROUP = 128

    def host_chunk_bytes(self, chunk_elems: int, itemsize: int) -> int:
        if chunk_elems % self.GROUP:
            raise ValueError("fp8 offload needs chunk elements divisible by 128")
        return chunk_elems + (chunk_elems // self.GROUP) * 4

    def __init__(self) -> None:
        self._link = None

    def attach(self, worker) -> None:
        super().attach(worker)
        self._link = codec_link(worker, 32 << 20, _native.C.CodecLink.MIN_QUANT_BYTES)

    def detach(self) -> None:
        self._link = None

    def run(self, params, rank_index, num_ctas, stream) -> None:
        if self._link is not None:
            self._link.quant_fp8(params, num_ctas, stream)
        else:
            _native.C.kv_quant_fp8(params, num_ctas, stream)


class ExponentPackStrategy(CompressionStrategy):
    """Lossless bf16 codec: sign+mantissa bytes stay raw, exponents are prefix coded by their frequency
    rank in the tile (about 0.68x bytes on unit-normal data)."""
    name = "bf16_xp"
    TILE_ELEMS = 8192
    TILE_SLOT = 2 * TILE_ELEMS + 128

    def __init__(self, size_table=None, spec=None) -> None:
        self.size_table = size_table
        self.spec = spec
        self._link = None

    def attach(self, worker) -> None:
        super().attach(worker)
        # restores only; rows of about 1000 tiles per copy need a larger buffer than whole blocks do
        C = _native.C.CodecLink
        self._link = codec_link(worker, 64 << 20, C.MIN_ROW_BYTES, C.MIN_ROW_CHUNK) if worker.h2d else None

    def detach(self) -> None:
        self._link = None

    @property
    def needs_size_table(self) -> bool:
        return True

    def host_chunk_bytes(self, chunk_elems: int, itemsize: int) -> int:
        if chunk_elems % 1024:
            raise ValueError("the exponent-packing codec needs chunk elements divisible by 1024")
        full, rest = divmod(chunk_elems, self.TILE_ELEMS)
        return full * self.TILE_SLOT + ((2 * rest + 128) if rest else 0)

    def run(self, params, rank_index, num_ctas, stream) -> None:
        if self.size_table is None or self.spec is None:
            raise RuntimeError("exponent-packing strategy used without a size table")
        off = self.spec.rank_offset_entries(rank_index)
        table, layers = self.size_table.data_ptr() + 4 * off, self.spec.kernel_layers()
        if self._link is not None:
            self._link.compress_bf16(params, table, layers, num_ctas, self.worker.staged_num_ctas, stream)
        else:
            _native.C.kv_compress_bf16(params, table, layers, num_ctas, stream)


def strategy_for(codec: str, size_table=None, spec=None) -> CompressionStrategy:
    if codec == "fp8_e4m3":
        return Fp8BlockScaleStrategy()
    if codec == "bf16_xp":
        return ExponentPackStrategy(size_table, spec)
    if codec == "none":
        return NullCompressionStrategy()
    raise ValueError(f"unknown host codec {codec!r}")
