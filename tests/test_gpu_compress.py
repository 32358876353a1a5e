"""Lossless exponent coder: packed bytes equal a CPU reference written from the format
description, the CPU decoder restores the GPU's output, every bit pattern round-trips,
sizes land in the table, ratio on N(0,1)."""
import numpy as np
import pytest
import torch

from flexkv_b200 import _native
from flexkv_b200.models import KVShape, alloc_paged_cache
from flexkv_b200.ops.kv_compress import (TILE_ELEMS, TILE_SLOT, chunk_slot_bytes, kv_compress,
                                         reference_compress_tile, reference_decompress_tile, size_table_entries,
                                         tiles_per_chunk)
from flexkv_b200.ops.kv_copy import HostSide, decode_status, make_params, new_status
from flexkv_b200.storage.gpu_layout import register_tensors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [KVShape("c1", 2, 8, 128, tokens_per_block=16),                 # 16384-element chunks
                                   KVShape("c2", 2, 1, 576, use_mla=True, tokens_per_block=64),   # 36864: ragged tile
                                   KVShape("c3", 3, 1, 128, tokens_per_block=8)])                 # 1024-element chunks
def test_roundtrip_is_bit_exact_and_bytes_match_reference(shape):
    dev = torch.device("cuda:0")
    NB, n = 24, 13
    kv, layout = alloc_paged_cache(shape, NB, dev, "vllm", fill="normal", seed=71)
    # adversarial content: zeros, denormals, huge, NaN/Inf patterns, a constant run, and (second block of
    # layer 0) uniformly random bits, whose exponents do not compress: those tiles travel raw
    kv[0].view(-1).view(torch.int16)[reg_elems(kv[0], shape):2 * reg_elems(kv[0], shape)] = torch.randint(
        -32768, 32767, (reg_elems(kv[0], shape),), dtype=torch.int16, device=dev)
    flat = kv[0].view(-1).view(torch.int16)
    flat[:128] = 0
    flat[128:256] = torch.randint(-32768, 32767, (128,), dtype=torch.int16, device=dev)
    flat[256:384] = 0x3F80                      # all 1.0
    flat[384:388] = torch.tensor([0x7F80, -128, 0x7FC0, 1], dtype=torch.int16, device=dev)   # inf, -inf, nan, denormal
    # the last layer has channels of very different scales (12 octaves): a flat exponent profile, which takes
    # the second code shape, with exponents beyond the 16 ranked ones (escapes of that shape)
    gsc = torch.Generator().manual_seed(3)
    kv[-1].mul_(torch.exp2(torch.rand(kv[-1].shape[-1], generator=gsc) * 12 - 6).to(dev).to(kv[-1].dtype))
    reg = register_tensors(kv, layout)
    E = reg.chunk_bytes // 2
    L, K, tpc = shape.num_layers, shape.kv_dim, tiles_per_chunk(E)
    slot = chunk_slot_bytes(E)
    modes_seen = set()
    pool = torch.zeros(NB, L, K, slot, dtype=torch.uint8).pin_memory()
    host = HostSide(pool.data_ptr(), K * slot, slot, L * K * slot, NB)
    table = torch.zeros(size_table_entries(NB, L, K, E), dtype=torch.int32).pin_memory()
    rng = np.random.default_rng(5)
    g = np.concatenate([[0, 1], rng.permutation(np.arange(2, NB))[:n - 2]]).astype(np.int64)
    c = rng.permutation(NB)[:n].astype(np.int64)
    status = new_status(dev)
    keep = kv_compress(reg, host, table, g, c, h2d=False, num_ctas=5, status=status)
    torch.cuda.synchronize()
    assert decode_status(status) == 0
    tv = table.view(NB, L, K, tpc)
    total_packed, total_raw = 0, 0
    for i in (0, 1, n - 1):                                  # byte-level check of a few blocks, all layers
        for l in range(L):
            for k in range(K):
                x = (kv[l][int(g[i])] if shape.use_mla else kv[l][k][int(g[i])]).reshape(-1).cpu()
                for t in range(tpc):
                    tile = x[t * TILE_ELEMS:(t + 1) * TILE_ELEMS]
                    want = reference_compress_tile(tile)
                    size = int(tv[int(c[i]), l, k, t])
                    assert size == want.numel(), (i, l, k, t, size, want.numel())
                    got = pool[int(c[i]), l, k, t * TILE_SLOT:t * TILE_SLOT + size]
                    assert torch.equal(got, want), (i, l, k, t)
                    modes_seen.add(int(got[0]))
                    back = reference_decompress_tile(got)
                    assert torch.equal(back.view(torch.int16), tile.view(torch.int16)), (i, l, k, t)
    assert {1, 2} <= modes_seen and (0 in modes_seen or shape.use_mla or E < TILE_ELEMS), modes_seen
    for i in range(2, n):                                    # blocks 0 and 1 carry the adversarial content
        total_packed += int(tv[int(c[i]), :L - 1].sum())
        total_raw += (L - 1) * K * E * 2
    # N(0,1) packs to 0.675 in full tiles; 1024-value tiles carry 48 bytes of header per 2 KiB
    assert total_packed < (0.70 if E >= TILE_ELEMS else 0.80) * total_raw
    saved = [t.clone() for t in kv]
    for t in kv:
        t.zero_()
    g2 = rng.permutation(NB)[:n].astype(np.int64)
    keep += kv_compress(reg, host, table, g2, c, h2d=True, num_ctas=3, status=status)
    torch.cuda.synchronize()
    assert decode_status(status) == 0
    gi, g2i = torch.from_numpy(g).to(dev), torch.from_numpy(g2).to(dev)
    for l in range(L):
        a = saved[l][gi] if shape.use_mla else saved[l][:, gi]
        b = kv[l][g2i] if shape.use_mla else kv[l][:, g2i]
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))


def reg_elems(t, shape):
    """elements of one (kv plane, block) chunk of a vLLM-layout layer tensor"""
    return t[0].numel() if shape.use_mla else t[0][0].numel()


def test_unwritten_slot_is_reported_not_decoded():
    dev = torch.device("cuda:0")
    shape = KVShape("c4", 2, 8, 128, tokens_per_block=16)
    kv, layout = alloc_paged_cache(shape, 8, dev, "vllm", fill="zeros")
    reg = register_tensors(kv, layout)
    E = reg.chunk_bytes // 2
    slot = chunk_slot_bytes(E)
    pool = torch.zeros(8, 2, 2, slot, dtype=torch.uint8).pin_memory()
    host = HostSide(pool.data_ptr(), 2 * slot, slot, 4 * slot, 8)
    table = torch.zeros(size_table_entries(8, 2, 2, E), dtype=torch.int32).pin_memory()
    status = new_status(dev)
    ids = np.array([1, 2], dtype=np.int64)
    kv_compress(reg, host, table, ids, ids, h2d=True, status=status)        # nothing was ever compressed there
    torch.cuda.synchronize()
    assert decode_status(status) == 16


def test_kvmanager_with_lossless_codec_host_and_ssd(tmp_path):
    from flexkv_b200 import CacheConfig, KVManager
    from flexkv_b200.models import make_model_config
    dev = torch.device("cuda:0")
    shape = KVShape("c5", 3, 8, 128, tokens_per_block=16)
    T, NB, n = 16, 64, 18
    kv, layout = alloc_paged_cache(shape, NB, dev, "vllm", fill="normal", seed=72)
    mgr = KVManager(make_model_config(shape), CacheConfig(tokens_per_block=T, num_cpu_blocks=40, enable_compression=True,
                                                          enable_ssd=True, num_ssd_blocks=96,
                                                          ssd_cache_dir=str(tmp_path)))
    mgr.register_gpu_tensors(kv, layout)
    mgr.start()
    mgr.wait_ready(120)
    try:
        host = mgr.transfer_manager.storage.host
        assert host.quant == "bf16_xp" and host.size_table is not None
        rng = np.random.default_rng(9)
        tok = rng.integers(0, 1000, size=n * T, dtype=np.int64)
        src = rng.permutation(NB)[:n].astype(np.int64)
        slot = np.repeat(src, T) * T + np.tile(np.arange(T), n)
        tid = mgr.put_async(tok, slot)
        assert mgr.wait(tid, completely=True)[tid].status.value == "success"
        saved = [t.clone() for t in kv]
        for rounds, clear in ((0, False), (1, True)):       # host hit, then SSD hit after dropping the host tier
            if clear:
                mgr._clear_cpu_cache()
                host.size_table.zero_()                      # sizes must come back from the SSD table
            for t in kv:
                t.zero_()
            dst = rng.permutation(NB)[:n].astype(np.int64)
            tid = mgr.get_async(tok, np.repeat(dst, T) * T + np.tile(np.arange(T), n))
            r = mgr.wait(tid)[tid]
            assert r.status.value == "success" and int(r.return_mask.sum()) == n * T
            torch.cuda.synchronize()
            si, di = torch.from_numpy(src).to(dev), torch.from_numpy(dst).to(dev)
            for l in range(shape.num_layers):
                assert torch.equal(kv[l][:, di].view(torch.int16), saved[l][:, si].view(torch.int16))
    finally:
        mgr.shutdown()


@pytest.mark.parametrize("shape,spread", [(KVShape("r1", 16, 8, 128, tokens_per_block=16), False),   # two full tiles a chunk
                                          (KVShape("r1", 16, 8, 128, tokens_per_block=16), True),    # some tiles raw
                                          (KVShape("r2", 15, 1, 576, use_mla=True, tokens_per_block=64), False),
                                          (KVShape("r3", 48, 1, 256, tokens_per_block=16), False)])  # 6 KiB rows, one tile a chunk
def test_restore_through_the_copy_engines_matches_the_kernel(shape, spread):
    """Host runs come in as rows of the used bytes, stray blocks by the kernel; a piece whose tiles differ much in
    size stays with the kernel. Tiles beyond the used bytes are never looked at: the slots hold garbage there."""
    dev = torch.device("cuda:0")
    n_run = 70 if shape.num_layers < 48 else 200
    NB = 2 * n_run + 20
    kv, layout = alloc_paged_cache(shape, NB, dev, "vllm", fill="normal", seed=71)
    if not shape.use_mla:
        for t in kv:
            t[0].mul_(torch.exp(torch.randn(t.shape[-1], device=dev)))          # keys pack worse than values
    if spread:
        kv[3].view(torch.int16).random_(-32768, 32767)
    reg = register_tensors(kv, layout)
    E = reg.chunk_bytes // 2
    slot = chunk_slot_bytes(E)
    L, K = shape.num_layers, shape.kv_dim
    pool = torch.full((NB, L * K * slot), 255, dtype=torch.uint8).pin_memory()
    table = torch.zeros(size_table_entries(NB, L, K, E), dtype=torch.int32).pin_memory()
    host = HostSide(pool.data_ptr(), K * slot, slot, L * K * slot, NB)
    rng = np.random.default_rng(6)
    c = np.concatenate([[2], np.arange(5, 5 + n_run), [4, 0], np.arange(8 + n_run, 8 + 2 * n_run)]).astype(np.int64)
    g = rng.permutation(NB)[:c.size].astype(np.int64)
    status = new_status(dev)
    keep = kv_compress(reg, host, table, g, c, h2d=False, num_ctas=80, status=status)
    torch.cuda.synchronize()
    saved = [t.clone() for t in kv]
    for t in kv:
        t.zero_()
    g2 = rng.permutation(NB)[:c.size].astype(np.int64)
    ids = [torch.from_numpy(a.copy()).pin_memory() for a in (g2, c)]
    link = _native.C.CodecLink(0, L, K, slot, 8 << 20)
    link.compress_bf16(make_params(reg, host, *ids, True, status_ptr=status.data_ptr()), table.data_ptr(), L, 80, 160,
                       torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert decode_status(status) == 0 and link.staged_ops == 1
    a, b = torch.from_numpy(g).to(dev), torch.from_numpy(g2).to(dev)
    other = torch.ones(NB, dtype=torch.bool)
    other[g2] = False
    for t, s in zip(kv, saved):
        t, s = (t.unsqueeze(0), s.unsqueeze(0)) if shape.use_mla else (t, s)
        assert torch.equal(t[:, b].view(torch.int16), s[:, a].view(torch.int16))
        assert not bool(t[:, other.to(dev)].view(torch.int16).any())
    # a slot that was never written: every size that is there is restored, the error is reported
    table.view(NB, -1)[c[10], 3] = 0
    link.compress_bf16(make_params(reg, host, *ids, True, status_ptr=status.data_ptr()), table.data_ptr(), L, 80, 160,
                       torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert decode_status(status) == 16


@pytest.mark.parametrize("elems", [1024, 2048, 3072, 4096, 5120])     # 32, 32, 64, 64 and 128 threads per tile
@pytest.mark.parametrize("ctas", [2, 80])
def test_small_chunks_pack_to_the_reference_bytes_and_back(elems, ctas):
    """A chunk of one short tile takes as many threads as it has 64-value pieces; scattered and wild exponents too."""
    dev = torch.device("cuda:0")
    shape = KVShape("s", 3, 1, elems // 8, tokens_per_block=8)
    NB, n = 80, 61
    kv, layout = alloc_paged_cache(shape, NB, dev, "vllm", fill="normal", seed=9)
    kv[1][0].mul_(torch.exp(3 * torch.randn(shape.head_size, device=dev)))            # more than 16 exponents: escapes
    kv[1][1, :NB // 2].view(torch.int16).random_(-32768, 32767)                       # more than 32 exponents, raw tiles
    kv[2][0].zero_()
    reg = register_tensors(kv, layout)
    E = reg.chunk_bytes // 2
    assert E == elems
    slot = chunk_slot_bytes(E)
    L, K = shape.num_layers, shape.kv_dim
    pool = torch.zeros(NB, L, K, slot, dtype=torch.uint8).pin_memory()
    table = torch.zeros(size_table_entries(NB, L, K, E), dtype=torch.int32).pin_memory()
    host = HostSide(pool.data_ptr(), K * slot, slot, L * K * slot, NB)
    rng = np.random.default_rng(2)
    g, c, g2 = (rng.permutation(NB)[:n].astype(np.int64) for _ in range(3))
    status = new_status(dev)
    keep = kv_compress(reg, host, table, g, c, h2d=False, num_ctas=ctas, status=status)
    torch.cuda.synchronize()
    sizes = table.view(NB, L, K)
    saved = [t.clone() for t in kv]
    for i in rng.permutation(n)[:9]:
        for l in range(L):
            for k in range(K):
                want = reference_compress_tile(saved[l][k, int(g[i])].reshape(-1).cpu())
                assert int(sizes[c[i], l, k]) == want.numel()
                assert torch.equal(pool[int(c[i]), l, k, :want.numel()], want)
    for t in kv:
        t.zero_()
    keep += kv_compress(reg, host, table, g2, c, h2d=True, num_ctas=ctas, status=status)
    torch.cuda.synchronize()
    assert decode_status(status) == 0
    a, b = torch.from_numpy(g).to(dev), torch.from_numpy(g2).to(dev)
    for t, s in zip(kv, saved):
        assert torch.equal(t[:, b].view(torch.int16), s[:, a].view(torch.int16))
