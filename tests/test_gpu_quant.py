"""Fused block-scaled FP8 offload against a plain PyTorch fp32 reference of the
same arithmetic: payload bytes and scales bit-exact, restored bf16 bit-exact to
the reference dequantisation, error bounded against the original."""
import numpy as np
import pytest
import torch

from flexkv_b200 import CacheConfig, KVManager, _native
from flexkv_b200.models import KVShape, alloc_paged_cache, make_model_config
from flexkv_b200.ops.kv_copy import HostSide, decode_status, make_params, new_status
from flexkv_b200.ops.kv_quant import kv_quant_fp8, packed_chunk_bytes, reference_pack, reference_unpack
from flexkv_b200.storage.gpu_layout import register_tensors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [KVShape("q1", 3, 8, 128, tokens_per_block=16),       # 16384-element chunks, 2 tiles
                                   KVShape("q2", 2, 1, 576, use_mla=True, tokens_per_block=64),   # 36864: ragged last tile
                                   KVShape("q3", 2, 2, 64, tokens_per_block=8)])       # 1024-element chunks
def test_pack_unpack_match_reference(shape):
    dev = torch.device("cuda:0")
    NB, n = 40, 23
    kv, layout = alloc_paged_cache(shape, NB, dev, "vllm", fill="normal", seed=61)
    # widen the dynamic range and plant exact zeros so scale selection is exercised
    kv[0].mul_(37.0)
    kv[1].view(-1)[:4096].zero_()
    reg = register_tensors(kv, layout)
    E = reg.chunk_bytes // 2
    pc = packed_chunk_bytes(E)
    L, K = shape.num_layers, shape.kv_dim
    pool = torch.zeros(NB, L, K, pc, dtype=torch.uint8).pin_memory()
    host = HostSide(pool.data_ptr(), K * pc, pc, L * K * pc, NB)
    rng = np.random.default_rng(4)
    g = rng.permutation(NB)[:n].astype(np.int64)
    c = rng.permutation(NB)[:n].astype(np.int64)
    status = new_status(dev)
    keep = kv_quant_fp8(reg, host, g, c, h2d=False, num_ctas=7, status=status)
    torch.cuda.synchronize()
    assert decode_status(status) == 0
    gi = torch.from_numpy(g).to(dev)
    for l in range(L):
        for k in range(K):
            x = (kv[l][gi] if shape.use_mla else kv[l][k][gi]).reshape(n, E)
            want_q, want_s = reference_pack(x)
            got = pool[torch.from_numpy(c), l, k]
            assert torch.equal(got[:, :E], want_q.cpu()), (l, k)
            assert torch.equal(got[:, E:].contiguous().view(torch.float32), want_s.cpu()), (l, k)
    saved = [t.clone() for t in kv]
    for t in kv:
        t.zero_()
    g2 = rng.permutation(NB)[:n].astype(np.int64)
    keep += kv_quant_fp8(reg, host, g2, c, h2d=True, num_ctas=5, status=status)
    torch.cuda.synchronize()
    assert decode_status(status) == 0
    g2i = torch.from_numpy(g2).to(dev)
    for l in range(L):
        for k in range(K):
            orig = (saved[l][gi] if shape.use_mla else saved[l][k][gi]).reshape(n, E)
            q, s = reference_pack(orig)
            want = reference_unpack(q, s)
            got = (kv[l][g2i] if shape.use_mla else kv[l][k][g2i]).reshape(n, E)
            assert torch.equal(got.view(torch.int16), want.view(torch.int16)), (l, k)
            # e4m3 keeps 3 mantissa bits: relative error of a group is bounded by 2^-4 of its amax
            err = (got.float() - orig.float()).abs().reshape(n, -1, 128).amax(-1)
            bound = orig.float().abs().reshape(n, -1, 128).amax(-1) / 16 + 1e-30
            assert bool((err <= bound).all())


@pytest.mark.parametrize("elems", [512, 1536, 2048, 2560, 4096, 4608])       # 64, 128 and 256 threads per tile
@pytest.mark.parametrize("ctas", [3, 48])
def test_small_chunks_pack_to_the_reference_bytes_and_back(elems, ctas):
    dev = torch.device("cuda:0")
    shape = KVShape("s", 3, 1, elems // 8, tokens_per_block=8)
    NB, n = 90, 71
    kv, layout = alloc_paged_cache(shape, NB, dev, "vllm", fill="normal", seed=64)
    # scales over the whole range of bf16, so that quotients meet rounding boundaries, zeros and saturation
    kv[0].mul_(torch.exp(12 * torch.randn(kv[0].shape[:-1], device=dev)).unsqueeze(-1).to(torch.bfloat16))
    kv[1][0].copy_((torch.randint(-64, 65, kv[1][0].shape, device=dev) * 7).to(torch.bfloat16))      # exact halves
    kv[2][1].zero_()
    reg = register_tensors(kv, layout)
    E = reg.chunk_bytes // 2
    assert E == elems
    pc = packed_chunk_bytes(E)
    L, K = shape.num_layers, shape.kv_dim
    pool = torch.zeros(NB, L, K, pc, dtype=torch.uint8).pin_memory()
    host = HostSide(pool.data_ptr(), K * pc, pc, L * K * pc, NB)
    rng = np.random.default_rng(4)
    g, c, g2 = (rng.permutation(NB)[:n].astype(np.int64) for _ in range(3))
    status = new_status(dev)
    keep = kv_quant_fp8(reg, host, g, c, h2d=False, num_ctas=ctas, status=status)
    torch.cuda.synchronize()
    gi, gi2, ci = torch.from_numpy(g).to(dev), torch.from_numpy(g2).to(dev), torch.from_numpy(c)
    want = {}
    for l in range(L):
        for k in range(K):
            q, s = want[l, k] = reference_pack(kv[l][k][gi].reshape(n, E))
            got = pool[ci, l, k]
            assert torch.equal(got[:, :E], q.cpu()), (l, k)
            assert torch.equal(got[:, E:].contiguous().view(torch.float32), s.cpu()), (l, k)
    for t in kv:
        t.zero_()
    keep += kv_quant_fp8(reg, host, g2, c, h2d=True, num_ctas=ctas, status=status)
    torch.cuda.synchronize()
    assert decode_status(status) == 0
    for l in range(L):
        for k in range(K):
            assert torch.equal(kv[l][k][gi2].reshape(n, E).view(torch.int16), reference_unpack(*want[l, k]).view(torch.int16))


@pytest.mark.parametrize("elems", [512, 4096, 8192])                        # 64, 128 and 256 threads per tile
def test_groups_of_tiny_values(elems):
    """Groups whose largest value lies where amax / 448 is no normal float any more, on both sides of the line
    (448 * FLT_MIN = 5.27e-36) and around the smallest normal value, with zeros and values far below it among them."""
    dev = torch.device("cuda:0")
    shape = KVShape("t", 1, 1, elems // 8, tokens_per_block=8)
    amax = torch.tensor([1e-39, 1.1e-38, 1.2e-38, 1e-37, 1.3e-36, 1.4e-36, 5e-36, 5.4e-36, 1e-35, 1e-33])
    n = NB = len(amax)
    kv, layout = alloc_paged_cache(shape, NB, dev, "vllm", fill="normal", seed=65)
    for t in kv[0]:
        x = t.float().reshape(NB, -1)
        x = x.clamp(-1, 1) * (torch.rand_like(x) < 0.7) * 10.0 ** -(torch.rand_like(x) < 0.2).float().mul(3)
        x[:, ::64] = -1
        t.copy_((x.double() * amax.to(dev).double().unsqueeze(-1)).reshape(t.shape).to(torch.bfloat16))
    src = [t.reshape(NB, elems).clone() for t in kv[0]]
    reg = register_tensors(kv, layout)
    pc = packed_chunk_bytes(elems)
    pool = torch.zeros(NB, 1, 2, pc, dtype=torch.uint8).pin_memory()
    host = HostSide(pool.data_ptr(), 2 * pc, pc, 2 * pc, NB)
    ids = np.arange(n, dtype=np.int64)
    keep = kv_quant_fp8(reg, host, ids, ids, h2d=False)
    torch.cuda.synchronize()
    for t in kv:
        t.fill_(1)
    keep += kv_quant_fp8(reg, host, ids, ids, h2d=True)
    torch.cuda.synchronize()
    for k in range(2):
        q, s = reference_pack(src[k])
        assert torch.equal(pool[:, 0, k, :elems], q.cpu())
        assert torch.equal(pool[:, 0, k, elems:].contiguous().view(torch.float32), s.cpu())
        got = kv[0][k].reshape(NB, elems)
        assert torch.equal(got.view(torch.int16), reference_unpack(q, s).view(torch.int16))
        assert bool((got[src[k] == 0] == 0).all())


@pytest.mark.parametrize("shape", [KVShape("l1", 16, 8, 128, tokens_per_block=16),
                                   KVShape("l2", 15, 1, 576, use_mla=True, tokens_per_block=64)])   # ragged last tile
def test_copy_engine_route_moves_the_same_bytes(shape):
    """Host runs through the staging buffer, stray host blocks by the kernel, in one op; against the kernel alone."""
    dev = torch.device("cuda:0")
    n_run = 70
    NB = 2 * n_run + 20
    kv, layout = alloc_paged_cache(shape, NB, dev, "vllm", fill="normal", seed=63)
    reg = register_tensors(kv, layout)
    pc = packed_chunk_bytes(reg.chunk_bytes // 2)
    L, K = shape.num_layers, shape.kv_dim
    pool = torch.zeros(NB, L * K * pc, dtype=torch.uint8).pin_memory()
    rng = np.random.default_rng(5)
    c = np.concatenate([[2], np.arange(5, 5 + n_run), [4, 0], np.arange(8 + n_run, 8 + 2 * n_run)]).astype(np.int64)
    g = rng.permutation(NB)[:c.size].astype(np.int64)
    g2 = rng.permutation(NB)[:c.size].astype(np.int64)
    host = HostSide(pool.data_ptr(), K * pc, pc, L * K * pc, NB)
    status = new_status(dev)
    keep = kv_quant_fp8(reg, host, g, c, h2d=False, status=status)
    torch.cuda.synchronize()
    want = pool.clone()
    assert int(want.count_nonzero()) > 0
    for h2d, pages in ((False, g), (True, g2)):
        link = _native.C.CodecLink(0, L, K, pc)
        ids = [torch.from_numpy(a.copy()).pin_memory() for a in (pages, c)]
        if h2d:
            saved = [t.clone() for t in kv]
            keep += kv_quant_fp8(reg, host, pages, c, h2d=True, status=status)
            torch.cuda.synchronize()
            restored = [t.clone() for t in kv]
            for t, s in zip(kv, saved):
                t.copy_(s)
        else:
            pool.zero_()
        link.quant_fp8(make_params(reg, host, *ids, h2d, status_ptr=status.data_ptr()), 32,
                       torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert link.staged_ops == 1 and decode_status(status) == 0
        if h2d:
            assert all(torch.equal(t.view(torch.int16), r.view(torch.int16)) for t, r in zip(kv, restored))
        else:
            assert torch.equal(pool, want)


def test_kvmanager_with_fp8_host_pool_halves_the_host_block():
    dev = torch.device("cuda:0")
    shape = KVShape("q4", 4, 8, 128, tokens_per_block=16)
    T, NB, n = 16, 64, 20
    kv, layout = alloc_paged_cache(shape, NB, dev, "vllm", fill="normal", seed=62)
    mgr = KVManager(make_model_config(shape), CacheConfig(tokens_per_block=T, num_cpu_blocks=48,
                                                          offload_quant="fp8_e4m3"))
    mgr.register_gpu_tensors(kv, layout)
    mgr.start()
    mgr.wait_ready(120)
    try:
        host = mgr.transfer_manager.storage.host
        assert host.block_bytes == shape.block_bytes // 2 + shape.block_bytes // 64
        rng = np.random.default_rng(8)
        tok = rng.integers(0, 1000, size=n * T, dtype=np.int64)
        src = rng.permutation(NB)[:n].astype(np.int64)
        slot = np.repeat(src, T) * T + np.tile(np.arange(T), n)
        tid = mgr.put_async(tok, slot)
        assert mgr.wait(tid, completely=True)[tid].status.value == "success"
        saved = [t.clone() for t in kv]
        for t in kv:
            t.zero_()
        dst = rng.permutation(NB)[:n].astype(np.int64)
        tid = mgr.get_async(tok, np.repeat(dst, T) * T + np.tile(np.arange(T), n))
        assert mgr.wait(tid)[tid].status.value == "success"
        torch.cuda.synchronize()
        si, di = torch.from_numpy(src).to(dev), torch.from_numpy(dst).to(dev)
        for l in range(shape.num_layers):
            orig = saved[l][:, si].reshape(2, n, -1)
            q, s = reference_pack(orig)
            assert torch.equal(kv[l][:, di].reshape(2, n, -1).view(torch.int16), reference_unpack(q, s).view(torch.int16))
    finally:
        mgr.shutdown()
