"""The work a serving engine hands to flexkv_b200, as cases that can be timed.

A case is one engine-side situation: requests whose KV leaves the GPU for the host pool and comes back
(``put_get``), a prefix hit that is restored (``get``), an offload and a restore in flight together (``duplex``),
a restore that signals layer by layer (``layerwise``), or the block keys of prompts that live on the GPU
(``hash``). All but the last go through ``KVManager`` with an engine's paged cache registered in place: random,
non-contiguous pages, lengths that are not multiples of the page, the KV shapes of ``flexkv_b200.models``.

Fields: ``kind``; ``kv`` (name of the KV shape); ``codec`` of the host pool (``none`` | ``bf16_xp`` lossless |
``fp8_e4m3``); ``requests`` and ``tokens`` (longest request; with several requests the others are shorter and
ragged); ``block`` (tokens per page of a ``hash`` case).
"""
from __future__ import annotations

import dataclasses
import math
import random

import numpy as np
import torch

from flexkv_b200 import CacheConfig, KVManager
from flexkv_b200.common.config import GLOBAL_CONFIG_FROM_ENV
from flexkv_b200.common.storage import KVCacheLayout, KVCacheLayoutType
from flexkv_b200.models import get_shape, make_model_config
from flexkv_b200.ops.kv_hash import gpu_block_hashes

VOCAB = 128256
PASS_STEP = 131072        # added to every token id from one pass to the next: a prompt never seen before
MOST_BYTES = 2 << 30      # KV of one direction of the largest case


def listed():
    return [
        # one page finished in decode, parked and picked up again: latency of the control plane and two launches
        dict(name="turn_16_raw", kind="put_get", kv="llama3-8b", codec="none", requests=1, tokens=16),
        # a short chat turn with a partly filled last page
        dict(name="turn_200_lossless", kind="put_get", kv="llama3-8b", codec="bf16_xp", requests=1, tokens=200),
        # an 8K-token prompt with the default configuration: offload, then restore
        dict(name="prompt_8k_raw", kind="put_get", kv="llama3-8b", codec="none", requests=1, tokens=8192),
        # the prefix hit behind the benchmark's p50 latency of an 8K-token get
        dict(name="hit_8k_lossless", kind="get", kv="llama3-8b", codec="bf16_xp", requests=1, tokens=8192),
        # throughput: a batch of ragged prompts offloaded and restored as one launch each
        dict(name="batch_lossless", kind="put_get", kv="llama3-8b", codec="bf16_xp", requests=8, tokens=4096),
        # the block-scaled fp8 host format on a deeper model
        dict(name="batch_fp8", kind="put_get", kv="qwen3-32b", codec="fp8_e4m3", requests=4, tokens=1500),
        # latent (MLA) cache: one plane, 64-token pages, chunks that are no multiple of the codec's tile
        dict(name="mla_4k_lossless", kind="put_get", kv="deepseek-v3", codec="bf16_xp", requests=1, tokens=4100),
        # packed NVFP4 cache moved as bytes
        dict(name="hit_nvfp4_raw", kind="get", kv="qwen3-32b-nvfp4", codec="none", requests=4, tokens=1500),
        # one rank of an eight-way tensor-parallel SGLang deployment: 160 tensors, one head, 4 KiB chunks
        dict(name="tp8_rank_raw", kind="put_get", kv="llama3-70b-rank", codec="none", requests=1, tokens=3000),
        # an engine that offloads finished requests while it restores others
        dict(name="duplex_lossless", kind="duplex", kv="llama3-8b", codec="bf16_xp", requests=2, tokens=2048),
        # a batched prefix hit restored layer by layer under the forward pass
        dict(name="layerwise_raw", kind="layerwise", kv="llama3-8b", codec="none", requests=4, tokens=1100),
        # block keys of a batch of prompts whose token ids are on the GPU
        dict(name="hash_64x4k", kind="hash", requests=64, tokens=4096, block=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.1:
        return dict(kind="hash", requests=_log_int(rng, 1, 64), tokens=_log_int(rng, 64, 32768),
                    block=rng.choice([1, 16, 64]))
    kind = rng.choice(["put_get", "put_get", "put_get", "get", "get", "duplex", "layerwise"])
    kv = rng.choice(["llama3-8b", "llama3-8b", "qwen3-32b", "deepseek-v3", "qwen3-32b-nvfp4", "llama3-70b-rank"])
    if kind == "layerwise" or kv == "qwen3-32b-nvfp4":
        codec = "none"
    else:
        codec = rng.choice(["none", "bf16_xp", "bf16_xp", "fp8_e4m3"])
    shape = _shape(kv)
    requests = rng.choice([1, 1, 2, 3, 5, 8])
    most = MOST_BYTES // (2 if kind == "duplex" else 1) // (shape.bytes_per_token * requests)
    tokens = _log_int(rng, shape.tokens_per_block, min(16384, most))
    return dict(kind=kind, kv=kv, codec=codec, requests=requests, tokens=tokens)


# ---------------------------------------------------------------- sizes

def _shape(name):
    if name == "llama3-70b-rank":      # what one of eight tensor-parallel ranks holds of llama3-70b
        return dataclasses.replace(get_shape("llama3-70b"), num_kv_heads=1)
    return get_shape(name)


def _lengths(case):
    """Tokens of every request: the longest first, the others between half of it and all of it."""
    n, t = case["requests"], case["tokens"]
    r = random.Random(1000003 * n + t)
    floor = case.get("block", 1) if case["kind"] == "hash" else _shape(case["kv"]).tokens_per_block
    return [t] + [max(min(t, floor), t - r.randrange(t // 2 + 1)) for _ in range(n - 1)]


def _blocks(case):
    T = _shape(case["kv"]).tokens_per_block
    return sum(n // T for n in _lengths(case))


def work(case):
    """Bytes one pass cannot do without: the KV read on one side and written on the other, once per direction; on the
    host side what the format stores (lossless: 0.66 of the raw bytes, the entropy of unit-normal bf16)."""
    if case["kind"] == "hash":
        lens = _lengths(case)
        return {"bytes": 8 * (sum(lens) + sum(n // case["block"] for n in lens)), "flops": 0}
    shape = _shape(case["kv"])
    raw = _blocks(case) * shape.block_bytes
    host = {"none": 1.0, "bf16_xp": 0.66, "fp8_e4m3": 0.5 + 4 / 256}[case["codec"]] * raw
    directions = 2 if case["kind"] in ("put_get", "duplex") else 1
    return {"bytes": directions * (raw + host), "flops": 0}


def tolerance(case):
    """Bytes and keys are exact, lossless included. fp8: the round trip in 64-bit arithmetic lies 2.6e-4 (2-norm)
    from the one in 32-bit arithmetic, from values that sit on a rounding boundary."""
    if case["kind"] != "hash" and case["codec"] == "fp8_e4m3":
        return {"rel": 1e-3}
    return "exact"


# ---------------------------------------------------------------- inputs

def _alloc_cache(shape, num_blocks, dev):
    """The engine's paged cache as views of one allocation, in the shape's engine layout."""
    L, T, H, D, K = shape.num_layers, shape.tokens_per_block, shape.num_kv_heads, shape.head_size, shape.kv_dim
    if shape.use_mla:
        base = torch.zeros(L, num_blocks, T, H * D, dtype=shape.dtype, device=dev)
    elif shape.engine_layout == "sglang":
        base = torch.zeros(2 * L, num_blocks, T, H, D, dtype=shape.dtype, device=dev)
    else:
        base = torch.zeros(L, 2, num_blocks, T, H, D, dtype=shape.dtype, device=dev)
    layout = KVCacheLayout(KVCacheLayoutType.LAYERFIRST, L, num_blocks, T, H, D, is_mla=shape.use_mla,
                           kv_dim_override=K)
    return base, list(base.unbind(0)), layout


def _fill(shape, base, pages, gen):
    """KV as models produce it: keys with a scale per channel (a few channels far out) and per layer, values closer
    to unit normal. Packed 4-bit caches are uniform bytes."""
    dev = base.device
    n = int(pages.numel())
    if shape.dtype == torch.uint8:
        for t in base.unbind(0):
            t[:, pages] = torch.randint(0, 256, (t.shape[0], n) + tuple(t.shape[2:]), dtype=torch.uint8, device=dev,
                                        generator=gen)
        return
    planes = base.unbind(0) if shape.use_mla or shape.engine_layout == "sglang" else base.flatten(0, 1).unbind(0)
    L = shape.num_layers
    for i, t in enumerate(planes):                                  # t: [num_blocks, T, ..., channels]
        if shape.use_mla:
            is_key = True
        else:
            is_key = i < L if shape.engine_layout == "sglang" else i % 2 == 0
        x = torch.randn((n,) + tuple(t.shape[1:]), dtype=torch.bfloat16, device=dev, generator=gen)
        width = tuple(t.shape[2:])
        scale = torch.exp(0.25 * torch.randn((), device=dev, generator=gen)).expand(width)
        if is_key:
            scale = scale * torch.exp(0.4 * torch.randn(width, device=dev, generator=gen))
            scale = torch.where(torch.rand(width, device=dev, generator=gen) < 0.02, scale * 8, scale)
        t[pages] = x * scale.to(torch.bfloat16)


def _slots(pages, T):
    """Token slots of the full pages of a request (a partly filled last page is neither stored nor restored)."""
    return np.repeat(pages, T) * T + np.tile(np.arange(T, dtype=np.int64), len(pages))


class _Session:
    """A manager with the engine's cache registered; shut down with the state that holds it."""

    def __init__(self, model, config, tensors, layout, layerwise):
        before = GLOBAL_CONFIG_FROM_ENV.enable_layerwise_transfer
        GLOBAL_CONFIG_FROM_ENV.enable_layerwise_transfer = layerwise
        try:
            self.mgr = KVManager(model, config)
            self.mgr.register_gpu_tensors(tensors, layout)
            self.mgr.start()
            self.mgr.wait_ready(120)
        finally:
            GLOBAL_CONFIG_FROM_ENV.enable_layerwise_transfer = before

    def __del__(self):
        mgr = getattr(self, "mgr", None)
        if mgr is not None:
            mgr.shutdown()


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed)
    lens = _lengths(case)
    if case["kind"] == "hash":
        seqs = [torch.randint(0, VOCAB, (n,), dtype=torch.int64, device=dev, generator=gen) for n in lens]
        return {"case": case, "seqs": seqs}
    shape = _shape(case["kv"])
    T = shape.tokens_per_block
    counts = [n // T for n in lens]
    total = sum(counts)
    num_pages = 2 * total + 8
    base, tensors, layout = _alloc_cache(shape, num_pages, dev)
    perm = rng.permutation(num_pages).astype(np.int64)
    src, dst = perm[:total], perm[total:2 * total]
    _fill(shape, base, torch.from_numpy(src).to(dev), gen)
    torch.cuda.synchronize()
    # room for the working set twice over and some: offloads of new prompts evict old ones once it is full
    config = CacheConfig(tokens_per_block=T, num_cpu_blocks=3 * total + 64,
                         enable_compression=case["codec"] == "bf16_xp",
                         offload_quant="fp8_e4m3" if case["codec"] == "fp8_e4m3" else "none")
    session = _Session(make_model_config(shape), config, tensors, layout, case["kind"] == "layerwise")
    ends = np.cumsum([0] + counts)

    def slots_of(pages):
        return [_slots(pages[a:b], T) for a, b in zip(ends[:-1], ends[1:])]

    state = {"case": case, "session": session, "base": base, "passes": 0,
             "tokens": [rng.integers(0, VOCAB, size=n, dtype=np.int64) for n in lens],
             "src_slots": slots_of(src), "dst_slots": slots_of(dst)}
    if case["kind"] != "put_get":
        # the prefix that the passes hit is in the host pool already
        state["hit_tokens"] = [rng.integers(0, VOCAB, size=n, dtype=np.int64) for n in lens]
        _put(session.mgr, state["hit_tokens"], state["src_slots"])
    return state


# ---------------------------------------------------------------- one pass

def _launch_put(mgr, prompts, slots):
    ids = [mgr.put_match(t)[0] for t in prompts]
    return mgr.launch(ids, slots, as_batch=len(ids) > 1)


def _launch_get(mgr, prompts, slots, layerwise=False):
    ids, masks = [], []
    for t in prompts:
        task, mask = mgr.get_match(t)
        ids.append(task)
        masks.append(mask)
    launched = mgr.launch(ids, slots, as_batch=layerwise or len(ids) > 1, layerwise_transfer=layerwise)
    return launched, masks


def _finish(mgr, ids, completely=False):
    for task, answer in mgr.wait(ids, timeout=60, completely=completely).items():
        if answer.status.value != "success":
            raise RuntimeError(f"task {task}: {answer.status}")


def _put(mgr, prompts, slots):
    _finish(mgr, _launch_put(mgr, prompts, slots), completely=True)


def run(state):
    case = state["case"]
    if case["kind"] == "hash":
        return gpu_block_hashes(state["seqs"], case["block"])
    mgr = state["session"].mgr
    if case["kind"] in ("put_get", "duplex"):
        state["passes"] += 1
        new = [t + state["passes"] * PASS_STEP for t in state["tokens"]]
    if case["kind"] == "put_get":
        _put(mgr, new, state["src_slots"])
        ids, masks = _launch_get(mgr, new, state["dst_slots"])
        _finish(mgr, ids)
    elif case["kind"] == "duplex":
        out = _launch_put(mgr, new, state["src_slots"])
        ids, masks = _launch_get(mgr, state["hit_tokens"], state["dst_slots"])
        _finish(mgr, ids)
        _finish(mgr, out, completely=True)
    else:
        ids, masks = _launch_get(mgr, state["hit_tokens"], state["dst_slots"], layerwise=case["kind"] == "layerwise")
        _finish(mgr, ids)
    return {"kv": state["base"], "hit": masks}
