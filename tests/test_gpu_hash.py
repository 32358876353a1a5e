"""GPU batched block keys against the host hasher (which is itself pinned to canonical XXH64
vectors in test_hash.py): ragged batches, namespaces, block sizes that do and do not align with
the 32-byte stripes."""
import numpy as np
import pytest
import torch

from flexkv_b200.common.block import hash_blocks
from flexkv_b200.ops.kv_hash import gpu_block_hashes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tpb", [1, 3, 4, 16, 64])
@pytest.mark.parametrize("namespace", [None, ["lora-7"], ["tenant", "a", "salt123"]])
def test_matches_host_hasher(tpb, namespace):
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(tpb)
    lens = [0, 1, 2, 5, 31, 64, 257, 1000, 8192, 4099]
    seqs = [rng.integers(-2**62, 2**62, size=n, dtype=np.int64) for n in lens]
    got = gpu_block_hashes([torch.from_numpy(s).to(dev) for s in seqs], tpb, namespace)
    torch.cuda.synchronize()
    for s, g in zip(seqs, got):
        want = hash_blocks(s, tpb, namespace)
        assert g.cpu().numpy().view(np.uint64).tolist() == want.tolist()


def test_large_batch_is_consistent():
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(0)
    seqs = [rng.integers(0, 128256, size=2048, dtype=np.int64) for _ in range(300)]
    got = gpu_block_hashes([torch.from_numpy(s).to(dev) for s in seqs], 16)
    torch.cuda.synchronize()
    for i in (0, 1, 150, 299):
        assert got[i].cpu().numpy().view(np.uint64).tolist() == hash_blocks(seqs[i], 16).tolist()


@pytest.mark.parametrize("nseq,lens", [(3, (1024, 1025, 1023)), (128, (2047, 2048, 2050)), (129, (1027, 3)),
                                       (900, (129, 127, 4100))])
@pytest.mark.parametrize("tpb,namespace", [(1, None), (16, ["x"]), (64, ["tenant" * 50])])
def test_segment_edges_and_both_forms(nseq, lens, tpb, namespace):
    """Lengths around the segment size of either kernel form (one and eight sequences per CTA), sequence counts on
    both sides of the list form's limit and of the change of form, prefixes on both sides of the inline limit; an
    empty sequence among them, and a stream of its own."""
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(nseq + tpb)
    seqs = [rng.integers(-2**62, 2**62, size=lens[i % len(lens)] if i != 1 else 0, dtype=np.int64) for i in range(nseq)]
    got = gpu_block_hashes([torch.from_numpy(s).to(dev) for s in seqs], tpb, namespace, stream=torch.cuda.Stream(dev))
    torch.cuda.synchronize()
    for i in sorted({0, 1, 2, nseq // 2, nseq - 2, nseq - 1}):
        assert got[i].cpu().numpy().view(np.uint64).tolist() == hash_blocks(seqs[i], tpb, namespace).tolist()


@pytest.mark.parametrize("count", [2, 200])
def test_host_tensor_among_the_sequences_is_refused(count):
    dev = torch.device("cuda:0")
    seqs = [torch.arange(64, device=dev) for _ in range(count)]
    seqs[-1] = torch.arange(64)
    with pytest.raises(ValueError):
        gpu_block_hashes(seqs, 16)


@pytest.mark.parametrize("count", [5, 130])
def test_side_stream_reads_converted_inputs(count):
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(count)
    full = [rng.integers(0, 128256, size=4096 + i, dtype=np.int64) for i in range(count)]
    seqs = [torch.from_numpy(f).to(dev) for f in full]
    seqs = [t.to(torch.int32) if i % 2 else t[::2] for i, t in enumerate(seqs)]
    side = torch.cuda.Stream(dev)
    torch.cuda._sleep(2_000_000)            # a millisecond of work in front of the conversions
    got = gpu_block_hashes(seqs, 16, stream=side)
    side.synchronize()
    for i, (f, g) in enumerate(zip(full, got)):
        assert g.cpu().numpy().view(np.uint64).tolist() == hash_blocks(f if i % 2 else f[::2].copy(), 16).tolist()
