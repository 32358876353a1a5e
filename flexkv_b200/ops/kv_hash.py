"""Batched block keys on the GPU (``csrc/kernels/kv_hash.cu``): cumulative streaming XXH64 over
int64 token ids, bit-identical to the host hasher. Worth it for token ids that already live on
the device or for thousands of long sequences at once; a single request is faster on the host."""
from __future__ import annotations

from typing import List, Optional, Sequence

import numpy as np
import torch

from .. import _native
from ..common.block import namespace_prefix


def gpu_block_hashes(seqs: Sequence[torch.Tensor], tokens_per_block: int, namespace: Optional[List[str]] = None,
                     stream: Optional[torch.cuda.Stream] = None) -> List[torch.Tensor]:
    """``seqs``: int64 CUDA tensors (one per sequence, same device; ``ValueError`` otherwise). Returns one uint64-valued
    int64 CUDA tensor of block keys per sequence (view with ``.view(torch.uint64)`` or copy to numpy).

    With a ``stream`` of its own the keys are computed there, behind what the current stream holds. Several sequences
    are copied first, in the order of the current stream, which may then overwrite them; a single one is read where it
    is and has to stay until ``stream`` has passed the call."""
    if not seqs:
        return []
    # the kernel reads these addresses: memory of the host or of another GPU must not get there
    where = [t.get_device() for t in seqs]
    if where.count(where[0]) != len(where) or not seqs[0].is_cuda:
        raise ValueError("gpu_block_hashes: every sequence must be a CUDA tensor on the device of the first")
    dev = seqs[0].device
    C = _native.C
    current = torch.cuda.current_stream(dev)
    s = current if stream is None else stream
    side = stream is not None and stream != current
    lens = [t.numel() for t in seqs]
    nblk = [n // tokens_per_block for n in lens]
    ns = namespace_prefix(namespace)
    out = torch.empty(sum(nblk), dtype=torch.int64, device=dev)
    if len(seqs) <= C.HASH_LIST_SEQS and (ns is None or ns.size <= C.HASH_LIST_NS) and max(lens) < 2**31:
        # addresses, lengths and prefix travel in the launch parameters; on the current stream the sequences are read
        # where they are
        i64 = torch.int64
        if side and len(seqs) > 1:
            seqs = list(torch.cat([t.reshape(-1).to(i64) for t in seqs]).split(lens))
        else:
            seqs = [t if t.dtype is i64 and t.is_contiguous() else t.to(i64).contiguous() for t in seqs]
        if side:
            s.wait_stream(current)          # behind the copies
        C.kv_block_hashes_list([t.data_ptr() for t in seqs], lens, int(tokens_per_block),
                               b"" if ns is None else ns.astype(np.uint8).tobytes(), out.data_ptr(), s.cuda_stream)
        if side:
            for t in seqs + [out]:
                t.record_stream(s)
        return list(out.split(nblk))
    flat = torch.cat([t.reshape(-1) for t in seqs]).to(torch.int64)
    offs = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int64, device=dev)
    ooffs = torch.tensor(np.concatenate([[0], np.cumsum(nblk)]), dtype=torch.int64, device=dev)
    ns_t = torch.from_numpy(np.ascontiguousarray(ns, dtype=np.int64)).to(dev) if ns is not None and len(ns) else None
    if side:
        s.wait_stream(current)              # behind the concatenation and the uploads
    C.kv_block_hashes(flat.data_ptr(), offs.data_ptr(), len(seqs), int(tokens_per_block),
                      ns_t.data_ptr() if ns_t is not None else 0, int(ns_t.numel()) if ns_t is not None else 0,
                      out.data_ptr(), ooffs.data_ptr(), s.cuda_stream)
    if side:
        # the temporaries and the keys stay alive until the stream has passed the launch
        for t in (flat, offs, ooffs, ns_t, out):
            if t is not None:
                t.record_stream(s)
    return list(out.split(nblk))
