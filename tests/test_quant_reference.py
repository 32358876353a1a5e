"""The CPU restatement of the block-scaled fp8 format that the kernels are compared with."""
import pytest
import torch

from flexkv_b200.ops.kv_quant import reference_pack, reference_unpack


@pytest.mark.parametrize("amax", [1e-39, 1.2e-38, 1e-37, 1.3e-36, 5e-36, 5.4e-36, 1e-30, 1.0, 3e38])
def test_zeros_stay_zero_whatever_the_group_holds(amax):
    x = torch.zeros(2, 256, dtype=torch.float64)
    x[:, ::3] = -amax
    x[:, 1::3] = amax / 3
    x = x.to(torch.bfloat16)
    q, s = reference_pack(x)
    y = reference_unpack(q, s)
    tiny = torch.finfo(torch.float32).tiny
    assert bool((s >= tiny).all()) and bool(torch.isfinite(y.float()).all()) and bool((y[x == 0] == 0).all())
    # e4m3 keeps 3 mantissa bits; next to FLT_MIN steps are 2^-9 of it, and what is below it is flushed
    assert bool(((y.double() - x.double()).abs() <= x.double().abs().amax() / 16 + tiny).all())
