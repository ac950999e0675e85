"""moe_sum_reduce and moe_gather_sum_reduce around the sizes of their vector kernel: columns that are
not whole blocks or warps, top-k around the load batch.  The sums run in ascending k in fp32, as in the
check (a fused multiply-add may round once where the check rounds twice)."""

import pytest
import torch

import xkernels_b200 as xkb
from xkernels_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [8, 24, 256, 2048, 2056, 7168, 12])
@pytest.mark.parametrize("top_k", [0, 1, 4, 7, 8, 9, 17])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_sum_reduce(H, top_k, dtype, cuda_device):
    g = torch.Generator(device=cuda_device).manual_seed(H + top_k)
    y = torch.randn(5, top_k, H, generator=g, device=cuda_device).to(dtype)
    w = torch.randn(5, top_k, generator=g, device=cuda_device)
    want = (y.double() * w.double().unsqueeze(-1)).sum(1)
    mag = (y.double() * w.double().unsqueeze(-1)).abs().sum(1)
    got = xkb.moe_sum_reduce(y, w).double()
    # top_k roundings of 2^-24 of the running sum, and the rounding to the output's type (bf16: 8 significant
    # bits, half a unit in the last place is at most 2^-8 of the value; fp32: 2^-24)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -24
    assert bool(((got - want).abs() <= (top_k + 1) * 2.0 ** -24 * mag + eps * want.abs() * 1.01).all())


@pytest.mark.parametrize("H", [4, 8, 2048, 2056])
@pytest.mark.parametrize("k", [1, 3, 8])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gather_sum_reduce(H, k, dtype, cuda_device):
    g = torch.Generator(device=cuda_device).manual_seed(H + k)
    rows = torch.randn(11, H, generator=g, device=cuda_device)
    index = torch.randint(-3, 11, (7, k), generator=g, device=cuda_device, dtype=torch.int32)
    at = index.long()
    picked = rows[at.clamp(min=0)].double() * (at >= 0).unsqueeze(-1)
    got = ops.moe_gather_sum_reduce(rows, index, None, out_dtype=dtype).double()
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -24
    assert bool(((got - picked.sum(1)).abs() <= k * 2.0 ** -24 * picked.abs().sum(1) + eps * picked.sum(1).abs() * 1.01).all())


@pytest.mark.parametrize("H", [8, 24, 64, 128, 136, 1024])
@pytest.mark.parametrize("M", [1183, 1184, 1185, 151553])
def test_narrow_rows_share_a_block(M, H, cuda_device):
    """Many tokens of narrow rows: several per block from twice 592 tokens on, up to a whole block of them."""
    if M * H > 2 ** 25:
        M = 20001
    g = torch.Generator(device=cuda_device).manual_seed(M + H)
    y = torch.randn(M, 3, H, generator=g, device=cuda_device)
    w = torch.randn(M, 3, generator=g, device=cuda_device)
    term = y.double() * w.double().unsqueeze(-1)
    bound = 4 * 2.0 ** -24 * term.abs().sum(1) + 2.0 ** -24 * 1.01 * term.sum(1).abs()
    assert bool(((xkb.moe_sum_reduce(y, w).double() - term.sum(1)).abs() <= bound).all())
    rows, index = y.reshape(-1, H), torch.randint(-2, 3 * M, (M, 3), generator=g, device=cuda_device, dtype=torch.int32)
    picked = rows[index.long().clamp(min=0)].double() * (index >= 0).unsqueeze(-1)
    got = ops.moe_gather_sum_reduce(rows, index, None, out_dtype=torch.float32).double()
    assert bool(((got - picked.sum(1)).abs() <= 4 * 2.0 ** -24 * picked.abs().sum(1)).all())
