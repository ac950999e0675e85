"""The router's loads: pieces of two or four neighbouring logits where E and the base address allow them, one by one
elsewhere; expert counts around those that fill the lanes.  Ids exact (few distinct logits, so that ties cross pieces and
lanes), weights within fp32 round-off of the oracle."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("offset", [0, 1, 2, 4])      # logits between the base and a 16-byte boundary
@pytest.mark.parametrize("E", [2, 31, 48, 64, 65, 96, 128, 129, 192, 256, 260, 383, 384, 512, 1000, 1024])
def test_loads(E, offset, dtype, cuda_device):
    M, topk = 9, min(8, E)
    x = (torch.randn(M, E, generator=torch.Generator().manual_seed(E)) * 3).round().div(2).to(dtype)
    buf = torch.empty(M * E + 8, dtype=dtype, device=cuda_device)
    view = buf[offset:offset + M * E].view(M, E)
    view.copy_(x)
    want_w, want_ids = oracle.topk_softmax(x, topk, True)
    w, ids = xkb.topk_softmax(view, topk, True)
    assert torch.equal(ids.cpu(), want_ids)
    assert bool(((w.cpu() - want_w).abs() <= 1e-6).all())
