"""Rows whose live logits are neighbours, as a router leaves them that masks all groups of experts but a few, and sorted
rows: the pieces of neighbouring logits that a lane of the router holds, at every number of experts per lane, with and
without pieces (E odd, a base off its boundary).  Few distinct logits, so that ties cross pieces and lanes.  Ids
exact, weights within fp32 round-off of the oracle."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("E,groups,live", [(40, 5, 2), (128, 8, 2), (130, 13, 4), (132, 11, 3), (256, 8, 1), (256, 8, 4), (260, 13, 2),
                                           (384, 8, 2), (388, 4, 1), (512, 8, 1), (516, 12, 2), (1024, 16, 1), (1000, 10, 2), (257, 257, 40)])
def test_live_groups(E, groups, live, offset, dtype, cuda_device):
    M, topk = 33, 8
    g = torch.Generator().manual_seed(E + live)
    x = (torch.randn(M, E, generator=g) * 8).round().div(8)
    keep = torch.zeros(M, groups, dtype=torch.bool).scatter_(1, torch.rand(M, groups, generator=g).topk(live, dim=1).indices, True)
    x = x.masked_fill(~keep.repeat_interleave(E // groups, dim=1), float("-inf")).to(dtype)
    x[::3] = x[::3].sort(dim=1, descending=True).values
    buf = torch.empty(M * E + 1, dtype=dtype, device=cuda_device)
    view = buf[offset:offset + M * E].view(M, E)
    view.copy_(x)
    want_w, want_ids = oracle.topk_softmax(x, topk, True)
    w, ids = xkb.topk_softmax(view, topk, True)
    assert torch.equal(ids.cpu(), want_ids)
    assert bool(((w.cpu() - want_w).abs() <= 1e-6).all())
