"""Rows that take the router's rounds with expert counts that leave places behind the row: up to all experts selected, most
probabilities exactly 0 (which the places behind the row are too), at every number of experts per lane, with and without
pieces.  Ids exact, weights within fp32 round-off of the oracle; a row of NaN or with an infinite logit selects no expert
behind the row either."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle

pytestmark = pytest.mark.gpu

EXPERTS = [33, 70, 130, 257, 260, 300, 388, 389, 516, 600, 1000, 1023]


@pytest.mark.parametrize("E", EXPERTS)
@pytest.mark.parametrize("part", [0.1, 1.0])
def test_zeros_at_the_end(E, part, cuda_device):
    M, topk = 9, max(21, int(E * part))
    g = torch.Generator().manual_seed(E)
    x = (torch.randn(M, E, generator=g) * 2).round()
    x = torch.where(torch.rand(M, E, generator=g) < 0.7, torch.full_like(x, -300.0), x)
    want_w, want_ids = oracle.topk_softmax(x, topk, True)
    w, ids = xkb.topk_softmax(x.to(cuda_device), topk, True)
    assert torch.equal(ids.cpu(), want_ids)
    assert bool(((w.cpu() - want_w).abs() <= 1e-6).all())


@pytest.mark.parametrize("E", EXPERTS)
@pytest.mark.parametrize("topk", [8, 24])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_rows_without_probabilities(E, topk, value, cuda_device):
    x = torch.zeros(3, E, device=cuda_device)
    x[1, E - 1] = value
    _, ids = xkb.topk_softmax(x, topk, False)
    assert not bool(((ids[1] >= E) & (ids[1] < 0x7FFFFFFF)).any())     # none, or a number that is no place of the row
    assert torch.equal(ids[0].cpu(), torch.arange(topk, dtype=torch.int32)) and torch.equal(ids[0], ids[2])
