"""Rows on which the router's short way (few candidates, ranked against each other) ends or is left:
long runs of equal logits, probabilities that underflow, -inf logits, NaN, expert counts at the edges
of a warp.  Ids exact, weights within fp32 round-off of the oracle."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle

pytestmark = pytest.mark.gpu


def _rows(kind, M, E, g):
    x = torch.randn(M, E, generator=g)
    if kind == "levels":                       # a few distinct values: ties across lanes and inside them
        return (x * 1.5).round()
    if kind == "underflow":                    # most exponentials are exactly 0
        return x * 200.0
    if kind == "minus_inf":
        keep = (x >= 0.5) | torch.nn.functional.one_hot(torch.arange(M) % E, E).bool()   # one finite logit at least
        return torch.where(keep, x, torch.full_like(x, float("-inf")))
    if kind == "neighbours":                   # logits that differ in the last bits: equal probabilities
        return 1.0 + torch.randint(0, 3, (M, E), generator=g) * 2.0 ** -23
    return x


@pytest.mark.parametrize("kind", ["random", "levels", "underflow", "minus_inf", "neighbours"])
@pytest.mark.parametrize("E,topk", [(1, 1), (31, 8), (32, 8), (33, 32), (64, 6), (256, 8), (257, 33), (1024, 32)])
def test_edges_against_oracle(kind, E, topk, cuda_device):
    x = _rows(kind, 65, E, torch.Generator().manual_seed(E + topk))
    want_w, want_ids = oracle.topk_softmax(x, topk, True)
    w, ids = xkb.topk_softmax(x.to(cuda_device), topk, True)
    if kind != "neighbours":   # there the oracle's own sum order decides which probabilities are equal
        assert torch.equal(ids.cpu(), want_ids)
    assert bool(((w.cpu() - want_w).abs() <= 1e-6 + 1e-5 * want_w.abs()).all())
    assert all(len(set(r)) == topk for r in ids.tolist())


def test_a_row_with_nan_leaves_the_others_alone(cuda_device):
    x = torch.randn(9, 128, generator=torch.Generator().manual_seed(3))
    want_w, want_ids = oracle.topk_softmax(x, 8, False)
    x[4, 77] = float("nan")
    w, ids = xkb.topk_softmax(x.to(cuda_device), 8, False)
    keep = [i for i in range(9) if i != 4]
    assert torch.equal(ids.cpu()[keep], want_ids[keep])
    assert bool(((w.cpu() - want_w).abs()[keep] <= 1e-6).all())
