"""Rows on which the router's short way (few candidates, ranked against each other) ends or is left:
long runs of equal logits, probabilities that underflow or are subnormal, -inf logits, NaN, expert counts at
the edges of a warp.  Ids exact, weights within fp32 round-off of the oracle; where the last place of a
subnormal exponential decides, against the kernel's own ordering of all experts."""

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
@pytest.mark.parametrize("E,topk", [(1, 1), (31, 8), (32, 8), (32, 32), (33, 32), (64, 6), (64, 20), (64, 21), (256, 8), (257, 33), (1024, 32)])
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


def _far_rows(kind, M, E, g):
    """A few comparable leaders, every other logit so far below them that its probability is subnormal or 0."""
    depth = {"subnormal": (88.0, 103.0), "last_units": (100.0, 103.5), "zeros": (102.0, 106.0)}[kind]
    x = -(depth[0] + (depth[1] - depth[0]) * torch.rand(M, E, generator=g))
    lead = torch.rand(M, E, generator=g).argsort(dim=1)[:, :3]
    return x.scatter(1, lead, 0.1 * torch.randn(M, 3, generator=g))


@pytest.mark.parametrize("kind", ["subnormal", "last_units", "zeros"])
@pytest.mark.parametrize("E,topk", [(33, 4), (64, 3), (64, 5), (256, 8), (384, 32)])
def test_subnormal_probabilities_keep_the_tie_rule(kind, E, topk, cuda_device):
    """Equal probabilities go by ascending id also where the division merges exponentials far apart.  The oracle
    is the order of ALL experts (top-k above 32: the general way over every probability of the row)."""
    x = _far_rows(kind, 257, E, torch.Generator().manual_seed(E + topk)).to(cuda_device)
    all_w, all_ids = xkb.topk_softmax(x, E, False)
    steps = all_w[:, 1:] - all_w[:, :-1]
    assert bool((steps <= 0).all()) and bool(((steps < 0) | (all_ids[:, 1:] > all_ids[:, :-1])).all())
    w, ids = xkb.topk_softmax(x, topk, False)
    assert torch.equal(ids, all_ids[:, :topk])
    assert torch.equal(w, all_w[:, :topk])


def test_rows_whose_kth_exponentials_merge(cuda_device):
    """Pinned rows: 27 and 28 * 2^-149 over a sum of 2, and 3 and 5 * 2^-149 over a sum of 3.9, are one
    probability each, so the smaller id is taken."""
    x = torch.full((2, 64), -1000.0)
    x[0, 0], x[0, 33], x[0, 10], x[0, 40] = 0.0, -0.01, -99.98309, -99.946724
    x[1, 40:44] = torch.tensor([0.0, -0.01, -0.02, -0.07])
    x[1, 50], x[1, 3] = -101.68, -102.15
    ids = xkb.topk_softmax(x.to(cuda_device), 3, False)[1]
    assert ids[0].tolist() == [0, 33, 10]
    ids = xkb.topk_softmax(x.to(cuda_device), 5, False)[1]
    assert ids[1].tolist() == [40, 41, 42, 43, 3]
