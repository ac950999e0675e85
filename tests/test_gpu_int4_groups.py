"""INT4 scale groups of 64, 128 and 256 on the tcgen05 path (K a multiple of eight groups), at the edges
of its token tiles, against the oracle and against the generic path that all other shapes take."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle
from tests.gpu_util import assert_within, to_dev
from xkernels_b200 import ops, synth

pytestmark = pytest.mark.gpu
KEYS = ("A", "packed", "scale", "topk_ids", "topk_w")


@pytest.mark.parametrize("M,K,N,E,top_k,group", [
    (1, 1024, 128, 8, 2, 128),     # one tile row, one lap of a scale tile
    (16, 2048, 256, 8, 2, 128),    # 16-token tiles, two laps
    (17, 1024, 384, 8, 3, 64),
    (64, 1024, 128, 8, 3, 64),     # 64-token tiles
    (33, 2048, 256, 2, 2, 256),    # 64-token tiles, one scale per stage
    (96, 1024, 256, 6, 4, 128),    # 128-token tiles, two row tiles per token tile
    (300, 2048, 128, 3, 2, 256),   # 128-token tiles, one row tile
    (5, 1280, 128, 4, 2, 128),     # K is not a multiple of eight groups: the generic path
])
def test_groups_against_oracle(M, K, N, E, top_k, group, cuda_device):
    g = torch.Generator().manual_seed(M + K + group)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16)
    packed, scale = synth.int4_weights(E, N, K, group, seed=M, device="cpu")
    ids, w = synth.routing(M, E, top_k, seed=K, device="cpu")
    want = oracle.moe_w4a16(A, packed, scale, ids, w, group)
    d = to_dev(dict(zip(KEYS, (A, packed, scale, ids, w))), cuda_device)
    args = [d[k] for k in KEYS]
    got = xkb.fused_moe_int4_w4a16(*args, group_size=group)
    ops.check_status(cuda_device)
    assert_within(got, want, 2e-2, 1e-2, what="auto")
    # same bf16 weights, fp32 sums in another order: the bf16 result moves by one rounding at most
    assert_within(got, xkb.fused_moe_int4_w4a16(*args, group_size=group, path="simt"), 1e-2, 1e-2, what="auto vs simt")


def test_weights_tma_cannot_read_keep_the_generic_path(cuda_device):
    """A scale tensor that does not start on 16 bytes was accepted at these groups, and still is."""
    M, K, N, E, top_k, group = 8, 1024, 128, 4, 2, 128
    A = synth.activations(M, K, seed=1, device=cuda_device)
    packed, scale = synth.int4_weights(E, N, K, group, seed=2, device=cuda_device)
    ids, w = synth.routing(M, E, top_k, seed=3, device=cuda_device)
    flat = torch.empty(scale.numel() + 1, dtype=scale.dtype, device=cuda_device)
    shifted = flat[1:].view(scale.shape)
    shifted.copy_(scale)
    want = xkb.fused_moe_int4_w4a16(A, packed, scale, ids, w, group_size=group, path="simt")
    assert torch.equal(xkb.fused_moe_int4_w4a16(A, packed, shifted, ids, w, group_size=group), want)
    with pytest.raises(RuntimeError, match="tcgen05"):
        xkb.fused_moe_int4_w4a16(A, packed, scale, ids, w, group_size=group, path="tc")


def test_two_gemm_layer_at_group_128(cuda_device):
    M, hidden, inter, E, top_k, group = 20, 1024, 1024, 4, 2, 128
    g = torch.Generator().manual_seed(5)
    A = torch.randn(M, hidden, generator=g).to(torch.bfloat16)
    w13, s13 = synth.int4_weights(E, 2 * inter, hidden, group, seed=1)
    w2, s2 = synth.int4_weights(E, hidden, inter, group, seed=2)
    s13, s2 = s13 * 0.125, s2 * 0.25
    ids, w = synth.routing(M, E, top_k, seed=3)
    t = [x.to(cuda_device) for x in (A, w13, s13, w2, s2, ids, w)]
    got = xkb.fused_moe_int4_ffn(*t, group_size=group)
    ops.check_status(cuda_device)
    assert_within(got, xkb.fused_moe_int4_ffn(*t, group_size=group, path="simt"), 2e-2, 1e-2, what="auto vs simt")


@pytest.mark.parametrize("M,group", [(8, 128), (100, 64), (200, 256)])
def test_scales_of_any_magnitude(M, group, cuda_device, monkeypatch):
    """A C caller may pass any bf16 scale at these groups: the generic path answered them, so the tensor-core path
    gives the same (weights rounded once; infinities and NaN where the generic path has them).  Below 2^-118 its
    weights are off by 2^-126 at most."""
    monkeypatch.setattr(ops, "_check_int4_scales", lambda scale: None)   # Python refuses them before the library sees them
    K, N, E, top_k = 2048, 256, 4, 2
    A = synth.activations(M, K, seed=1, device=cuda_device)
    packed, scale = synth.int4_weights(E, N, K, group, seed=2, device=cuda_device)
    ids, w = synth.routing(M, E, top_k, seed=3, device=cuda_device)
    scale[:, 0:32] *= 2.0 ** 100                       # rows of their own magnitude
    scale[:, 32:64] *= 2.0 ** -100
    scale[:, 64:96] = torch.finfo(torch.bfloat16).tiny / 8   # subnormal
    scale[:, 112:128, ::2] = 100.0                     # in and out of the fast conversion's range inside a row
    scale[:, 96, 0], scale[:, 97, 1], scale[:, 98, 2] = float("inf"), float("nan"), 3.0e38
    got = xkb.fused_moe_int4_w4a16(A, packed, scale, ids, w, group_size=group)
    want = xkb.fused_moe_int4_w4a16(A, packed, scale, ids, w, group_size=group, path="simt")
    ops.check_status(cuda_device)
    off = 2.0 ** -126 * A.double().abs().sum(dim=1, keepdim=True)
    assert bool(((got - want)[:, 64:96].double().abs() <= 1.01 * off).all())
    for rows in (slice(0, 32), slice(32, 64), slice(96, 112), slice(112, 256)):
        a, b = got[:, rows].double(), want[:, rows].double()
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
        ok = b.isfinite()
        # sums in another order, then one bf16 rounding; relative to the rows' own magnitude
        assert bool(((a - b).abs()[ok] <= 1e-2 * b[ok].abs() + 1e-2 * b[ok].abs().median()).all())
