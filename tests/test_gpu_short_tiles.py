"""Tiles of one, two and three 256-K stages at 16-token tiles, where the read-out of a tile is due before much else has
happened: several tiles per CTA, so that every accumulator set is used again and again.  Against the oracle (tolerance
as in test_gpu_int4.py), and the same call repeated, which has to give the same bits: the sums have one order."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle
from tests.gpu_util import assert_within, int4_tile
from xkernels_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [256, 512, 768])
@pytest.mark.parametrize("M,E,N,group", [(8, 16, 16384, 32), (1, 8, 16384, 32), (3, 8, 8192 + 128, 32)])
def test_int4(M, E, N, group, K, cuda_device):
    top_k = 8
    assert int4_tile(M, E, top_k) == 16
    A = synth.activations(M, K, seed=M)
    packed, scale = synth.int4_weights(E, N, K, group, seed=E)
    ids, w = synth.routing(M, E, top_k, seed=7)
    want = oracle.moe_w4a16(A, packed, scale, ids, w, group)
    args = [t.to(cuda_device) for t in (A, packed, scale, ids, w)]
    got = xkb.fused_moe_int4_w4a16(*args, group_size=group, path="tc")
    ops.check_status(cuda_device)
    assert_within(got, want, 2e-2, 1e-2, what=f"K={K} M={M}")
    other = torch.flip(args[0], dims=[1]).contiguous()   # other sums in the accumulators in between
    same = torch.ones((), dtype=torch.bool, device=cuda_device)
    for _ in range(100):
        xkb.fused_moe_int4_w4a16(other, *args[1:], group_size=group, path="tc")
        same &= (xkb.fused_moe_int4_w4a16(*args, group_size=group, path="tc") == got).all()
    ops.check_status(cuda_device)
    assert bool(same)


def test_int4_two_gemm_layer(cuda_device):
    """inter 256: the second GEMM's tiles are one stage long."""
    M, E, hidden, inter, top_k = 4, 8, 4096, 256, 8
    A = synth.activations(M, hidden, seed=1, device=cuda_device)
    w13, s13 = synth.int4_weights(E, 2 * inter, hidden, 32, seed=2, device=cuda_device)
    w2, s2 = synth.int4_weights(E, hidden, inter, 32, seed=3, device=cuda_device)
    ids, w = synth.routing(M, E, top_k, seed=4, device=cuda_device)
    args = (A, w13, s13 * 0.0625, w2, s2 * 0.25, ids, w)
    got = xkb.fused_moe_int4_ffn(*args)
    ops.check_status(cuda_device)
    assert_within(got, xkb.fused_moe_int4_ffn(*args, path="simt"), 2e-2, 1e-2, what="layer")
    for _ in range(100):
        assert torch.equal(got, xkb.fused_moe_int4_ffn(*args))
