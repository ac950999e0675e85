"""Decode batches, whose routing the activation gather sorts itself (up to 512 slots, 148 blocks and a top-k of 32):
both sides of those limits, few and many experts, dropped slots, an expert map.  The generic path, which
takes the sort's own kernels, is the check: same bf16 weights, fp32 sums in another order."""

import pytest
import torch

import xkernels_b200 as xkb
from tests.gpu_util import assert_within
from xkernels_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,top_k,E", [
    (1, 1, 1), (1, 8, 48), (3, 32, 40), (3, 33, 40), (63, 8, 48), (64, 8, 48), (65, 8, 48), (128, 8, 48),
    (129, 8, 48), (148, 2, 7), (149, 2, 7), (512, 1, 7), (513, 1, 7), (1025, 1, 7), (20, 8, 1024),
])
@pytest.mark.parametrize("dropped", [False, True])
def test_int4(M, top_k, E, dropped, cuda_device):
    K, N = 256, 128
    A = synth.activations(M, K, seed=M, device=cuda_device)
    packed, scale = synth.int4_weights(E, N, K, 32, seed=E, device=cuda_device)
    ids, w = synth.routing(M, E, top_k, seed=7, device=cuda_device)
    emap = None
    if dropped:
        g = torch.Generator(device=cuda_device).manual_seed(1)
        ids[torch.rand(ids.shape, generator=g, device=cuda_device) < 0.3] = -1
        emap = torch.arange(E, dtype=torch.int32, device=cuda_device).flip(0).contiguous()
        emap[::5] = -1
    args = (A, packed, scale, ids, w)
    got = xkb.fused_moe_int4_w4a16(*args, expert_map=emap, path="tc")
    ops.check_status(cuda_device)
    assert_within(got, xkb.fused_moe_int4_w4a16(*args, expert_map=emap, path="simt"), 1e-2, 1e-2, what="tc vs simt")
    assert torch.equal(got, xkb.fused_moe_int4_w4a16(*args, expert_map=emap, path="tc"))


@pytest.mark.parametrize("M,top_k,E", [(1, 6, 256), (5, 32, 64), (5, 33, 64), (85, 6, 256), (86, 6, 256), (171, 6, 256)])
def test_mxfp4(M, top_k, E, cuda_device):
    A = synth.activations(M, 512, seed=M, device=cuda_device)
    t = synth.mxfp4_weights(E, 512, 512, seed=E, device=cuda_device, scale_lo=117, scale_hi=121)
    ids, w = synth.routing(M, E, top_k, seed=7, device=cuda_device)
    args = (A, t["w13"], t["w13_scale"], t["w2"], t["w2_scale"], ids, w)
    got = xkb.fused_moe_mxfp4(*args)
    ops.check_status(cuda_device)
    simt = xkb.fused_moe_mxfp4(*args, path="simt")
    assert_within(got, simt, 2e-2, 1e-2, what="auto vs simt", allowed=max(1, simt.numel() // 2000))


@pytest.mark.parametrize("M,top_k", [(65, 8), (300, 33), (700, 1), (4736, 8), (4737, 8), (5001, 33)])
def test_most_tokens_without_a_slot_here(M, top_k, cuda_device):
    """A rank that holds 2 of 64 experts (expert_map).  From 4737 blocks on the gather goes through the kept slots'
    positions instead of the tokens; outputs of tokens without a local expert are zero."""
    A = synth.activations(M, 512, seed=M, device=cuda_device)
    ids, w = synth.routing(M, 64, top_k, seed=7, device=cuda_device)
    emap = torch.full((64,), -1, dtype=torch.int32, device=cuda_device)
    emap[5], emap[60] = 1, 0
    none = (emap[ids.long()] < 0).all(dim=1)
    packed, scale = synth.int4_weights(2, 256, 512, 32, seed=3, device=cuda_device)
    t = synth.mxfp4_weights(2, 512, 512, seed=4, device=cuda_device, scale_lo=117, scale_hi=121)
    calls = ((xkb.fused_moe_int4_w4a16, (A, packed, scale, ids, w)),
             (xkb.fused_moe_mxfp4, (A, t["w13"], t["w13_scale"], t["w2"], t["w2_scale"], ids, w)))
    for call, args in calls:
        got = call(*args, expert_map=emap)
        ops.check_status(cuda_device)
        simt = call(*args, expert_map=emap, path="simt")
        assert_within(got, simt, 2e-2, 1e-2, what="auto vs simt", allowed=max(1, simt.numel() // 2000))
        assert bool((got[none] == 0).all())
