"""INT4 at 48 to 93 slots per expert, 128-token tiles: blocks that are full, one over and nearly empty, one and
several pairs of row tiles, short and long contractions, scale groups; and the two-GEMM layer, whose both GEMMs
take them.  Against the oracle, tolerance as in test_gpu_int4.py; the layer against the generic path."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle
from tests.gpu_util import assert_within
from xkernels_b200 import ops, synth

pytestmark = pytest.mark.gpu


def _ids(counts, seed):
    """one slot per token, `counts[e]` tokens for expert e, in a shuffled order"""
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)])
    return ids[torch.randperm(ids.numel(), generator=torch.Generator().manual_seed(seed))].reshape(-1, 1).contiguous()


@pytest.mark.parametrize("counts", [
    (80, 81, 10), (160, 1, 0),          # 57 and 54 slots per expert on average
    (96, 97, 20), (193, 0, 32),         # 71 and 75
    (112, 113, 30), (225, 16, 1),       # 85 and 81
])
@pytest.mark.parametrize("K,N,group", [(256, 256, 32), (1024, 512, 32), (2048, 768, 128)])
def test_against_oracle(counts, K, N, group, cuda_device):
    M, E = sum(counts), len(counts)
    g = torch.Generator().manual_seed(M + K)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16)
    packed, scale = synth.int4_weights(E, N, K, group, seed=M)
    ids, w = _ids(counts, K), torch.rand(M, 1, generator=g)
    want = oracle.moe_w4a16(A, packed, scale, ids, w, group)
    args = [t.to(cuda_device) for t in (A, packed, scale, ids, w)]
    got = xkb.fused_moe_int4_w4a16(*args, group_size=group)
    ops.check_status(cuda_device)
    assert_within(got, want, 2e-2, 1e-2, what=f"{counts}")
    for _ in range(3):
        assert torch.equal(got, xkb.fused_moe_int4_w4a16(*args, group_size=group))


@pytest.mark.parametrize("M", [110, 140, 170])      # 55, 70, 85 slots per expert
def test_two_gemm_layer(M, cuda_device):
    hidden, inter, E, top_k = 512, 256, 4, 2
    A = synth.activations(M, hidden, seed=1, device=cuda_device)
    w13, s13 = synth.int4_weights(E, 2 * inter, hidden, 32, seed=2, device=cuda_device)
    w2, s2 = synth.int4_weights(E, hidden, inter, 32, seed=3, device=cuda_device)
    ids, w = synth.routing(M, E, top_k, seed=4, device=cuda_device)
    args = (A, w13, s13 * 0.125, w2, s2 * 0.25, ids, w)
    got = xkb.fused_moe_int4_ffn(*args)
    ops.check_status(cuda_device)
    assert_within(got, xkb.fused_moe_int4_ffn(*args, path="simt"), 2e-2, 1e-2, what="layer")
