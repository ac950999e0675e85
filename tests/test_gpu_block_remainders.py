"""Token blocks that are not full: the tcgen05 kernel loads and multiplies a block's slots only, in groups of eight to 32
positions.  Experts of one slot, of one less and one more than a group, a tile and two tiles, behind a call
of the same routing with NaN activations (what padding positions hold is test_gpu_token_tiles.py's).  Against the oracle, the
two-GEMM layer against the generic path; tolerances as in test_gpu_int4.py and test_gpu_mxfp4.py."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle
from tests.gpu_util import assert_within
from xkernels_b200 import ops, synth

pytestmark = pytest.mark.gpu

COUNTS = [
    (1, 7, 8, 9, 0, 2, 0, 1),               # token tiles of 16 (8: MXFP4)
    (1, 7, 8, 0, 0, 0, 0, 0),               # the fewest tokens that take them whatever the average
    (16, 17, 0, 1, 0, 0, 0, 0),             # experts of more slots than a tile
    (15, 16, 17, 31, 32, 33, 1, 23),        # 64 (32: MXFP4)
    (5, 16, 17, 31, 32, 33, 1, 0),          # 64
    (8, 9, 31, 32, 33, 7, 1, 0),            # 32, the most slots per expert
    (33, 47, 48, 49, 64, 65, 8, 1),         # 64 (128: MXFP4)
    (81, 80, 1, 66, 63, 65, 17, 97),        # 128 (MXFP4 too)
    (128, 129, 96, 97, 255, 1, 150, 127),
]


def _ids(counts, seed):
    """one slot per token, `counts[e]` tokens for expert e, in a shuffled order"""
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)])
    return ids[torch.randperm(ids.numel(), generator=torch.Generator().manual_seed(seed))].reshape(-1, 1).contiguous()


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("K,N,group", [(512, 256, 32), (1024, 256, 128)])
def test_int4(counts, K, N, group, cuda_device):
    M, E = sum(counts), len(counts)
    g = torch.Generator().manual_seed(M + K)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16)
    packed, scale = synth.int4_weights(E, N, K, group, seed=M)
    ids, w = _ids(counts, K), torch.rand(M, 1, generator=g)
    want = oracle.moe_w4a16(A, packed, scale, ids, w, group)
    dev = [t.to(cuda_device) for t in (packed, scale, ids, w)]
    xkb.fused_moe_int4_w4a16(torch.full((M, K), float("nan"), dtype=torch.bfloat16, device=cuda_device), *dev, group_size=group)
    got = xkb.fused_moe_int4_w4a16(A.to(cuda_device), *dev, group_size=group)
    ops.check_status(cuda_device)
    assert_within(got, want, 2e-2, 1e-2, what=f"{counts}")


@pytest.mark.parametrize("counts", COUNTS)
def test_int4_two_gemm_layer(counts, cuda_device):
    hidden, inter, M, E = 512, 256, sum(counts), len(counts)
    A = synth.activations(M, hidden, seed=1, device=cuda_device)
    w13, s13 = synth.int4_weights(E, 2 * inter, hidden, 32, seed=2, device=cuda_device)
    w2, s2 = synth.int4_weights(E, hidden, inter, 32, seed=3, device=cuda_device)
    rest = (w13, s13 * 0.125, w2, s2 * 0.25, _ids(counts, 5).to(cuda_device), torch.ones(M, 1, device=cuda_device))
    xkb.fused_moe_int4_ffn(torch.full_like(A, float("nan")), *rest)
    got = xkb.fused_moe_int4_ffn(A, *rest)
    ops.check_status(cuda_device)
    assert_within(got, xkb.fused_moe_int4_ffn(A, *rest, path="simt"), 2e-2, 1e-2, what=f"{counts}")


@pytest.mark.parametrize("counts", COUNTS)
def test_mxfp4(counts, cuda_device):
    hidden, ispp, M, E = 512, 512, sum(counts), len(counts)
    t = synth.mxfp4_weights(E, hidden, ispp, seed=M, device=cuda_device, scale_lo=117, scale_hi=121)
    A = synth.activations(M, hidden, seed=2, device=cuda_device)
    ids, w = _ids(counts, 6).to(cuda_device), torch.ones(M, 1, device=cuda_device)

    def call(x):
        return xkb.fused_moe_mxfp4(x, t["w13"], t["w13_scale"], t["w2"], t["w2_scale"], ids, w)

    call(torch.full_like(A, float("nan")))
    got = call(A)
    ops.check_status(cuda_device)
    want = oracle.moe_mxfp4(A.cpu(), *(t[k].cpu() for k in ("w13", "w13_scale", "w2", "w2_scale")), ids.cpu(), w.cpu())
    assert_within(got, want, 2e-2, 1e-2, what=f"{counts}", allowed=max(1, want.numel() // 2000))
