"""Token blocks that are not full: the tcgen05 kernel loads and multiplies a block's slots only, in groups of eight to 32
positions.  Experts of one slot, of one less and one more than a group, a tile and two tiles, at every token tile, in a
workspace full of NaN, so that a padding position's activations are NaN and may not reach an output.  Against the
oracle, the two-GEMM layer against the generic path; tolerances as in test_gpu_int4.py and test_gpu_mxfp4.py."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle
from tests.gpu_util import assert_within, int4_tile, mxfp4_tile, poisoned_workspace
from xkernels_b200 import ops, synth

pytestmark = pytest.mark.gpu

# slots per expert, the token tiles of INT4 and MXFP4
COUNTS = [
    ((1, 7, 8, 9, 0, 2, 0, 1), 16, 8),
    ((1, 7, 8, 0, 0, 0, 0, 0), 16, 8),
    ((1, 7, 8, 9, 0, 2, 0, 15), 32, 16),
    ((15, 1, 0, 0), 16, 8),                        # sixteen tokens, the most that take the INT4 tile whatever the average
    ((16, 17, 0, 1, 0, 0, 0, 0), 32, 8),           # experts of more slots than a tile (MXFP4)
    ((15, 16, 17, 31, 32, 33, 1, 23), 64, 32),
    ((5, 16, 17, 31, 32, 33, 1, 0), 64, 32),
    ((8, 9, 31, 32, 33, 7, 1, 0), 32, 32),
    ((33, 47, 48, 49, 64, 65, 8, 1), 64, 128),
    ((81, 80, 1, 66, 63, 65, 17, 97), 128, 128),
    ((128, 129, 96, 97, 255, 1, 150, 127), 128, 128),
]


def _ids(counts, seed):
    """one slot per token, `counts[e]` tokens for expert e, in a shuffled order"""
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)])
    return ids[torch.randperm(ids.numel(), generator=torch.Generator().manual_seed(seed))].reshape(-1, 1).contiguous()


@pytest.mark.parametrize("counts,tile,_", COUNTS)
@pytest.mark.parametrize("K,N,group", [(512, 256, 32), (1024, 256, 128)])
def test_int4(counts, tile, _, K, N, group, cuda_device):
    M, E = sum(counts), len(counts)
    assert int4_tile(M, E, 1) == tile
    g = torch.Generator().manual_seed(M + K)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16)
    packed, scale = synth.int4_weights(E, N, K, group, seed=M)
    ids, w = _ids(counts, K), torch.rand(M, 1, generator=g)
    want = oracle.moe_w4a16(A, packed, scale, ids, w, group)
    ws = poisoned_workspace("xkb_fused_moe_int4_w4a16_workspace_bytes", M, N, K, E, 1, 0, device=cuda_device)
    got = xkb.fused_moe_int4_w4a16(*(t.to(cuda_device) for t in (A, packed, scale, ids, w)), group_size=group, workspace=ws)
    ops.check_workspace_status(ws)
    assert_within(got, want, 2e-2, 1e-2, what=f"{counts}")


@pytest.mark.parametrize("counts,tile,_", COUNTS)
def test_int4_two_gemm_layer(counts, tile, _, cuda_device):
    hidden, inter, M, E = 512, 256, sum(counts), len(counts)
    assert int4_tile(M, E, 1) == tile
    A = synth.activations(M, hidden, seed=1, device=cuda_device)
    w13, s13 = synth.int4_weights(E, 2 * inter, hidden, 32, seed=2, device=cuda_device)
    w2, s2 = synth.int4_weights(E, hidden, inter, 32, seed=3, device=cuda_device)
    rest = (w13, s13 * 0.125, w2, s2 * 0.25, _ids(counts, 5).to(cuda_device), torch.ones(M, 1, device=cuda_device))
    ws = poisoned_workspace("xkb_fused_moe_int4_ffn_workspace_bytes", M, hidden, inter, E, 1, 0, device=cuda_device)
    got = xkb.fused_moe_int4_ffn(A, *rest, workspace=ws)
    ops.check_workspace_status(ws)
    assert_within(got, xkb.fused_moe_int4_ffn(A, *rest, path="simt"), 2e-2, 1e-2, what=f"{counts}")


@pytest.mark.parametrize("counts,_,tile", COUNTS)
def test_mxfp4(counts, _, tile, cuda_device):
    hidden, ispp, M, E = 512, 512, sum(counts), len(counts)
    assert mxfp4_tile(M, E, 1) == tile
    t = synth.mxfp4_weights(E, hidden, ispp, seed=M, device=cuda_device, scale_lo=117, scale_hi=121)
    A = synth.activations(M, hidden, seed=2, device=cuda_device)
    ids, w = _ids(counts, 6).to(cuda_device), torch.ones(M, 1, device=cuda_device)
    ws = poisoned_workspace("xkb_fused_moe_mxfp4_workspace_bytes", M, hidden, ispp, E, 1, device=cuda_device)
    got = xkb.fused_moe_mxfp4(A, t["w13"], t["w13_scale"], t["w2"], t["w2_scale"], ids, w, workspace=ws)
    ops.check_workspace_status(ws)
    want = oracle.moe_mxfp4(A.cpu(), *(t[k].cpu() for k in ("w13", "w13_scale", "w2", "w2_scale")), ids.cpu(), w.cpu())
    assert_within(got, want, 2e-2, 1e-2, what=f"{counts}", allowed=max(1, want.numel() // 2000))
