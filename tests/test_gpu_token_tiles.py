"""Calls on both sides of every line between token tiles, each with the tile that it takes (asked of the library, so that
a line that moves fails here): the dequantised weights bit for bit, the oracle at an odd number of stages, the two-GEMM
layer, the MXFP4 kernels.  And blocks that are not full in a workspace full of NaN, where a padding position's
activations are NaN and may not reach an output.  Tolerances as in test_gpu_int4.py and test_gpu_mxfp4.py."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle
from tests import test_gpu_int4, test_gpu_int4_ffn, test_gpu_mxfp4_block_scaled
from tests.gpu_util import assert_within, int4_tile, mxfp4_tile, poisoned_workspace, to_dev
from xkernels_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,per_expert,tile", [(64, 4, 16), (32, 8, 32), (32, 16, 32), (32, 32, 64), (2, 256, 128)])
def test_dequantised_weights_are_bit_exact(E, per_expert, tile, cuda_device):
    assert int4_tile(E * per_expert, E, 1) == tile
    test_gpu_int4.test_dequantised_weights_are_bit_exact(E, per_expert, 128, cuda_device)


@pytest.mark.parametrize("M,K,N,E,top_k,tile", [
    (16, 512, 256, 8, 2, 16),       # four slots per expert, the most
    (24, 768, 384, 8, 4, 32),       # an odd number of stages
    (17, 512, 256, 17, 4, 16),      # the same average with more tokens than a tile
    (17, 768, 256, 16, 4, 32),      # a little above it
    (32, 256, 128, 8, 4, 32),       # sixteen, the most
    (33, 768, 128, 8, 4, 64),       # one token more
    (40, 768, 384, 8, 4, 64),
    (80, 512, 256, 8, 4, 64),       # forty, the most
    (81, 768, 256, 8, 4, 128),      # one token more
])
def test_int4(M, K, N, E, top_k, tile, cuda_device):
    assert int4_tile(M, E, top_k) == tile
    test_gpu_int4.test_tensor_core_path_against_oracle(M, K, N, E, top_k, tile, cuda_device)


@pytest.mark.parametrize("M,tile", [(24, 32), (40, 64), (81, 128)])
def test_int4_two_gemm_layer(M, tile, cuda_device):
    assert int4_tile(M, 8, 4) == tile
    test_gpu_int4_ffn.test_tensor_core_path_against_oracle(M, 768, 512, 8, 4, cuda_device)


@pytest.mark.parametrize("M,hidden,ispp,bias,tile", [
    (20, 512, 512, True, 8),         # five slots per expert, the most
    (21, 512, 1024, False, 16),      # one slot more
    (48, 512, 512, False, 16),       # twelve, the most
    (49, 1024, 512, True, 32),       # one slot more
    (112, 512, 512, False, 32),      # 28, the most
    (113, 512, 512, True, 128),      # one slot more: the kernel that converts to bf16
])
def test_mxfp4(M, hidden, ispp, bias, tile, cuda_device):
    assert mxfp4_tile(M, 4, 1) == tile
    test_gpu_mxfp4_block_scaled.test_token_tiles(M, hidden, ispp, 4, 1, bias, cuda_device)


@pytest.mark.parametrize("byte", [191, 200])
def test_scale_bytes_above_190_in_the_block_scaled_kernel(byte, cuda_device):
    """Ordinary weights up to 48 slots per expert, and so in this kernel."""
    c = test_gpu_mxfp4_block_scaled._case(40, 512, 512, 4, 2)
    c["w2_scale"][:, 5, 3] = byte
    assert mxfp4_tile(40, 4, 2) == 32
    got = test_gpu_mxfp4_block_scaled._call(c, cuda_device)
    ops.check_status(cuda_device)
    want = test_gpu_mxfp4_block_scaled._want(c)
    assert_within(got, want, 2e-2, 1e-2, what="scale bytes", allowed=max(1, want.numel() // 2000))


# slots per expert, the token tiles of INT4 and MXFP4
COUNTS = [
    ((1, 7, 8, 9, 0, 2, 0, 1), 16, 8),
    ((1, 7, 8, 9, 0, 2, 0, 15), 32, 16),
    ((15, 1, 0, 0), 16, 8),                        # sixteen tokens, the most that take the INT4 tile whatever the average
    ((16, 17, 0, 1, 0, 0, 0, 0), 32, 8),           # experts of more slots than a tile (MXFP4)
    ((15, 16, 17, 31, 32, 33, 1, 23), 64, 32),
    ((8, 9, 31, 32, 33, 7, 1, 0), 32, 32),
    ((33, 47, 48, 49, 64, 65, 8, 1), 64, 128),
    ((128, 129, 96, 97, 255, 1, 150, 127), 128, 128),
]


def _ids(counts, seed):
    """one slot per token, `counts[e]` tokens for expert e, in a shuffled order"""
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)])
    return ids[torch.randperm(ids.numel(), generator=torch.Generator().manual_seed(seed))].reshape(-1, 1).contiguous()


@pytest.mark.parametrize("counts,tile,_", COUNTS)
@pytest.mark.parametrize("K,N,group", [(512, 256, 32), (1024, 256, 128)])
def test_int4_padding_is_nan(counts, tile, _, K, N, group, cuda_device):
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
def test_int4_layer_padding_is_nan(counts, tile, _, cuda_device):
    hidden, inter, M, E = 512, 256, sum(counts), len(counts)
    assert int4_tile(M, E, 1) == tile
    A = synth.activations(M, hidden, seed=1)
    w13, s13 = synth.int4_weights(E, 2 * inter, hidden, 32, seed=2)
    w2, s2 = synth.int4_weights(E, hidden, inter, 32, seed=3)
    args = (A, w13, s13 * 0.125, w2, s2 * 0.25, _ids(counts, 5), torch.ones(M, 1))
    want = oracle.moe_int4_ffn(*args, 32)
    ws = poisoned_workspace("xkb_fused_moe_int4_ffn_workspace_bytes", M, hidden, inter, E, 1, 0, device=cuda_device)
    got = xkb.fused_moe_int4_ffn(*(t.to(cuda_device) for t in args), workspace=ws)
    ops.check_workspace_status(ws)
    assert_within(got, want, 2e-2, 1e-2, what=f"{counts}", allowed=max(1, want.numel() // 2000))


@pytest.mark.parametrize("counts,_,tile", COUNTS)
def test_mxfp4_padding_is_nan(counts, _, tile, cuda_device):
    hidden, ispp, M, E = 512, 512, sum(counts), len(counts)
    assert mxfp4_tile(M, E, 1) == tile
    t = synth.mxfp4_weights(E, hidden, ispp, seed=M, scale_lo=117, scale_hi=121)
    args = (synth.activations(M, hidden, seed=2), t["w13"], t["w13_scale"], t["w2"], t["w2_scale"], _ids(counts, 6), torch.ones(M, 1))
    want = oracle.moe_mxfp4(*args)
    ws = poisoned_workspace("xkb_fused_moe_mxfp4_workspace_bytes", M, hidden, ispp, E, 1, device=cuda_device)
    got = xkb.fused_moe_mxfp4(*(x.to(cuda_device) for x in args), workspace=ws)
    ops.check_workspace_status(ws)
    assert_within(got, want, 2e-2, 1e-2, what=f"{counts}", allowed=max(1, want.numel() // 2000))


@pytest.mark.parametrize("M,top_k,E", [(1, 8, 48), (3, 33, 40), (65, 8, 48), (513, 1, 7), (20, 8, 1024)])
def test_neither_path_returns_rows_of_the_other(M, top_k, E, cuda_device):
    """Decode routing on both paths, each in a workspace of its own."""
    K, N = 256, 128
    A = synth.activations(M, K, seed=M)
    packed, scale = synth.int4_weights(E, N, K, 32, seed=E)
    ids, w = synth.routing(M, E, top_k, seed=7)
    want = oracle.moe_w4a16(A, packed, scale, ids, w, 32)
    d = to_dev(dict(enumerate((A, packed, scale, ids, w))), cuda_device)
    for path in ("tc", "simt"):
        ws = poisoned_workspace("xkb_fused_moe_int4_w4a16_workspace_bytes", M, N, K, E, top_k, 0, device=cuda_device)
        got = xkb.fused_moe_int4_w4a16(*d.values(), path=path, workspace=ws)
        ops.check_workspace_status(ws)
        assert_within(got, want, 2e-2, 1e-2, what=path)


def _repeat(call, want, times, dev):
    same = torch.ones((), dtype=torch.bool, device=dev)
    for _ in range(times):
        same &= (call() == want).all()
    ops.check_status(dev)
    assert bool(same)


@pytest.mark.parametrize("M,E,top_k,K,N,group", [
    (700, 8, 4, 2048, 2048, 32),        # pairs of row tiles, ragged blocks
    (700, 8, 4, 2048, 2048, 128),
    (500, 4, 2, 2048, 1920, 32),        # one row tile per token tile
])
def test_repeated_calls(M, E, top_k, K, N, group, cuda_device):
    """128-token tiles, many times: the same bits (a stage of weights handed back too early shows in a few calls of hundreds)."""
    assert int4_tile(M, E, top_k) == 128
    A = synth.activations(M, K, seed=1, device=cuda_device)
    packed, scale = synth.int4_weights(E, N, K, group, seed=2, device=cuda_device)
    ids, w = synth.routing(M, E, top_k, seed=3, device=cuda_device)
    args = (A, packed, scale, ids, w)
    want = xkb.fused_moe_int4_w4a16(*args, group_size=group)
    assert_within(want, xkb.fused_moe_int4_w4a16(*args, group_size=group, path="simt"), 2e-2, 1e-2, what="tc vs simt")
    _repeat(lambda: xkb.fused_moe_int4_w4a16(*args, group_size=group), want, 400, cuda_device)


def test_repeated_layer_calls(cuda_device):
    M, hidden, inter, E, top_k = 700, 2048, 1024, 8, 4
    A = synth.activations(M, hidden, seed=1, device=cuda_device)
    w13, s13 = synth.int4_weights(E, 2 * inter, hidden, 32, seed=2, device=cuda_device)
    w2, s2 = synth.int4_weights(E, hidden, inter, 32, seed=3, device=cuda_device)
    ids, w = synth.routing(M, E, top_k, seed=4, device=cuda_device)
    args = (A, w13, s13 * 0.125, w2, s2 * 0.25, ids, w)
    _repeat(lambda: xkb.fused_moe_int4_ffn(*args), xkb.fused_moe_int4_ffn(*args), 400, cuda_device)
