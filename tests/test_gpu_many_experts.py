"""Fused calls with fewer slots than experts, at expert counts that no slice of the workspace is rounded up to: the sort
writes more block entries at 16-token blocks than at 8-token ones.  A workspace full of NaN, so that a row that nobody
wrote shows, and both kernels against the oracle; tolerance as in test_gpu_int4.py and test_gpu_mxfp4.py."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle
from tests.gpu_util import assert_within, poisoned_workspace
from xkernels_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["tc", "simt"])
@pytest.mark.parametrize("E,M,top_k", [(65, 5, 8), (257, 29, 8), (272, 1, 8), (272, 16, 8), (288, 1, 8), (416, 18, 8),
                                       (1024, 20, 8), (1024, 62, 8)])
def test_int4(E, M, top_k, path, cuda_device):
    K, N = 512, 128
    A = synth.activations(M, K, seed=M)
    packed, scale = synth.int4_weights(E, N, K, 32, seed=E)
    ids, w = synth.routing(M, E, top_k, seed=7)
    want = oracle.moe_w4a16(A, packed, scale, ids, w, 32)
    args = [t.to(cuda_device) for t in (A, packed, scale, ids, w)]
    ws = poisoned_workspace("xkb_fused_moe_int4_w4a16_workspace_bytes", M, N, K, E, top_k, 0, device=cuda_device)
    for _ in range(3):
        ws.fill_(0xFF)
        got = xkb.fused_moe_int4_w4a16(*args, workspace=ws, path=path)
        ops.check_workspace_status(ws)
        assert_within(got, want, 2e-2, 1e-2, what=f"{path} E={E} M={M}")


@pytest.mark.parametrize("E,M,top_k", [(272, 1, 8), (257, 29, 8)])
def test_mxfp4_generic_path(E, M, top_k, cuda_device):
    hidden, ispp = 64, 64
    A = synth.activations(M, hidden, seed=2)
    t = synth.mxfp4_weights(E, hidden, ispp, seed=M, scale_lo=117, scale_hi=121)
    ids, w = synth.routing(M, E, top_k, seed=7)
    want = oracle.moe_mxfp4(A, t["w13"], t["w13_scale"], t["w2"], t["w2_scale"], ids, w)
    dev = [x.to(cuda_device) for x in (A, t["w13"], t["w13_scale"], t["w2"], t["w2_scale"], ids, w)]
    ws = poisoned_workspace("xkb_fused_moe_mxfp4_workspace_bytes", M, hidden, ispp, E, top_k, device=cuda_device)
    got = xkb.fused_moe_mxfp4(*dev, workspace=ws)
    ops.check_workspace_status(ws)
    assert_within(got, want, 2e-2, 1e-2, what=f"E={E} M={M}", allowed=max(1, want.numel() // 2000))
