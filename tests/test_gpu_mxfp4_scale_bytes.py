"""The kernel that converts MXFP4 weights to bf16 takes any scale byte: the smallest, both sides of the line (133 / 134) from
which a second multiplication is made, and 0xFF, which means weight 0; bytes of one stage on either side of the line.
Against the oracle with fp32 contractions; the bound is four roundings to bf16 (gate_up, activation, rows, output), so the
activations are large enough (about 10^3) for outputs behind weights of 2^-127 to be normal numbers."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle
from xkernels_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w2_bytes", [(0, 1), (4, 5, 6, 7), (56, 57), (132, 133, 134, 135), (127, 190), (120, 121, 255)])
@pytest.mark.parametrize("w13_bytes", [(126, 127), (128, 134), (127, 133, 255)])
@pytest.mark.parametrize("M", [60, 150])      # 30 and 75 slots per expert
def test_scale_bytes(M, w13_bytes, w2_bytes, cuda_device):
    hidden, ispp, E, top_k = 512, 512, 4, 2
    g = torch.Generator().manual_seed(M + w2_bytes[0])
    t = synth.mxfp4_weights(E, hidden, ispp, seed=M)
    for name, choice in (("w13_scale", w13_bytes), ("w2_scale", w2_bytes)):
        at = torch.randint(0, len(choice), t[name].shape, generator=g)
        t[name] = torch.tensor(choice, dtype=torch.uint8)[at].contiguous()
    A = torch.randn(M, hidden, generator=g).to(torch.bfloat16)
    ids, w = synth.routing(M, E, top_k, seed=3)
    args = (A, t["w13"], t["w13_scale"], t["w2"], t["w2_scale"], ids, w)
    want = oracle.moe_mxfp4(*args, swiglu_limit=None, fp32_matmul=True).double()
    got = xkb.fused_moe_mxfp4(*(x.to(cuda_device) for x in args), swiglu_limit=None)
    ops.check_status(cuda_device)
    rel = float((got.cpu().double() - want).norm() / want.norm())
    assert rel <= 4 * 2.0 ** -9, rel
