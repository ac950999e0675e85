"""The block-scaled MXFP4 kernels at the edges of their token tiles and of the activations' two-term split,
against the oracle and against the generic path.  Tolerances as in test_gpu_mxfp4.py."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle
from tests.gpu_util import assert_within, to_dev
from xkernels_b200 import ops, synth

pytestmark = pytest.mark.gpu
KEYS = ("A", "w13", "w13_scale", "w2", "w2_scale", "topk_ids", "topk_w", "b13", "b2")


def _case(M, hidden, ispp, E, top_k, bias=False, seed=0):
    g = torch.Generator().manual_seed(seed + M)
    wts = synth.mxfp4_weights(E, hidden, ispp, seed=M, scale_lo=117, scale_hi=121, with_bias=bias)
    A = torch.randn(M, hidden, generator=g).to(torch.bfloat16)
    ids, w = synth.routing(M, E, top_k, seed=seed)
    return {"A": A, **wts, "topk_ids": ids, "topk_w": w}


def _call(c, dev, **kw):
    d = to_dev({k: c[k] for k in KEYS}, dev)
    return xkb.fused_moe_mxfp4(d["A"], d["w13"], d["w13_scale"], d["w2"], d["w2_scale"], d["topk_ids"], d["topk_w"],
                               b13=d["b13"], b2=d["b2"], **kw)


def _want(c, **kw):
    return oracle.moe_mxfp4(c["A"], c["w13"], c["w13_scale"], c["w2"], c["w2_scale"], c["topk_ids"], c["topk_w"],
                            b13=c["b13"], b2=c["b2"], **kw)


@pytest.mark.parametrize("M,hidden,ispp,E,top_k,bias", [
    (1, 512, 512, 4, 2, False),        # 16-token tiles, one slot each
    (33, 1024, 512, 4, 2, True),       # 32-token tiles
    (90, 512, 1024, 4, 2, False),      # 64-token tiles
    (112, 512, 512, 2, 2, True),       # 112-token tiles, exactly full
    (113, 1024, 512, 2, 2, False),     # one more: a second block
    (700, 512, 512, 3, 2, True),       # several blocks, ragged
])
def test_token_tiles(M, hidden, ispp, E, top_k, bias, cuda_device):
    c = _case(M, hidden, ispp, E, top_k, bias)
    got = _call(c, cuda_device)
    ops.check_status(cuda_device)
    want = _want(c)
    assert_within(got, want, 2e-2, 1e-2, what="block-scaled", allowed=max(1, want.numel() // 2000))
    assert torch.equal(got, _call(c, cuda_device))


def test_wide_range_activations(cuda_device):
    """Magnitudes over 2^-20 .. 2^20 inside every block of 32: the small ones only matter to the bits that an
    fp32 sum beside the large ones keeps."""
    c = _case(24, 512, 512, 4, 2)
    g = torch.Generator().manual_seed(7)
    c["A"] = (c["A"].float() * torch.exp2(torch.randint(-20, 21, c["A"].shape, generator=g).float()) * 2.0 ** -18).to(torch.bfloat16)
    want = _want(c)
    assert_within(_call(c, cuda_device), want, 2e-2, 1e-2, what="wide range", allowed=max(1, want.numel() // 2000))
    c["A"] = torch.zeros_like(c["A"])
    c["A"][:, 3] = 2.0 ** -130          # a bf16 subnormal alone in its block
    c["w13_scale"][:] = 180             # weights of 2^53: gate and up of 2^-77, activations of 0
    got = _call(c, cuda_device)
    assert torch.equal(got, torch.zeros_like(got))


def test_nan_scale_bytes_are_zero_weights(cuda_device):
    """Scale byte 0xFF decodes to weight 0 (as in the reference), in whole rows and single groups."""
    c = _case(40, 512, 512, 4, 2)
    g = torch.Generator().manual_seed(3)
    for k in ("w13_scale", "w2_scale"):
        kill = torch.rand(c[k].shape, generator=g) < 0.05
        kill[:, ::17] = True
        c[k][kill] = 0xFF
    want = _want(c)
    assert_within(_call(c, cuda_device), want, 2e-2, 1e-2, what="0xFF", allowed=max(1, want.numel() // 2000))
    c["w2_scale"][:] = 0xFF
    got = _call(c, cuda_device)
    assert torch.equal(got, torch.zeros_like(got))


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("limit", [10.0, None])
def test_non_finite_activations(value, limit, cuda_device):
    """What an infinity or NaN in one token does: the same outputs turn NaN or infinite as on the generic path,
    and no other token changes."""
    c = _case(20, 512, 512, 4, 2)
    clean = _call(c, cuda_device, swiglu_limit=limit)
    c["A"][5, 100] = value
    got, simt = _call(c, cuda_device, swiglu_limit=limit), _call(c, cuda_device, swiglu_limit=limit, path="simt")
    assert torch.equal(torch.isnan(got), torch.isnan(simt)) and torch.equal(torch.isinf(got), torch.isinf(simt))
    keep = [i for i in range(20) if i != 5]
    assert torch.equal(got[keep], clean[keep])


def test_weights_on_16_byte_boundaries_keep_the_bf16_kernel(cuda_device):
    c = to_dev({k: v for k, v in _case(20, 512, 512, 4, 2).items()}, cuda_device)
    flat = torch.empty(c["w13"].numel() + 16, dtype=torch.uint8, device=cuda_device)
    shifted = flat[16:].view(c["w13"].shape)
    shifted.copy_(c["w13"])
    args = (c["w13_scale"], c["w2"], c["w2_scale"], c["topk_ids"], c["topk_w"])
    got = xkb.fused_moe_mxfp4(c["A"], shifted, *args, path="tc")
    ops.check_status(cuda_device)
    assert_within(got, xkb.fused_moe_mxfp4(c["A"], c["w13"], *args), 2e-2, 1e-2, what="shifted", allowed=got.numel() // 2000)
