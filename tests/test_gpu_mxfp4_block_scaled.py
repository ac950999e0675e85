"""The tensor-core MXFP4 kernels - the block-scaled one of decode batches and the one that converts weights to
bf16 - at the edges of their token tiles, of their dispatch and of the activations' split into three terms,
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
    (1, 512, 512, 4, 2, False),        # 8-token tiles, one slot each
    (33, 1024, 512, 4, 2, True),       # 32-token tiles (16.5 slots per expert)
    (24, 512, 512, 4, 2, False),       # 16-token tiles, the most slots per expert
    (64, 512, 512, 4, 2, True),        # the bf16 kernel, from here on
    (65, 512, 512, 4, 2, False),
    (90, 512, 1024, 4, 2, False),
    (112, 1024, 512, 4, 2, True),
    (113, 512, 512, 4, 2, True),
    (700, 512, 512, 3, 2, True),       # several of its blocks, ragged
])
def test_token_tiles(M, hidden, ispp, E, top_k, bias, cuda_device):
    c = _case(M, hidden, ispp, E, top_k, bias)
    got = _call(c, cuda_device)
    ops.check_status(cuda_device)
    want = _want(c)
    assert_within(got, want, 2e-2, 1e-2, what="block-scaled", allowed=max(1, want.numel() // 2000))
    assert torch.equal(got, _call(c, cuda_device))


def test_wide_range_activations(cuda_device):
    """Magnitudes over 2^-20 .. 2^20 inside every block of 32, the large ones in every sum (sums without them:
    test_large_elements_under_zero_weights)."""
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


def _shift(t):
    """The same tensor 16 bytes into a buffer: not on 32 bytes, which the block-scaled kernel's weights need."""
    flat = torch.empty(t.numel() + 16, dtype=t.dtype, device=t.device)
    shifted = flat[16:].view(t.shape)
    shifted.copy_(t)
    assert shifted.data_ptr() % 32 == 16
    return shifted


@pytest.mark.parametrize("power", [14, 16, 18, 24, 30])
@pytest.mark.parametrize("where", ["input", "swiglu"])
@pytest.mark.parametrize("M", [8, 40, 90, 300])
def test_large_elements_under_zero_weights(M, where, power, cuda_device):
    """One element of every 32-block 2^power times as large as the others, and weight codes of 0 at all of them: the
    others alone make the sums, so every bit of theirs counts.  The bf16 products are exact and so must the split be.
    Bound: gate, up, activation and down rows each round to bf16 and may land on the other side of a boundary
    (half a unit in the last place, 2^-9 of the value, each)."""
    c = _case(M, 512, 512, 4, 2)
    g = torch.Generator().manual_seed(power)
    if where == "input":
        at = torch.arange(0, 512, 32) + torch.randint(0, 32, (16,), generator=g)
        c["A"][:, at] = (torch.randn(M, 16, generator=g).sign() * (1 + torch.rand(M, 16, generator=g)) * 2.0 ** power).to(torch.bfloat16)
        _zero_codes(c["w13"], at)
    else:
        at = torch.arange(7, 512, 32)          # gate and up rows 2^(power / 2) times as large each
        for rows in (at, at + 512):
            c["w13_scale"][:, rows] += power // 2
        _zero_codes(c["w2"], at)
    want = _want(c, swiglu_limit=None, fp32_matmul=True).double()
    got = _call(c, cuda_device, swiglu_limit=None)
    ops.check_status(cuda_device)
    rel = float((got.cpu().double() - want).norm() / want.norm())
    assert rel <= 4 * 2.0 ** -9, rel


def _zero_codes(w, columns):
    """Weight codes of 0 in the given K columns of w [E, rows, K / 2] (low nibble = even k)."""
    for k in columns.tolist():
        w[:, :, k // 2] &= 0xF0 if k % 2 == 0 else 0x0F


@pytest.mark.parametrize("shifted", [False, True])
@pytest.mark.parametrize("M,E,top_k", [
    (20, 4, 2),      # decode: 16-token tiles
    (300, 4, 3),     # more than 48 slots per expert: 128-token tiles, ragged blocks, the sort's own kernels
    (513, 2, 1),
])
def test_both_kernels(M, E, top_k, shifted, cuda_device):
    """Weights on 32 bytes and on 16, decode and prefill sized, with biases, a clamp, an expert map and dropped slots."""
    c = _case(M, 1024, 512, E, top_k, bias=True)
    g = torch.Generator().manual_seed(M)
    c["topk_ids"][torch.rand(M, top_k, generator=g) < 0.2] = E + 1
    emap = torch.cat([torch.arange(E, dtype=torch.int32).flip(0), torch.tensor([-1, -1], dtype=torch.int32)])
    want = _want(c, swiglu_limit=2.0, expert_map=emap)
    d = to_dev(c, cuda_device)
    if shifted:
        d["w13"], d["w2"] = _shift(d["w13"]), _shift(d["w2"])
    args = (d["A"], d["w13"], d["w13_scale"], d["w2"], d["w2_scale"], d["topk_ids"], d["topk_w"])
    kw = dict(b13=d["b13"], b2=d["b2"], swiglu_limit=2.0, expert_map=emap.to(cuda_device), path="tc")
    got = xkb.fused_moe_mxfp4(*args, **kw)
    ops.check_status(cuda_device)
    assert_within(got, want, 2e-2, 1e-2, what="tc", allowed=max(1, want.numel() // 2000))
    assert torch.equal(got, xkb.fused_moe_mxfp4(*args, **kw))


@pytest.mark.parametrize("shifted", [False, True])
def test_scale_bytes_above_190(shifted, cuda_device):
    """Scale bytes 191 .. 254 (weights of 2^64 and more) are reported in batches of more than 48 slots per expert,
    and are ordinary weights in smaller ones."""
    def run(M, byte):
        c = _case(M, 512, 512, 4, 2)
        c["w2_scale"][:, 5, 3] = byte
        d = to_dev(c, cuda_device)
        if shifted:
            d["w13"], d["w2"] = _shift(d["w13"]), _shift(d["w2"])
        got = xkb.fused_moe_mxfp4(d["A"], d["w13"], d["w13_scale"], d["w2"], d["w2_scale"], d["topk_ids"], d["topk_w"])
        return c, got

    for byte in (191, 200):
        for M in (104, 300):          # 52 and 150 slots per expert
            run(M, byte)
            with pytest.raises(RuntimeError, match="191..254"):
                ops.check_status(cuda_device)
        c, got = run(60, byte)
        ops.check_status(cuda_device)
        want = _want(c)
        assert_within(got, want, 2e-2, 1e-2, what="decode", allowed=max(1, want.numel() // 2000))
    c, got = run(300, 190)
    ops.check_status(cuda_device)
    want = _want(c)
    assert_within(got, want, 2e-2, 1e-2, what="190", allowed=max(1, want.numel() // 2000))
