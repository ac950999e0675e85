"""fused_moe_int4_ffn (gate_up GEMM -> SwiGLU -> down GEMM -> combine in one call) on the GPU, through
the C-ABI, against fixtures made by composing the reference's own ops and against the oracle.
Tolerance: the INT4 op spec's bf16 tolerance |a-e| <= 1e-2 + 2e-2|e| (registry/ops/moe_int4_w4a16.spec.json:30-41);
the kernels round where the composition rounds, so only fp32 accumulation order differs and, as for
MXFP4, an occasional element lands on the other side of a bf16 rounding boundary of an intermediate."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle
from tests.golden.golden_io import load_case
from tests.gpu_util import assert_within, to_dev
from xkernels_b200 import ops, synth

pytestmark = pytest.mark.gpu
KEYS = ("A", "w13_packed", "w13_scale", "w2_packed", "w2_scale", "topk_ids", "topk_w")


def call(c, dev, **kw):
    d = to_dev({k: c[k] for k in KEYS}, dev)
    return xkb.fused_moe_int4_ffn(*(d[k] for k in KEYS), **kw)


@pytest.mark.parametrize("name", ["int4_ffn_small", "int4_ffn_tc", "int4_ffn_fp32"])
@pytest.mark.parametrize("path", ["auto", "simt"])
def test_golden(name, path, cuda_device):
    c = load_case(name)
    out = call(c, cuda_device, swiglu_limit=c["swiglu_limit"] or None, path=path)
    ops.check_status(cuda_device)
    tol = (2e-2, 1e-2) if c["A"].dtype == torch.bfloat16 else (1e-3, 1e-3)
    assert_within(out, c["out"], *tol, what=f"{name}/{path}", allowed=max(1, c["out"].numel() // 2000))


@pytest.mark.parametrize("M,hidden,inter,E,top_k", [
    (16, 512, 256, 8, 2),       # 4 slots per expert: 16-token tiles
    (40, 768, 512, 8, 4),       # 20 per expert: 64-token tiles
    (64, 256, 256, 4, 2),       # 32 per expert: the same
    (300, 512, 256, 3, 2),      # 200 per expert: 128-token tiles, ragged last blocks
    (7, 2048, 1024, 48, 8),     # decode-like: mostly empty experts
])
def test_tensor_core_path_against_oracle(M, hidden, inter, E, top_k, cuda_device):
    g = torch.Generator().manual_seed(M + hidden)
    A = torch.randn(M, hidden, generator=g).to(torch.bfloat16)
    w13, s13 = synth.int4_weights(E, 2 * inter, hidden, 32, seed=M)
    w2, s2 = synth.int4_weights(E, hidden, inter, 32, seed=M + 1)
    # keep the layer's outputs O(1), where the spec's absolute tolerance of 1e-2 is meant to apply: the
    # per-slot results are bf16 numbers, and with outputs of ~40 (the raw synthetic scales at these K)
    # one rounding step of a single slot row is 0.25, far above it
    s13 = (s13.float() * (256.0 / hidden) ** 0.5).to(torch.bfloat16)
    s2 = (s2.float() * (16.0 / inter)).to(torch.bfloat16)
    ids, w = synth.routing(M, E, top_k, seed=hidden)
    c = {"A": A, "w13_packed": w13, "w13_scale": s13, "w2_packed": w2, "w2_scale": s2, "topk_ids": ids, "topk_w": w}
    want = oracle.moe_int4_ffn(A, w13, s13, w2, s2, ids, w, 32)
    got = call(c, cuda_device, path="tc")
    ops.check_status(cuda_device)
    assert_within(got, want, 2e-2, 1e-2, what="tc", allowed=max(1, want.numel() // 2000))
    simt = call(c, cuda_device, path="simt")
    assert_within(simt, want, 2e-2, 1e-2, what="simt", allowed=max(1, want.numel() // 2000))
    assert torch.equal(got, call(c, cuda_device, path="tc")), "second run differs: the layer must be deterministic"


def test_dropped_slots_and_refused_shapes(cuda_device):
    cfg_M, hidden, inter, E, top_k = 24, 256, 256, 6, 3
    g = torch.Generator().manual_seed(5)
    A = torch.randn(cfg_M, hidden, generator=g).to(torch.bfloat16)
    w13, s13 = synth.int4_weights(E, 2 * inter, hidden, 32, seed=1)
    w2, s2 = synth.int4_weights(E, hidden, inter, 32, seed=2)
    ids, w = synth.routing(cfg_M, E, top_k, seed=3)
    ids = ids.clone()
    ids[0] = -1
    ids[1, 0] = E + 2
    emap = torch.cat([torch.arange(E, dtype=torch.int32), torch.tensor([-1], dtype=torch.int32)])
    o_ids = torch.where((ids < 0) | (ids >= E), torch.full_like(ids, E), ids)
    want = oracle.moe_int4_ffn(A, w13, s13, w2, s2, o_ids, w, 32, expert_map=emap)
    c = {"A": A, "w13_packed": w13, "w13_scale": s13, "w2_packed": w2, "w2_scale": s2, "topk_ids": ids, "topk_w": w}
    for path in ("tc", "simt"):
        got = call(c, cuda_device, path=path)
        assert_within(got, want, 2e-2, 1e-2, what=f"dropped slots/{path}", allowed=2)
        assert bool((got[0] == 0).all())
    with pytest.raises(RuntimeError, match="tcgen05"):
        small = load_case("int4_ffn_small")          # hidden 64: not a multiple of 256
        call(small, cuda_device, path="tc")
    with pytest.raises(RuntimeError, match="CUDA"):
        xkb.fused_moe_int4_ffn(A, w13, s13, w2, s2, ids, w)
