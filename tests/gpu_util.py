"""Helpers shared by the GPU parity tests."""

import torch

from oracle import moe_oracle as oracle
from xkernels_b200 import _lib


def to_dev(case: dict, dev) -> dict:
    return {k: (v.to(dev) if isinstance(v, torch.Tensor) else v) for k, v in case.items()}


def int4_tile(M: int, E: int, top_k: int) -> int:
    """The token tile of an INT4 call on the tensor cores."""
    return _lib.load().xkb_int4_token_tile(M * top_k, E, top_k)


def mxfp4_tile(M: int, E: int, top_k: int) -> int:
    """The same of an MXFP4 call whose weights lie on 32 bytes (128: the kernel that converts to bf16)."""
    return _lib.load().xkb_mxfp4_token_tile(M * top_k, E)


def poisoned_workspace(query: str, *dims, device) -> torch.Tensor:
    """A call's workspace, every bf16 and fp32 in it a NaN: what the call uses without writing it shows."""
    return torch.full((getattr(_lib.load(), query)(*dims),), 0xFF, dtype=torch.uint8, device=device)


def assert_within(actual: torch.Tensor, expected: torch.Tensor, rtol: float, atol: float, what: str = "",
                  allowed: int = 0):
    a, e = actual.detach().cpu(), expected.detach().cpu()
    assert a.shape == e.shape and a.dtype == e.dtype, f"{what}: {a.shape}/{a.dtype} vs {e.shape}/{e.dtype}"
    bad = oracle.count_violations(a, e, rtol, atol)
    if bad > allowed:
        d = (a.double() - e.double()).abs()
        idx = int(d.argmax())
        raise AssertionError(
            f"{what}: {bad}/{a.numel()} elements outside |a-e| <= {atol} + {rtol}|e| (allowed {allowed}); "
            f"max abs diff {d.max().item():.4g} at flat index {idx}: got {a.flatten()[idx].item()}, "
            f"want {e.flatten()[idx].item()}")
