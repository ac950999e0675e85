"""The native call path of the small ops against their Python form: which calls it serves, that the others reach the Python
form, the same results bit for bit, the same refusals."""

import contextlib

import numpy as np
import pytest
import torch
from torch.overrides import TorchFunctionMode

import xkernels_b200 as xkb
from xkernels_b200 import _lib

pytestmark = pytest.mark.gpu


class _Passive(TorchFunctionMode):
    """A mode that changes nothing: calls under it belong to the Python form."""

    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def _both(fn):
    direct = fn()
    with _Passive():
        python = fn()
    direct, python = (r if isinstance(r, tuple) else (r,) for r in (direct, python))
    assert len(direct) == len(python)
    for a, b in zip(direct, python):
        assert a.dtype == b.dtype and a.shape == b.shape and a.is_contiguous() and torch.equal(a, b)


@pytest.mark.parametrize("M,E,k,dtype", [(0, 8, 2, torch.float32), (1, 1, 1, torch.bfloat16), (7, 48, 4, torch.float16), (300, 256, 8, torch.bfloat16)])
@pytest.mark.parametrize("renorm", [True, False])
def test_router(M, E, k, dtype, renorm, cuda_device):
    x = torch.randn(M, E, generator=torch.Generator().manual_seed(M)).to(dtype).to(cuda_device)
    assert _lib.load_calls().topk_softmax(x, k, renorm) is not None
    _both(lambda: xkb.topk_softmax(x, k, renorm))


@pytest.mark.parametrize("M,k,E,block", [(1, 1, 1, 1), (5, 2, 8, 16), (128, 8, 48, 16), (129, 8, 48, 64), (2000, 8, 256, 128)])
@pytest.mark.parametrize("truncate", [True, False])
def test_align(M, k, E, block, truncate, cuda_device):
    ids = torch.randint(-1, E + 1, (M, k), generator=torch.Generator().manual_seed(M), dtype=torch.int32).to(cuda_device)
    assert _lib.load_calls().moe_align_block_size(ids, block, E) is not None
    _both(lambda: xkb.moe_align_block_size(ids, block, E, truncate=truncate))


@pytest.mark.parametrize("M,k,H", [(0, 2, 8), (1, 1, 8), (9, 8, 72), (33, 6, 100)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("w_dtype", [None, torch.float32, torch.bfloat16])
def test_reduce(M, k, H, dtype, w_dtype, cuda_device):
    g = torch.Generator().manual_seed(H)
    y = torch.randn(M, k, H, generator=g).to(dtype).to(cuda_device)
    w = None if w_dtype is None else torch.rand(M, k, generator=g).to(w_dtype).to(cuda_device)
    assert _lib.load_calls().moe_sum_reduce(y, w, 0.5) is not None
    _both(lambda: xkb.moe_sum_reduce(y, w, 0.5))


def test_calls_of_the_python_form(cuda_device):
    calls = _lib.load_calls()
    x = torch.randn(16, 64, device=cuda_device)
    ids = torch.randint(0, 8, (16, 2), device=cuda_device)
    y = torch.randn(4, 2, 16, device=cuda_device)
    w, i = xkb.topk_softmax(x, 4)
    strided = x.t().contiguous().t()
    assert calls.topk_softmax(strided, 4, True) is None
    for got in (xkb.topk_softmax(strided, 4), xkb.topk_softmax(torch.nn.Parameter(x), 4), xkb.topk_softmax(x, np.int64(4)),
                xkb.topk_softmax(x, 4, 1)):
        assert torch.equal(got[0], w) and torch.equal(got[1], i)
    assert calls.topk_softmax(x, np.int64(4), True) is None
    assert calls.moe_align_block_size(ids, 16, 8) is None                  # int64 ids
    a, b = xkb.moe_align_block_size(ids, 16, 8), xkb.moe_align_block_size(ids.int(), np.int32(16), 8)
    assert all(torch.equal(p, q) for p, q in zip(a, b))
    assert calls.moe_sum_reduce(y.transpose(0, 1), None, 1.0) is None
    assert calls.moe_sum_reduce(y, None, 1) is None and torch.equal(xkb.moe_sum_reduce(y, None, 1), xkb.moe_sum_reduce(y))
    assert calls.moe_sum_reduce(y, torch.ones(4, 2, device=cuda_device, dtype=torch.float16), 1.0) is None


@pytest.mark.parametrize("mode", [contextlib.nullcontext, _Passive])
def test_refusals(mode, cuda_device):
    x = torch.randn(4, 8, device=cuda_device)
    y = torch.randn(4, 2, 16, device=cuda_device)
    ids = torch.zeros(4, 2, dtype=torch.int32, device=cuda_device)
    with mode():
        for call, error in ((lambda: xkb.topk_softmax(x.cpu(), 2), RuntimeError), (lambda: xkb.topk_softmax(x, 0), ValueError),
                            (lambda: xkb.topk_softmax(x, 9), ValueError), (lambda: xkb.topk_softmax(x.double(), 2), TypeError),
                            (lambda: xkb.topk_softmax([1], 2), TypeError), (lambda: xkb.topk_softmax(x[0], 2), ValueError),
                            (lambda: xkb.topk_softmax(torch.zeros(1, 2000, device=cuda_device), 2), _lib.XkbError),
                            (lambda: xkb.moe_align_block_size(ids, 0, 8), ValueError),
                            (lambda: xkb.moe_align_block_size(ids, 16, 2000), _lib.XkbError),
                            (lambda: xkb.moe_sum_reduce(y[0]), ValueError), (lambda: xkb.moe_sum_reduce(y.half()), TypeError),
                            (lambda: xkb.moe_sum_reduce(y, torch.ones(4, 3, device=cuda_device)), ValueError)):
            with pytest.raises(error):
                call()


def test_capture(cuda_device):
    x = torch.randn(64, 256, device=cuda_device)
    want = xkb.topk_softmax(x, 8)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = xkb.topk_softmax(x, 8)
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
