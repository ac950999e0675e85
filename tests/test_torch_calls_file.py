"""The call path of the small ops is a file of its own, built for one torch and one Python: where there is none for those
that run, the ops take their Python form, and the library is built all the same."""

import sys

import pytest
import torch

import xkernels_b200 as xkb
from xkernels_b200 import _lib, build


def test_the_name_says_what_it_was_built_for():
    assert torch.__version__ in _lib.CALLS_PATH.name and sys.implementation.cache_tag in _lib.CALLS_PATH.name


def test_a_missing_file_leaves_the_python_form(monkeypatch, tmp_path):
    build.build()
    monkeypatch.setattr(_lib, "_calls", None)
    monkeypatch.setattr(_lib, "CALLS_PATH", tmp_path / "none.so")
    calls = _lib.load_calls()
    x, ids, y = torch.zeros(2, 4), torch.zeros(2, 2, dtype=torch.int32), torch.zeros(2, 2, 8)
    assert calls.topk_softmax(x, 2, True) is None and calls.moe_align_block_size(ids, 16, 4) is None
    assert calls.moe_sum_reduce(y, None, 1.0) is None
    for call in (lambda: xkb.topk_softmax(x, 2), lambda: xkb.moe_align_block_size(ids, 16, 4), lambda: xkb.moe_sum_reduce(y)):
        with pytest.raises(RuntimeError, match="needs CUDA tensors"):   # the Python form's own refusal
            call()


def test_no_compiler_is_a_warning(monkeypatch, tmp_path):
    monkeypatch.setattr(build, "CALLS_PATH", tmp_path / "calls.so")
    monkeypatch.setattr(build, "OBJ_DIR", tmp_path)
    monkeypatch.setenv("CXX", str(tmp_path / "no-such-compiler"))
    with pytest.warns(UserWarning, match="Python form"):
        assert build.build_calls() is False
    assert not build.calls_are_current()
    monkeypatch.setattr(build, "build_library", lambda force, verbose: None)
    with pytest.warns(UserWarning, match="Python form"):
        assert build.build() == build.LIB_PATH


@pytest.mark.gpu
def test_same_results_without_it(monkeypatch, cuda_device):
    x = torch.randn(9, 48, device=cuda_device)
    ids = torch.randint(0, 48, (300, 8), dtype=torch.int32, device=cuda_device)
    y, w = torch.randn(9, 4, 72, device=cuda_device), torch.rand(9, 4, device=cuda_device)

    def results():
        return [*xkb.topk_softmax(x, 4), *xkb.moe_align_block_size(ids, 16, 48), xkb.moe_sum_reduce(y, w)]

    native = results()
    monkeypatch.setattr(_lib, "_calls", _lib.PythonCalls)
    assert all(torch.equal(a, b) for a, b in zip(native, results()))
