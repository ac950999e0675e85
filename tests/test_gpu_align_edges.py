"""moe_align_block_size where its launch shape changes: one CTA up to 1024 slots, then one round per
chunk up to 148 x 1024 slots, then several rounds per chunk.  Bit-exact against the oracle."""

import pytest
import torch

import xkernels_b200 as xkb
from oracle import moe_oracle as oracle
from tests.test_gpu_align import check

from xkernels_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("numel", [1, 31, 1023, 1024, 1025, 148 * 1024, 148 * 1024 + 1, 3 * 148 * 1024 - 5])
@pytest.mark.parametrize("E,block", [(1, 16), (48, 16), (1024, 8), (257, 100)])
def test_edges(numel, E, block, cuda_device):
    g = torch.Generator().manual_seed(numel + E)
    ids = torch.randint(0, E + 1, (numel, 1), generator=g, dtype=torch.int32)   # E: an id outside [0, E)
    ids = torch.where((ids == E) & (torch.rand(numel, 1, generator=g) < 0.5), torch.zeros_like(ids), ids)
    check(ids, block, E, False, cuda_device)


@pytest.mark.parametrize("numel", [7, 1024, 1025, 4097, 8192])
@pytest.mark.parametrize("E,block", [(48, 16), (1024, 8)])
@pytest.mark.parametrize("mapped", [False, True])
def test_no_workspace_up_to_8192_slots(numel, E, block, mapped, cuda_device):
    """C callers may pass no workspace there.  Above, the call is refused."""
    lib = _lib.load()
    g = torch.Generator().manual_seed(numel + E)
    ids = torch.randint(0, E + 1, (numel, 1), generator=g, dtype=torch.int32)
    emap, local = None, ids
    if mapped:
        emap = torch.randperm(E, generator=g).to(torch.int32)
        emap[::3] = -1
        local = torch.cat([emap, torch.tensor([-1], dtype=torch.int32)])[ids.long()]
        local = torch.where(local < 0, torch.full_like(local, E), local)
    want = oracle.align_block_size(local.numpy(), block, E, truncate=False)
    d_ids, d_map = ids.to(cuda_device), None if emap is None else emap.to(cuda_device)
    pad = numel + (E + 1) * (block - 1)
    out = [torch.full((n,), -7, dtype=torch.int32, device=cuda_device) for n in (pad, -(-pad // block), 1)]

    def call(n):
        return lib.xkb_moe_align_block_size(d_ids.data_ptr(), n, E, block, 0 if d_map is None else d_map.data_ptr(),
                                            0 if d_map is None else E, *(t.data_ptr() for t in out), 0, 0, 0,
                                            torch.cuda.current_stream().cuda_stream)

    assert call(numel) == 0, lib.xkb_last_error()
    for got, exp in zip(out, want):
        assert torch.equal(got.cpu(), torch.as_tensor(exp).to(torch.int32).reshape(-1))
    assert call(8193) != 0 and b"workspace" in lib.xkb_last_error()


@pytest.mark.parametrize("numel", [1024, 1025, 5000])
def test_outputs_own_no_scratch(numel, cuda_device):
    """What a caller keeps or saves is the result alone: the kernels' scratch is not part of its storage."""
    ids = torch.zeros(numel, 1, dtype=torch.int32, device=cuda_device)
    for t in xkb.moe_align_block_size(ids, 16, 48, truncate=False):
        assert t.untyped_storage().nbytes() == 4 * t.numel()
