"""moe_align_block_size where its launch shape changes: one CTA up to 1024 slots, then one round per
chunk up to 148 x 1024 slots, then several rounds per chunk.  Bit-exact against the oracle."""

import pytest
import torch

from tests.test_gpu_align import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("numel", [1, 31, 1023, 1024, 1025, 148 * 1024, 148 * 1024 + 1, 3 * 148 * 1024 - 5])
@pytest.mark.parametrize("E,block", [(1, 16), (48, 16), (1024, 8), (257, 100)])
def test_edges(numel, E, block, cuda_device):
    g = torch.Generator().manual_seed(numel + E)
    ids = torch.randint(0, E + 1, (numel, 1), generator=g, dtype=torch.int32)   # E: an id outside [0, E)
    ids = torch.where((ids == E) & (torch.rand(numel, 1, generator=g) < 0.5), torch.zeros_like(ids), ids)
    check(ids, block, E, False, cuda_device)
