"""The routing sort of one cluster: around the sizes where a warp's segment grows, where the cluster ends, and where the
callers' workspace starts to matter; runs of one expert, dropped slots, expert counts around the warps and the block.
Bit-exact against the oracle."""

import pytest
import torch

from tests.test_gpu_align import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("numel", [1025, 2049, 8191, 8192, 8193, 12345, 16383, 16384, 16385])
@pytest.mark.parametrize("E,block", [(1, 1), (31, 16), (32, 64), (48, 128), (256, 16), (1024, 8)])
@pytest.mark.parametrize("kind", ["uniform", "one", "dropped"])
def test_sizes(numel, E, block, kind, cuda_device):
    g = torch.Generator().manual_seed(numel + E)
    ids = torch.randint(0, E, (numel, 1), generator=g, dtype=torch.int32)
    if kind == "one":          # long runs of one expert beside the others
        ids = torch.where(torch.rand(numel, 1, generator=g) < 0.9, torch.full_like(ids, E - 1), ids)
    if kind == "dropped":
        ids = torch.where(torch.rand(numel, 1, generator=g) < 0.5, torch.full_like(ids, E), ids)
    check(ids, block, E, False, cuda_device)
