"""The routing sort of one cluster where paddings and tails are no multiples of a warp: the loops that fill them end lane by
lane right before the cluster's last barrier, which takes whole warps.  Bit-exact against the oracle."""

import pytest
import torch

from tests.test_gpu_align import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("numel,E,block", [(1025, 5, 1000), (3001, 37, 100), (16381, 1000, 77)])
def test_fills_that_end_lane_by_lane(numel, E, block, cuda_device):
    ids = torch.randint(0, E, (numel, 1), generator=torch.Generator().manual_seed(E), dtype=torch.int32)
    for _ in range(5):
        check(ids, block, E, False, cuda_device)
