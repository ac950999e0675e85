"""The arrays with one entry per token block in a fused call's workspace, which the routing sort writes in full: long
enough at every block size from 8 to 256 (the token tiles), also where there are fewer slots than experts."""

import pytest

BLOCKS = [8, 16, 32, 64, 128, 256]


@pytest.fixture(scope="module")
def lib():
    from xkernels_b200 import _lib
    from xkernels_b200.build import build

    build()
    return _lib.load()


def test_block_arrays_hold_every_block_size(lib):
    for E in [*range(1, 70), 127, 128, 129, 255, 256, 257, 264, 272, 288, 384, 385, 416, 512, 513, 1023, 1024]:
        for numel in [*range(1, 300), 360, 500, 511, 512, 513, 1024, 2047, 2048, 100_003]:
            room = lib.xkb_routing_blocks(numel, E)
            for block in BLOCKS:
                need = -(-(numel + (E + 1) * (block - 1)) // block)   # entries that the sort writes
                assert need <= room, f"E={E} numel={numel} block={block}: {need} entries, room for {room}"


def test_negative_sizes(lib):
    assert lib.xkb_routing_blocks(-1, 4) == -1 and lib.xkb_routing_blocks(4, -1) == -1
