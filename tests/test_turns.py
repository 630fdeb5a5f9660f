"""How the blocks of the zero-copy collectives take turns along a buffer (``csrc/tl/nvlink/nvl_kernels.cu``), on the CPU."""
import ctypes as C

import pytest

from xccl_b200 import _capi as K


def _tile(n, blocks, most):
    fn = K.load().xccl_nvlink_turn_tile
    fn.restype, fn.argtypes = C.c_size_t, [C.c_size_t] * 3
    return fn(n, blocks, most)


@pytest.mark.parametrize("most", [512, 1024, 2048])
@pytest.mark.parametrize("blocks", [1, 16, 37, 74, 128, 296])
def test_every_block_has_its_share(blocks, most):
    for n in (0, 1, 31, 33, 4096, 4097, 49152, 65536, 131072, 131077, 1 << 20, (1 << 26) + 5):
        tile = _tile(n, blocks, most)
        assert 32 <= tile <= most and tile % 32 == 0
        tiles = -(-n // tile)
        share = [sum(min(tile, n - t * tile) for t in range(b, tiles, blocks)) for b in range(blocks)]
        assert sum(share) == n
        # as few turns as tiles of `most` packs allow (one per block and piece where that holds a block's part), and nobody has
        # more than an even part of the packs, up to 32 packs a turn
        per = -(-n // blocks)
        turns = -(-per // most)
        assert -(-tiles // blocks) == turns
        assert max(share) <= per + 32 * turns
        assert sum(s > 0 for s in share) >= min(blocks, n // (per // max(turns, 1) + 32))   # a tile is rounded up by 31 at most


def test_segments_and_shares_that_fixed_tiles_cut_unevenly():
    """A segment of 1 MiB for 128 blocks: all of them, not 32; the share of 131072 packs for 37 blocks: seven passes, not eight."""
    assert -(-65536 // _tile(65536, 128, 2048)) == 128
    tile = _tile(131072, 37, 512)
    assert -(-(-(-131072 // tile)) // 37) == 7
