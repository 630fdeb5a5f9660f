"""How the tensor-parallel GEMM lays a launch out (``csrc/fused/tp_gemm.cu``), asked on the CPU: pairs or single CTAs, how
many of them walk tiles, and the tile width that is chosen for exactly these walkers."""
import pytest

from xccl_b200 import _capi as K

NONE, ALLGATHER, REDUCE_SCATTER = 0, 1, 2


def _walk(M, tp, comm, ctas, gemm, copy_mode=0, may_pair=1):
    v = K.load().xccl_tp_tile_walk(M, tp, comm, ctas, gemm, copy_mode, may_pair)
    return v < 0, abs(v)


def _cost(M, N, bn, walkers):
    tiles = -(-M // 256) * (-(-N // bn))
    return -(-tiles // walkers) * (bn + 110)


@pytest.mark.parametrize("ctas", [2, 3, 18, 37, 49, 74, 148])
def test_walkers_are_those_of_the_launch(ctas):
    for copy in range(0, ctas // 4 + 1):
        pair, walkers = _walk(4096, 4, ALLGATHER, ctas, ctas - copy)
        # the grid has an even number of CTAs, the copiers take an even number of them
        want = (ctas - ctas % 2 - (copy + copy % 2)) // 2
        if want >= 1:
            assert (pair, walkers) == (True, want)
        assert _walk(4096, 4, ALLGATHER, ctas, ctas - copy, may_pair=0) == (False, ctas - copy)
        assert _walk(4096, 4, ALLGATHER, ctas, ctas - copy, copy_mode=1)[1] == ctas // 2     # the copiers are warps
    # shards of 384 rows are no whole 256-row tiles; without communication any row count is
    assert _walk(1536, 4, REDUCE_SCATTER, ctas, ctas) == (False, ctas)
    assert _walk(1536, 4, NONE, ctas, ctas) == (True, ctas // 2)


def test_width_is_chosen_for_the_walkers_of_the_launch():
    """Four ranks of 37 CTAs with nine that copy: the odd one copies too and 13 pairs walk, not 14. 28 tiles of 160 columns
    would be two waves of 14 but are three of 13."""
    M, N, k = 1024, 1024, 3072
    pair, walkers = _walk(M, 4, ALLGATHER, 37, 37 - 9)
    assert (pair, walkers) == (True, 13)
    bn = K.load().xccl_tp_tile_cols(M, N, k, 1, int(pair), walkers)
    assert _cost(M, N, bn, walkers) == min(_cost(M, N, b, walkers) for b in range(64, 257, 32)) and bn == 192


@pytest.mark.parametrize("M,N,k,swiglu,walkers,cols", [
    (512, 1280, 1280, 0, 37, 160),       # reduce-scatter, four ranks: 20 tiles on 37 walkers, 32 of 160 columns
    (512, 8192, 1280, 0, 37, 256),       # 128 tiles, four waves whatever the width
    (512, 5120, 1280, 1, 28, 256),       # three waves of 80 tiles; narrower ones promise 12 %, too little with SwiGLU
    (256, 512, 1024, 1, 74, 64),         # four tiles, or sixteen
    (2048, 512, 4096, 0, 148, 64)])
def test_width_of_single_cta_tiles(M, N, k, swiglu, walkers, cols):
    """128-row tiles: the least (waves x (columns + 370)), taken if it saves 10 % (20 % with SwiGLU)."""
    def cost(b):
        tiles = -(-M // 128) * (-(-(N // 2) // (b // 2)) if swiglu else -(-N // b))
        return -(-tiles // walkers) * (b + 370)
    got = K.load().xccl_tp_tile_cols(M, N, k, swiglu, 0, walkers)
    least = min(range(64, 257, 32), key=lambda b: (cost(b), -b))
    assert got == (least if cost(least) <= (0.8 if swiglu else 0.9) * cost(256) else 256) == cols


@pytest.mark.parametrize("N", [8, 32, 40, 256, 264, 1000, 4096, 8200])
def test_arrivals_of_a_row_block_do_not_depend_on_the_tile_width(N):
    """The owner of a row block waits for a count that a rank on another device, with other tiles, reaches as well."""
    fn = K.load().xccl_tp_rs_arrivals
    total = fn(N, 0, -1)
    for bn in range(32, 257, 32):
        parts = [fn(N, bn, nb) for nb in range(-(-N // bn))]
        assert all(p > 0 for p in parts) and sum(parts) == total


@pytest.mark.parametrize("tp", [3, 4, 8])
def test_copy_ctas_of_emulated_ranks(tp):
    """Fewer copy CTAs for wide products, but not where a shard is one 128-row block: its rows are wanted at once."""
    fn, ctas = K.load().xccl_tp_copy_ctas, 148 // tp
    most = min(16, ctas // 4)
    for columns in (512, 2048, 7168, 28672):
        assert fn(tp, 0, 16, 1, 128, columns, ctas) == most
        assert fn(tp, 0, 16, 0, 1024, columns, ctas) == most            # real ranks, or a number that was asked for
        assert fn(tp, 0, 16, 1, 256, columns, ctas) == max(1, min(most, max(2, -(-28672 // columns))))
        assert fn(tp, 1, 16, 1, 256, columns, ctas) == 0 and fn(1, 0, 16, 1, 256, columns, 148) == 0
