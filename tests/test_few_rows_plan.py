"""How the few-rows GEMM cuts its work (``csrc/fused/tp_skinny.cu``), walked on the CPU."""
import ctypes as C

import pytest

from xccl_b200 import _capi as K

FIELDS = ("mn", "tiles", "splits", "kblocks", "stages", "nbuf", "cols", "tmem_cols", "chunk", "smem", "occ")


def _plan(M, N, K_, fp8, swiglu, sms=148):
    out = (C.c_int * len(FIELDS))()
    fn = K.load().xccl_tp_skinny_plan
    fn.restype = C.c_int
    return dict(zip(FIELDS, out)) if fn(M, N, K_, int(fp8), int(swiglu), sms, out) else None


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("swiglu", [False, True])
def test_plan_covers_the_product_and_fits_the_sm(fp8, swiglu):
    for M in list(range(1, 129)):
        for N in (8, 128, 1000, 8192, 28672, 60000):
            for K_ in (8, 128, 520, 8192, 28672):
                if fp8 and (K_ % 128 or N % 128):
                    continue
                p = _plan(M, N, K_, fp8, swiglu)
                assert p is not None
                mats = 2 if swiglu else 1
                assert M <= p["mn"] <= 128 and p["mn"] % (32 if fp8 else 16) == 0
                assert (p["tiles"] - 1) * 128 < N <= p["tiles"] * 128
                # every K block belongs to exactly one CTA and none is without work
                cut = [s * p["kblocks"] // p["splits"] for s in range(p["splits"] + 1)]
                assert 1 <= p["splits"] <= 8 and cut[-1] == p["kblocks"] and all(a < b for a, b in zip(cut, cut[1:]))
                # shared memory and tensor memory of the CTAs that share an SM
                assert (p["smem"] + 1024 + 64) * p["occ"] <= 228 * 1024
                assert p["tmem_cols"] * p["occ"] <= 512 and p["nbuf"] * p["cols"] <= p["tmem_cols"]
                assert p["tmem_cols"] & (p["tmem_cols"] - 1) == 0 and p["cols"] >= mats * p["mn"]
                ring = p["stages"] * (16384 * mats + p["mn"] * 128)
                assert p["stages"] >= 2 and 16 <= p["chunk"] <= p["mn"] and p["chunk"] % 16 == 0
                assert p["chunk"] * 512 * mats <= ring


def test_more_rows_than_one_mma_are_left_to_the_large_kernel():
    assert _plan(129, 8192, 8192, False, False) is None
    assert _plan(0, 8192, 8192, False, False) is None


def test_a_cluster_the_device_does_not_place_becomes_a_smaller_one():
    """A partitioned device may place no cluster of eight: the call is served with fewer CTAs per tile instead of refused.
    One CTA always fits."""
    fn = K.load().xccl_tp_skinny_cluster
    for splits in range(1, 9):
        assert fn(splits, 0x1ff) == splits
        assert fn(splits, 0) == 1
        for most in range(1, 9):
            got = fn(splits, (2 << most) - 1)
            assert 1 <= got <= min(splits, most)
            assert got == splits or got >= min(splits, most) / 2


# clusters of 1 .. 8 CTAs that a B200 holds at a time, with one and with two CTAs per SM
B200 = {1: (0, 148, 74, 45, 33, 26, 22, 15, 15), 2: (0, 296, 148, 93, 71, 56, 45, 37, 33)}


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("swiglu", [False, True])
def test_tiles_run_in_one_wave_of_the_clusters_a_gpu_holds(fp8, swiglu):
    """K is shared only while all tiles' clusters are resident at once: a second wave costs more than a longer K loop."""
    for M in (1, 16, 33, 64, 100, 128):
        for N in range(128, 40001, 128):
            for K_ in (128, 512, 2048, 8192, 28672):
                p = _plan(M, N, K_, fp8, swiglu)
                assert p["splits"] == 1 or (p["tiles"] <= B200[p["occ"]][p["splits"]] and p["kblocks"] >= 4 * p["splits"])


@pytest.mark.parametrize("M,N,K_,fp8,swiglu,splits", [
    (16, 8192, 8192, False, False, 4), (128, 8192, 28672, False, False, 4), (64, 7168, 8192, True, False, 2),
    (128, 6144, 2048, False, False, 3), (128, 6144, 4096, False, True, 3), (128, 4096, 2048, False, False, 4),
    (64, 2048, 8192, True, False, 4), (16, 1024, 8192, False, False, 8), (128, 28672, 8192, False, True, 1)])
def test_share_at_the_measured_sizes(M, N, K_, fp8, swiglu, splits):
    assert _plan(M, N, K_, fp8, swiglu)["splits"] == splits


def _plan_rows(M, N, K_, fp8, swiglu, sms=148):
    out = (C.c_int * len(FIELDS))()
    fn = K.load().xccl_tp_skinny_plan_rows
    fn.restype = C.c_int
    n = fn(M, N, K_, int(fp8), int(swiglu), sms, out)
    return dict(zip(FIELDS, out), blocks=n) if n else None


@pytest.mark.parametrize("fp8,swiglu", [(False, False), (True, False), (True, True)])
def test_blocks_of_rows_cover_the_rows_and_keep_to_the_rule(fp8, swiglu):
    taken = 0
    for M in (1, 128, 129, 200, 256, 257, 500, 1024, 1500, 4000, 8192):
        for N in (128, 384, 1024, 2944, 7168):
            for K_ in (128, 512, 1536, 4096, 8192):
                p = _plan_rows(M, N, K_, fp8, swiglu)
                if M <= 128:
                    assert p is not None and p.pop("blocks") == 1 and p == _plan(M, N, K_, fp8, swiglu)
                    continue
                if p is None:
                    continue
                taken += 1
                # every row in one block, no block without rows, and as many CTAs as the measured rule allows
                assert p["mn"] <= 128 and (p["blocks"] - 1) * p["mn"] < M <= p["blocks"] * p["mn"]
                ctas = p["blocks"] * p["tiles"] * p["splits"]
                assert p["splits"] >= (1 if fp8 and not swiglu else 2 if fp8 else 3)
                assert ctas <= 148 if fp8 else p["kblocks"] >= 24 and ctas <= 2 * 148
    assert taken > 20
    assert _plan_rows(300, 1024, 8192, False, True) is None      # bf16 SwiGLU stays with the large kernel
    assert _plan_rows(1 << 30, 128, 128, True, False) is None


@pytest.mark.parametrize("M,N,K_,taken", [
    # large / few-rows kernel in us: 14.4 / 18.5, 21.4 / 26.7, 24.7 / 30.0, 34.9 / 41.6, 20.7 / 24.6, 13.9 / 14.4 (25 K blocks)
    (480, 1528, 1672, False), (379, 2048, 3480, False), (1006, 736, 4664, False), (1585, 520, 7176, False), (232, 2992, 3240, False),
    (1145, 288, 1592, False),
    # 33.5 / 18.8, 32.9 / 23.0, 26.7 / 22.5, 18.6 / 18.6
    (206, 576, 7160, True), (370, 1280, 7032, True), (480, 1328, 4984, True), (1654, 336, 3016, True)])
def test_blocks_of_rows_only_where_no_measured_product_is_slower(M, N, K_, taken):
    p = _plan_rows(M, N, K_, False, False)
    assert (p is not None) == taken
    if taken:
        assert p["blocks"] * p["tiles"] * p["splits"] <= 133 and p["kblocks"] > 32


@pytest.mark.parametrize("env,bf16,fp8", [({}, 1, 1), ({"XCCL_TP_GEMM_BN": "64"}, 0, 1), ({"XCCL_TP_GEMM_PAIR": "n"}, 0, 0)])
def test_tiles_that_are_asked_for_serve_more_than_one_block_of_rows(env, bf16, fp8):
    """A forced tile width or single CTAs: products of more than 128 rows run in the kernel with these tiles, as its options say
    (they are read once per process); up to 128 rows are the few-rows kernel's in any case."""
    import os
    import subprocess
    import sys
    from pathlib import Path
    script = ("from xccl_b200 import _capi as K\nf = K.load().xccl_tp_skinny_takes\n"
              "print(f(640, 232, 4104, 0, 0, 148), f(256, 512, 1536, 1, 0, 148), f(100, 512, 1536, 0, 0, 148), f(100, 512, 1536, 1, 0, 148))")
    full = {k: v for k, v in os.environ.items() if not k.startswith("XCCL_TP_")}
    full.update(env, PYTHONPATH=str(Path(__file__).resolve().parent.parent))
    r = subprocess.run([sys.executable, "-c", script], env=full, capture_output=True, text=True, timeout=120)
    assert r.stdout.split() == [str(bf16), str(fp8), "1", "1"], r.stdout + r.stderr[-2000:]
