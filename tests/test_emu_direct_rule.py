"""When the single-GPU emulation runs a collective zero-copy without being asked to (``csrc/tl/nvlink/nvl_emu.cu``), on
the CPU: the rule looks at addresses and sizes only."""
import ctypes as C

import pytest

from xccl_b200 import _capi as K

MB, BASE, STEP = 1 << 20, 1 << 40, 1 << 32


def _pays(coll, n, total, dt=K.DT_FLOAT32, shift=0, src=None, dst=None, out_dt=K.DT_UNSUPPORTED):
    """`total`: bytes of the larger side of all ranks together."""
    es = 2 if dt == K.DT_BFLOAT16 else 4
    per = total // n // (16 * n) * 16 * n
    count = per // es // (n if coll == K.REDUCE_SCATTER else 1)
    length = per // n if coll == K.ALLTOALL else per
    fn = K.load().xccl_nvlink_emu_direct_pays
    fn.argtypes = [C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_size_t, C.c_size_t, C.c_int, C.c_int]
    s = (C.c_void_p * n)(*(src or [BASE + r * STEP + shift for r in range(n)]))
    d = (C.c_void_p * n)(*(dst or [BASE + (n + r) * STEP for r in range(n)]))
    return bool(fn(n, coll, s, d, count, length, dt, out_dt))


@pytest.mark.parametrize("coll,n,dt,staged,direct", [
    (K.ALLREDUCE, 2, K.DT_FLOAT32, 12, 17), (K.ALLREDUCE, 4, K.DT_BFLOAT16, 4, 9), (K.ALLREDUCE, 8, K.DT_FLOAT32, 4, 128),
    # sizes at which the staged kernels were measured to be faster stay staged
    (K.REDUCE_SCATTER, 2, K.DT_FLOAT32, 28, 33), (K.REDUCE_SCATTER, 4, K.DT_FLOAT32, 20, 64),
    (K.REDUCE_SCATTER, 4, K.DT_BFLOAT16, 12, 17), (K.ALLGATHER, 4, K.DT_FLOAT32, 90, 128), (K.ALLGATHER, 6, K.DT_BFLOAT16, 112, 192),
    (K.ALLGATHER, 8, K.DT_FLOAT32, 144, 192), (K.ALLTOALL, 4, K.DT_FLOAT32, 24, 48), (K.ALLTOALL, 8, K.DT_BFLOAT16, 40, 48)])
def test_limits_lie_where_zero_copy_was_measured_to_win(coll, n, dt, staged, direct):
    assert not _pays(coll, n, staged * MB, dt)
    assert _pays(coll, n, direct * MB, dt)
    assert not _pays(coll, n, direct * MB, dt, shift=4)      # a source that is not 16-byte aligned


def test_types_and_overlaps_that_stay_staged():
    n, big = 4, 256 * MB
    assert not _pays(K.ALLREDUCE, n, big, K.DT_INT32) and not _pays(K.REDUCE_SCATTER, n, big, K.DT_INT32)
    assert not _pays(K.BCAST, n, big) and not _pays(K.REDUCE, n, big)
    buf = [BASE + r * STEP for r in range(n)]
    assert _pays(K.ALLREDUCE, n, big, src=buf, dst=buf)                                    # each rank in place
    assert not _pays(K.ALLREDUCE, n, big, src=buf, dst=buf[1:] + buf[:1])                  # a neighbour's source
    assert not _pays(K.ALLREDUCE, n, big, src=buf, dst=[b + 16 for b in buf])              # shifted onto the own source
    assert not _pays(K.ALLTOALL, n, big, src=buf, dst=buf) and not _pays(K.REDUCE_SCATTER, n, big, src=buf, dst=buf)
