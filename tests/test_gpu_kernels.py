"""GPU tests of the hand-written kernels against plain PyTorch fp32 references.

The multi-rank NVLink kernels run here through the single-GPU emulation (one cooperative launch
whose blockIdx.y is the rank); the real multi-process path has its own test module.
"""
import ctypes as C

import os

import pytest
import torch

from xccl_b200 import _capi as K

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.set_device(0)
    return torch.device("cuda:0")


def _loaded_native():
    # fail loudly if the native library is not the thing that runs
    with open("/proc/self/maps") as f:
        assert "libxccl.so" in f.read(), "libxccl.so is not loaded"


# ----------------------------------------------------------------------------- local reduce kernels
@pytest.mark.parametrize("dtype,dt", [(torch.float32, K.DT_FLOAT32), (torch.bfloat16, K.DT_BFLOAT16),
                                      (torch.float16, K.DT_FLOAT16), (torch.int32, K.DT_INT32),
                                      (torch.int64, K.DT_INT64), (torch.uint8, K.DT_UINT8)])
@pytest.mark.parametrize("count", [1, 7, 4099, 1 << 20])
def test_reduce_multi_kernel(dev, dtype, dt, count):
    from xccl_b200.ops import emu  # noqa: F401  (declares optional prototypes)
    L = K.load()
    L.xccl_cuda_reduce_multi.restype = C.c_int
    L.xccl_cuda_reduce_multi.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_size_t, C.c_size_t, C.c_size_t,
                                         C.c_int, C.c_int, C.c_float, C.c_int, C.c_void_p]
    g = torch.Generator(device="cpu").manual_seed(0)
    nvec = 5
    hi = 4 if dtype == torch.uint8 else 9
    a = torch.randint(0, hi, (count,), generator=g).to(dtype).to(dev)
    v = torch.randint(0, hi, (nvec, count), generator=g).to(dtype).to(dev)
    out = torch.empty_like(a)
    for op, ref in ((K.OP_SUM, lambda x: x.sum(0)), (K.OP_MAX, lambda x: x.max(0).values)):
        st = L.xccl_cuda_reduce_multi(a.data_ptr(), v.data_ptr(), out.data_ptr(), nvec, count,
                                      count * a.element_size(), dt, op, 1.0, K.DT_UNSUPPORTED,
                                      torch.cuda.current_stream().cuda_stream)
        assert st == K.OK
        allv = torch.cat([a[None], v]).to(torch.float64 if dtype.is_floating_point else torch.int64)
        want = ref(allv).to(dtype)
        torch.cuda.synchronize()
        assert torch.equal(out, want), (dtype, op, count)
    _loaded_native()


def test_reduce_scale_and_cast(dev):
    L = K.load()
    L.xccl_cuda_reduce_multi.restype = C.c_int
    L.xccl_cuda_reduce_multi.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_size_t, C.c_size_t, C.c_size_t,
                                         C.c_int, C.c_int, C.c_float, C.c_int, C.c_void_p]
    n = 100003
    a = torch.randn(n, device=dev)
    v = torch.randn(3, n, device=dev)
    out = torch.empty(n, device=dev, dtype=torch.bfloat16)
    st = L.xccl_cuda_reduce_multi(a.data_ptr(), v.data_ptr(), out.data_ptr(), 3, n, n * 4, K.DT_FLOAT32, K.OP_SUM,
                                  0.25, K.DT_BFLOAT16, torch.cuda.current_stream().cuda_stream)
    assert st == K.OK
    want = ((a + v.sum(0)) * 0.25).to(torch.bfloat16)
    torch.cuda.synchronize()
    torch.testing.assert_close(out.float(), want.float(), rtol=1e-2, atol=1e-2)


def test_stream_hold_times_out_without_hanging(dev):
    L = K.load()
    L.xccl_cuda_hold_timeout_probe.restype = C.c_int
    L.xccl_cuda_hold_timeout_probe.argtypes = [C.c_int, C.POINTER(C.c_float)]
    ms = C.c_float()
    st = L.xccl_cuda_hold_timeout_probe(50, C.byref(ms))
    assert st == K.ERR_TIMED_OUT
    assert 40.0 <= ms.value < 2000.0
    # the context is still usable
    assert float(torch.ones(4, device=dev).sum()) == 4.0


# ----------------------------------------------------------------------------- emulated NVLink team
@pytest.fixture(scope="module")
def world4(dev):
    from xccl_b200.ops.emu import EmuWorld
    w = EmuWorld(4, 8 << 20)
    yield w
    w.close()


def _ints(n, count, dtype, dev, seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return [torch.randint(-8, 9, (count,), generator=g).to(dtype).to(dev) for _ in range(n)]


@pytest.mark.parametrize("alg", [K.NVLINK_ALG_ONE_SHOT, K.NVLINK_ALG_TWO_SHOT])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.int32])
@pytest.mark.parametrize("count", [1, 33, 4096, 262147])
def test_emu_allreduce(world4, dev, alg, dtype, count):
    if alg == K.NVLINK_ALG_ONE_SHOT and count * 4 * 4 > (4 << 20):
        pytest.skip("one-shot needs size x message bytes in one workspace half")
    srcs = _ints(4, count, dtype, dev, seed=count)
    dsts = [torch.full_like(s, 99) for s in srcs]
    world4.allreduce(srcs, dsts, alg=alg)
    want = torch.stack([s.double() for s in srcs]).sum(0).to(dtype)
    for d in dsts:
        assert torch.equal(d, want)
    # max
    world4.allreduce(srcs, dsts, op=K.OP_MAX, alg=alg)
    want = torch.stack(srcs).max(0).values
    for d in dsts:
        assert torch.equal(d, want)


def test_emu_allreduce_chunks_through_small_workspace(world4, dev):
    # 12 MB per rank through a workspace half of 4 MB: three chunks, alternating halves
    count = 3 << 20
    srcs = [torch.randn(count, device=dev) for _ in range(4)]
    dsts = [torch.empty_like(s) for s in srcs]
    world4.allreduce(srcs, dsts, alg=K.NVLINK_ALG_TWO_SHOT)
    want = torch.stack(srcs).double().sum(0).float()
    for d in dsts:
        torch.testing.assert_close(d, want, rtol=1e-5, atol=1e-5)
    assert torch.equal(dsts[0], dsts[3])  # every rank adds in the same order


def test_emu_allreduce_fused_scale_cast_and_unaligned(world4, dev):
    count = 10007
    base = [torch.randn(count + 3, device=dev) for _ in range(4)]
    srcs = [b[3:] for b in base]  # 12-byte offset: not 16-byte aligned
    dsts = [torch.empty(count + 1, device=dev, dtype=torch.bfloat16)[1:] for _ in range(4)]
    for alg in (K.NVLINK_ALG_ONE_SHOT, K.NVLINK_ALG_TWO_SHOT):
        world4.allreduce(srcs, dsts, alg=alg, scale=0.25)
        want = (torch.stack(srcs).double().sum(0) * 0.25).float()
        for d in dsts:
            torch.testing.assert_close(d.float(), want, rtol=1e-2, atol=2e-2)


def test_emu_reduce_and_reduce_scatter(world4, dev):
    count = 5000
    srcs = _ints(4, count, torch.float32, dev, seed=3)
    for root in range(4):
        dsts = [torch.full((count,), -1.0, device=dev) for _ in range(4)]
        world4.reduce(srcs, dsts, root)
        assert torch.equal(dsts[root], torch.stack(srcs).sum(0))
        for r in range(4):
            if r != root:
                assert torch.all(dsts[r] == -1.0)
    per = 1237
    srcs = _ints(4, per * 4, torch.int32, dev, seed=4)
    dsts = [torch.zeros(per, dtype=torch.int32, device=dev) for _ in range(4)]
    world4.reduce_scatter(srcs, dsts)
    full = torch.stack(srcs).sum(0)
    for r in range(4):
        assert torch.equal(dsts[r], full[r * per:(r + 1) * per].to(torch.int32))


def test_emu_bcast_allgather_alltoall(world4, dev):
    n = 4
    for nbytes in (1, 13, 4096, 3 << 20):
        bufs = [torch.randint(0, 255, (nbytes,), dtype=torch.uint8, device=dev) for _ in range(n)]
        root = 2
        want = bufs[root].clone()
        world4.bcast(bufs, bufs, root)
        for b in bufs:
            assert torch.equal(b, want)
    for per in (3, 1000, 1 << 20):
        srcs = [torch.randint(0, 255, (per,), dtype=torch.uint8, device=dev) for _ in range(n)]
        dsts = [torch.zeros(per * n, dtype=torch.uint8, device=dev) for _ in range(n)]
        world4.allgather(srcs, dsts)
        for d in dsts:
            assert torch.equal(d, torch.cat(srcs))
    for per in (1, 1024, 100003):
        srcs = [torch.randn(per * n, device=dev) for _ in range(n)]
        dsts = [torch.zeros(per * n, device=dev) for _ in range(n)]
        world4.alltoall(srcs, dsts)
        for r in range(n):
            want = torch.cat([srcs[s][r * per:(r + 1) * per] for s in range(n)])
            assert torch.equal(dsts[r], want)


def test_emu_direct_zero_copy_algorithms(world4, dev):
    """The direct kernels read and write the ranks' own buffers (no workspace): allreduce with the fused
    scale and cast, in place, reduce-scatter, allgather (also in place) and alltoall."""
    n = 4
    D = K.NVLINK_ALG_DIRECT
    for dtype, count in ((torch.float32, 4 * 5000), (torch.bfloat16, 8 * 70001), (torch.float16, 8 * 16)):
        srcs = _ints(n, count, dtype, dev, seed=11)
        dsts = [torch.zeros(count, dtype=dtype, device=dev) for _ in range(n)]
        world4.allreduce(srcs, dsts, alg=D)
        want = torch.stack([s.float() for s in srcs]).sum(0)
        for d in dsts:
            assert torch.equal(d.float(), want)
    srcs = [torch.randn(4 * 3000, device=dev) for _ in range(n)]
    want = torch.stack(srcs).sum(0) * 0.25
    outs = [torch.zeros(4 * 3000, dtype=torch.bfloat16, device=dev) for _ in range(n)]
    world4.allreduce(srcs, outs, alg=D, scale=0.25)          # fp32 -> bf16 with the average fused
    for o in outs:
        torch.testing.assert_close(o.float(), want, rtol=1e-2, atol=1e-2)
    bufs = [s.clone() for s in srcs]
    world4.allreduce(bufs, bufs, alg=D, op=K.OP_MAX)        # in place
    for b in bufs:
        assert torch.equal(b, torch.stack(srcs).max(0).values)
    per = 4 * 1237
    srcs = _ints(n, per * n, torch.float32, dev, seed=12)
    dsts = [torch.zeros(per, device=dev) for _ in range(n)]
    world4.reduce_scatter(srcs, dsts, alg=D)
    full = torch.stack(srcs).sum(0)
    for r in range(n):
        assert torch.equal(dsts[r], full[r * per:(r + 1) * per])
    per = 16 * 4099
    srcs = [torch.randint(0, 255, (per,), dtype=torch.uint8, device=dev) for _ in range(n)]
    dsts = [torch.zeros(per * n, dtype=torch.uint8, device=dev) for _ in range(n)]
    world4.allgather(srcs, dsts, alg=D)
    for d in dsts:
        assert torch.equal(d, torch.cat(srcs))
    inplace = [torch.zeros(per * n, dtype=torch.uint8, device=dev) for _ in range(n)]
    for r in range(n):
        inplace[r][r * per:(r + 1) * per] = srcs[r]
    world4.allgather([inplace[r][r * per:(r + 1) * per] for r in range(n)], inplace, alg=D)
    for d in inplace:
        assert torch.equal(d, torch.cat(srcs))
    per = 4 * 25001
    srcs = [torch.randn(per * n, device=dev) for _ in range(n)]
    dsts = [torch.zeros(per * n, device=dev) for _ in range(n)]
    world4.alltoall(srcs, dsts, alg=D)
    for r in range(n):
        assert torch.equal(dsts[r], torch.cat([srcs[s][r * per:(r + 1) * per] for s in range(n)]))


class _Guarded:
    """A byte buffer with 256 sentinel bytes before and after the part a kernel may touch, placed at an odd
    offset so that the payload is not 16-byte aligned: an out-of-bounds pack store shows up in the guards."""
    PAD = 256

    def __init__(self, nbytes, dev, fill=0xA5, skew=3):
        self.raw = torch.full((nbytes + 2 * self.PAD + 16,), fill, dtype=torch.uint8, device=dev)
        self.off = self.PAD + skew
        self.n, self.fill = nbytes, fill

    @property
    def view(self):
        return self.raw[self.off:self.off + self.n]

    def guards_intact(self):
        return bool(torch.all(self.raw[:self.off] == self.fill)) and bool(torch.all(self.raw[self.off + self.n:] == self.fill))


def test_emu_byte_collectives_stay_inside_their_buffers(world4, dev):
    """bcast / allgather / alltoall on unaligned, odd-sized byte buffers: results exact, sources untouched,
    not one byte written outside the destination."""
    n = 4
    for per in (1, 13, 4099, 70001):
        srcs = [_Guarded(per, dev, fill=0x11) for _ in range(n)]
        for r, g in enumerate(srcs):
            g.view.copy_(torch.randint(0, 255, (per,), dtype=torch.uint8, generator=torch.Generator().manual_seed(per + r)).to(dev))
        keep = [g.view.clone() for g in srcs]
        dsts = [_Guarded(per * n, dev) for _ in range(n)]
        world4.allgather([g.view for g in srcs], [g.view for g in dsts])
        for g in dsts:
            assert torch.equal(g.view, torch.cat(keep)) and g.guards_intact(), ("allgather", per)
        a_src = [_Guarded(per * n, dev, fill=0x22) for _ in range(n)]
        for r, g in enumerate(a_src):
            g.view.copy_(torch.randint(0, 255, (per * n,), dtype=torch.uint8, generator=torch.Generator().manual_seed(7 * per + r)).to(dev))
        a_keep = [g.view.clone() for g in a_src]
        a_dst = [_Guarded(per * n, dev) for _ in range(n)]
        world4.alltoall([g.view for g in a_src], [g.view for g in a_dst])
        for r in range(n):
            want = torch.cat([a_keep[s][r * per:(r + 1) * per] for s in range(n)])
            assert torch.equal(a_dst[r].view, want) and a_dst[r].guards_intact(), ("alltoall", per)
        for g, k in zip(srcs + a_src, keep + a_keep):
            assert torch.equal(g.view, k) and g.guards_intact(), ("source modified", per)
        bufs = [_Guarded(per, dev) for _ in range(n)]
        bufs[1].view.copy_(keep[1])
        world4.bcast([g.view for g in bufs], [g.view for g in bufs], root=1)
        for g in bufs:
            assert torch.equal(g.view, keep[1]) and g.guards_intact(), ("bcast", per)


def test_emu_push_allgather_alltoall(world4, dev):
    """The push forms (stores into the destinations' workspaces) on odd, unaligned byte buffers, between pull-form
    calls so that both share the workspace parity bookkeeping."""
    n = 4
    for per in (1, 13, 4099, 70001):
        srcs = [_Guarded(per * n, dev, fill=0x11) for _ in range(n)]
        dsts = [_Guarded(per * n, dev, fill=0x22) for _ in range(n)]
        for r in range(n):
            srcs[r].view.copy_((torch.arange(per * n, device=dev) * 7 + r * 31) % 251)
        world4.alltoall([s.view for s in srcs], [d.view for d in dsts], alg=K.NVLINK_ALG_ONE_SHOT)
        for r in range(n):
            want = torch.cat([srcs[q].view[r * per:(r + 1) * per] for q in range(n)])
            assert torch.equal(dsts[r].view, want) and dsts[r].guards_intact(), ("alltoall push", per, r)
        parts = [_Guarded(per, dev, fill=0x33) for _ in range(n)]
        for r in range(n):
            parts[r].view.copy_((torch.arange(per, device=dev) * 3 + r * 17) % 253)
        world4.allgather([p_.view for p_ in parts], [d.view for d in dsts], alg=K.NVLINK_ALG_ONE_SHOT)
        want = torch.cat([p_.view for p_ in parts])
        for r in range(n):
            assert torch.equal(dsts[r].view, want) and dsts[r].guards_intact(), ("allgather push", per, r)
        world4.allgather([p_.view for p_ in parts], [d.view for d in dsts])   # pull form next to it
        for r in range(n):
            assert torch.equal(dsts[r].view, want)


def test_emu_alltoallv(world4, dev):
    n = 4
    sc = [[(s * 3 + d * 5 + 1) for d in range(n)] for s in range(n)]  # elements rank s sends to rank d
    srcs, dsts, metas, keep = [], [], [], []
    for r in range(n):
        scounts = sc[r]
        sdispl = [sum(scounts[:d]) for d in range(n)]
        rcounts = [sc[s][r] for s in range(n)]
        rdispl = [sum(rcounts[:s]) for s in range(n)]
        srcs.append(torch.cat([torch.full((scounts[d],), float(r * 10 + d), device=dev) for d in range(n)]))
        dsts.append(torch.zeros(sum(rcounts), device=dev))
        metas.append(torch.tensor(scounts + sdispl + rcounts + rdispl, dtype=torch.int32, device=dev))
        keep.append((rcounts,))
    world4.alltoallv(srcs, dsts, metas, max(s.numel() for s in srcs) * 4)
    for r in range(n):
        want = torch.cat([torch.full((sc[s][r],), float(s * 10 + r), device=dev) for s in range(n)])
        assert torch.equal(dsts[r], want)


def test_emu_alltoallv_larger_than_the_workspace(dev):
    """Uneven counts whose streams are several workspace halves long (and of different length per rank, one rank
    sending nothing): the kernel walks the exchange in windows and agrees on the number of rounds from the headers."""
    from xccl_b200.ops.emu import EmuWorld
    n = 4
    w = EmuWorld(n, 256 << 10)   # halves of 128 KiB, 8 KiB of it header
    try:
        for trial in range(2):   # the second exchange starts on the other workspace half
            sc = [[(7919 * (s + 1) + 15013 * d + 3 + trial) * (0 if s == 2 else 1) for d in range(n)] for s in range(n)]
            sc[1][3] = 0
            srcs, dsts, metas = [], [], []
            g = torch.Generator(device=dev).manual_seed(5 + trial)
            for r in range(n):
                scounts = sc[r]
                sdispl = [sum(scounts[:d]) for d in range(n)]
                rcounts = [sc[s][r] for s in range(n)]
                rdispl = [sum(rcounts[:s]) for s in range(n)]
                srcs.append(torch.randn(max(sum(scounts), 1), device=dev, generator=g))
                dsts.append(torch.full((max(sum(rcounts), 1) + 4,), -1.0, device=dev))
                metas.append(torch.tensor(scounts + sdispl + rcounts + rdispl, dtype=torch.int32, device=dev))
            assert max(sum(x) for x in sc) * 4 > 3 * (128 << 10)
            w.alltoallv(srcs, dsts, metas, max(sum(x) for x in sc) * 4)
            for r in range(n):
                parts = []
                for s_ in range(n):
                    o = sum(sc[s_][:r])
                    parts.append(srcs[s_][o:o + sc[s_][r]])
                want = torch.cat(parts)
                assert torch.equal(dsts[r][:want.numel()], want), (trial, r)
                assert torch.all(dsts[r][want.numel():] == -1.0)
            # the workspace parity bookkeeping still holds for what follows
            a = _ints(n, 3000, torch.float32, dev, seed=trial)
            b = [torch.empty_like(x) for x in a]
            w.allreduce(a, b, alg=K.NVLINK_ALG_TWO_SHOT)
            assert torch.equal(b[3], torch.stack(a).sum(0))
    finally:
        w.close()


_BOUNDS_SCRIPT = r"""
import ctypes as C, torch
from xccl_b200 import _capi as K
from xccl_b200.ops.emu import EmuWorld
dev = torch.device("cuda:0")
L = K.load()
rep = (C.c_ulonglong * 4)()
L.xccl_nvlink_debug_bounds_report.restype = C.c_int
assert L.xccl_nvlink_debug_bounds_report(rep) == K.OK, "not a bounds-checking build"
n = 4
w = EmuWorld(n, 1 << 20)            # small halves: the chunk loops, window rounds and parity changes all run
g = torch.Generator(device=dev).manual_seed(0)
for count in (1, 1000, 70001, 300000):
    srcs = [torch.randn(count, device=dev, generator=g) for _ in range(n)]
    dsts = [torch.empty_like(s) for s in srcs]
    for alg in (K.NVLINK_ALG_ONE_SHOT, K.NVLINK_ALG_TWO_SHOT, K.NVLINK_ALG_DIRECT):
        if alg == K.NVLINK_ALG_ONE_SHOT and count * 4 * n > (1 << 19):
            continue
        if alg == K.NVLINK_ALG_DIRECT and count % 4:
            continue
        w.allreduce(srcs, dsts, alg=alg)
        torch.testing.assert_close(dsts[2], torch.stack(srcs).sum(0), rtol=1e-5, atol=1e-5)
    w.reduce(srcs, dsts, root=1)
    rs = [torch.randn(count * n, device=dev, generator=g) for _ in range(n)]
    rd = [torch.empty(count, device=dev) for _ in range(n)]
    w.reduce_scatter(rs, rd)
for per in (13, 4099, 200003):
    bs = [torch.randint(0, 255, (per * n,), dtype=torch.uint8, device=dev) for _ in range(n)]
    bd = [torch.empty_like(b) for b in bs]
    w.alltoall(bs, bd)
    w.alltoall(bs, bd, alg=K.NVLINK_ALG_ONE_SHOT)
    w.bcast(bs, bd, 2)
    ps = [torch.randint(0, 255, (per,), dtype=torch.uint8, device=dev) for _ in range(n)]
    w.allgather(ps, bd)
    w.allgather(ps, bd, alg=K.NVLINK_ALG_ONE_SHOT)
sc = [[(7919 * (s + 1) + 15013 * d + 3) for d in range(n)] for s in range(n)]
srcs, dsts, metas = [], [], []
for r in range(n):
    rc = [sc[s][r] for s in range(n)]
    srcs.append(torch.randn(sum(sc[r]), device=dev, generator=g))
    dsts.append(torch.empty(sum(rc), device=dev))
    metas.append(torch.tensor(sc[r] + [sum(sc[r][:d]) for d in range(n)] + rc + [sum(rc[:s]) for s in range(n)],
                              dtype=torch.int32, device=dev))
w.alltoallv(srcs, dsts, metas, max(s.numel() for s in srcs) * 4)
assert torch.equal(dsts[1][:sc[0][1]], srcs[0][sc[0][0]:sc[0][0] + sc[0][1]])
w.barrier()
assert L.xccl_nvlink_debug_bounds_report(rep) == K.OK
w.close()
print("violations", rep[0], hex(rep[1]), rep[2], rep[3])
assert rep[0] == 0
"""


def test_emu_collectives_under_the_bounds_checking_build(dev):
    """Every NVLink collective with all ranks emulated, on the library built with -DXCCL_DEBUG_BOUNDS: each 16-byte
    access to a workspace or a peer buffer is checked against the ranges of its launch, an access outside them is
    recorded and skipped. Results stay right and the record stays empty."""
    import os
    import subprocess
    import sys
    from pathlib import Path
    root = Path(__file__).resolve().parent.parent
    lib = root / "xccl_b200" / "lib" / "libxccl_bounds.so"
    if not lib.exists():
        pytest.skip("libxccl_bounds.so is not built (python -m xccl_b200.build --debug-bounds)")
    env = dict(os.environ, XCCL_B200_LIB=str(lib), PYTHONPATH=str(root))
    r = subprocess.run([sys.executable, "-c", _BOUNDS_SCRIPT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    assert "violations 0" in r.stdout


_RANGES_SCRIPT = r"""
import ctypes as C, torch
from xccl_b200 import _capi as K
from xccl_b200.ops.emu import EmuWorld
dev = torch.device("cuda:0")
lo, hi = (C.c_ulonglong * 64)(), (C.c_ulonglong * 64)()
n, ws = 2, 1 << 20
w = EmuWorld(n, ws)
def may_touch(t):
    k = K.load().xccl_nvlink_debug_bounds_ranges(lo, hi, 64)
    assert 0 < k <= 64
    a, b = t.data_ptr(), t.data_ptr() + t.numel() * t.element_size()
    return any(lo[i] < b and a < hi[i] for i in range(k))
big = 16 << 20                        # 16 MB and more of all ranks together run zero-copy when no algorithm is named
for count, alg, direct in ((1024, 0, False), (1024, K.NVLINK_ALG_TWO_SHOT, False), (big // 8, K.NVLINK_ALG_TWO_SHOT, False),
                           (big // 8, 0, True), (1024, K.NVLINK_ALG_DIRECT, True)):
    src = [torch.ones(count, device=dev) for _ in range(n)]
    dst = [torch.empty(count, device=dev) for _ in range(n)]
    w.allreduce(src, dst, alg=alg)
    assert all(bool((d == n).all()) for d in dst)
    assert [may_touch(t) for t in src + dst] == [direct] * 2 * n, (count, alg)
w.close()
print("ranges ok")
"""


def test_bounds_of_a_staged_collective_leave_the_user_buffers_out(dev):
    """The bounds-checking build entitles a staged kernel's checked accesses to the workspaces alone; the ranks' buffers
    are added for the zero-copy kernels only."""
    import subprocess
    import sys
    from pathlib import Path
    root = Path(__file__).resolve().parent.parent
    lib = root / "xccl_b200" / "lib" / "libxccl_bounds.so"
    if not lib.exists():
        pytest.skip("libxccl_bounds.so is not built (python -m xccl_b200.build --debug-bounds)")
    env = dict(os.environ, XCCL_B200_LIB=str(lib), PYTHONPATH=str(root))
    r = subprocess.run([sys.executable, "-c", _RANGES_SCRIPT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


@pytest.mark.parametrize("ranks,kb", [(2, 8192), (2, 16400), (4, 2048), (4, 4112), (4, 8208), (8, 1024), (8, 4096)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.int32])
def test_emu_large_collectives_with_no_algorithm_named(dev, ranks, kb, dtype):
    """Around the sizes where the unnamed algorithm turns zero-copy, and the forms that must stay staged: types the
    zero-copy kernels do not have, unaligned buffers. Integers, so sums are exact."""
    from xccl_b200.ops.emu import EmuWorld
    w = EmuWorld(ranks, 8 << 20)
    try:
        n = (kb << 10) // torch.empty(0, dtype=dtype).element_size() // (16 * ranks) * (16 * ranks)
        pool = torch.randint(-8, 9, (ranks * (n + 16) + n,), device=dev).to(dtype)
        for shift in (0, 1):                        # shift 1: sources that are not 16-byte aligned
            src = [pool[r * (n + 16) + shift: r * (n + 16) + shift + n] for r in range(ranks)]
            total = sum(s.double() for s in src)
            dst = [torch.empty(n, dtype=dtype, device=dev) for _ in range(ranks)]
            w.allreduce(src, dst)
            assert all(torch.equal(d.double(), total) for d in dst)
            part = [torch.empty(n // ranks, dtype=dtype, device=dev) for _ in range(ranks)]
            w.reduce_scatter(src, part)
            assert torch.equal(torch.cat(part).double(), total)
            w.alltoall(src, dst)
            chunks = [s.chunk(ranks) for s in src]
            assert all(torch.equal(dst[d], torch.cat([chunks[s][d] for s in range(ranks)])) for d in range(ranks))
            full = [torch.empty(n * ranks, dtype=dtype, device=dev) for _ in range(ranks)]
            w.allgather(src, full)
            assert all(torch.equal(f, torch.cat(src)) for f in full)
        # in place
        src = [pool[r * (n + 16): r * (n + 16) + n].clone() for r in range(ranks)]
        total = sum(s.double() for s in src)
        w.allreduce(src, src)
        assert all(torch.equal(s.double(), total) for s in src)
    finally:
        w.close()


def test_emu_sync_collectives_and_bounded_wait(world4, dev):
    for _ in range(3):
        world4.barrier()
    for root in range(4):
        world4.fanin(root)
        world4.fanout(root)
    st, ms, st4 = world4.timeout_probe(30)
    assert st == K.ERR_TIMED_OUT and st4[0] == 1
    assert 20.0 <= ms < 2000.0
    # the team still works after the probe
    srcs = _ints(4, 100, torch.float32, dev, seed=9)
    dsts = [torch.empty_like(s) for s in srcs]
    world4.allreduce(srcs, dsts)
    assert torch.equal(dsts[1], torch.stack(srcs).sum(0))


def test_emu_allreduce_eight_ranks(dev):
    from xccl_b200.ops.emu import EmuWorld
    w = EmuWorld(8, 8 << 20)
    try:
        for count, alg in ((1000, K.NVLINK_ALG_ONE_SHOT), (300000, K.NVLINK_ALG_TWO_SHOT)):
            srcs = _ints(8, count, torch.bfloat16, dev, seed=count)
            dsts = [torch.empty_like(s) for s in srcs]
            w.allreduce(srcs, dsts, alg=alg)
            want = torch.stack([s.float() for s in srcs]).sum(0).to(torch.bfloat16)
            for d in dsts:
                assert torch.equal(d, want)
    finally:
        w.close()


# ----------------------------------------------------------------------------- tcgen05 GEMM
@pytest.mark.parametrize("M,N,K_", [(128, 256, 64), (256, 512, 256), (384, 768, 1024), (1000, 264, 520)])
def test_gemm_bf16_matches_fp32_reference(dev, M, N, K_):
    from xccl_b200.ops import gemm
    a = (torch.randn(M, K_, device=dev) * 0.5).to(torch.bfloat16)
    b = (torch.randn(N, K_, device=dev) * 0.5).to(torch.bfloat16)
    out = gemm.gemm_bf16(a, b)
    assert gemm.last_error() == 0
    want = a.float() @ b.float().t()
    torch.testing.assert_close(out.float(), want, rtol=2e-2, atol=2e-2 * K_ ** 0.5)
    _loaded_native()


def test_gemm_swiglu_matches_fp32_reference(dev):
    from xccl_b200.ops import gemm
    M, F, K_ = 512, 384, 512
    a = (torch.randn(M, K_, device=dev) * 0.5).to(torch.bfloat16)
    wg = (torch.randn(F, K_, device=dev) * 0.05).to(torch.bfloat16)
    wu = (torch.randn(F, K_, device=dev) * 0.05).to(torch.bfloat16)
    out = gemm.gemm_swiglu(a, wg, wu)
    assert gemm.last_error() == 0
    g = a.float() @ wg.float().t()
    u = a.float() @ wu.float().t()
    want = torch.nn.functional.silu(g) * u
    torch.testing.assert_close(out.float(), want, rtol=3e-2, atol=3e-2)


def test_gemm_many_tiles_persistent_schedule(dev):
    from xccl_b200.ops import gemm
    M, N, K_ = 4096, 4096, 512   # 512 tiles over 148 CTAs: several tiles per CTA, both accumulators in use
    a = (torch.randn(M, K_, device=dev) * 0.3).to(torch.bfloat16)
    b = (torch.randn(N, K_, device=dev) * 0.3).to(torch.bfloat16)
    out = gemm.gemm_bf16(a, b)
    assert gemm.last_error() == 0
    want = a.float() @ b.float().t()
    torch.testing.assert_close(out.float(), want, rtol=2e-2, atol=0.5)


# ----------------------------------------------------------------------------- fused TP-MLP kernels
def _full_weights(mlp):
    wg = torch.cat(mlp.w_gate, 0)
    wu = torch.cat(mlp.w_up, 0)
    wd = torch.cat(mlp.w_down, 1)
    return wg, wu, wd


@pytest.mark.parametrize("tp", [1, 2, 4])
def test_tp_mlp_fused_matches_fp32_reference(dev, tp):
    """allgather->GEMM(+SwiGLU) and GEMM->reduce-scatter, ranks emulated inside one launch."""
    from xccl_b200.models.tp_mlp import TpMlp, reference_forward_fp32
    tokens, hidden, ffn = 1024, 512, 1024
    mlp = TpMlp(tokens, hidden, ffn, tp=tp, emulate=True)
    try:
        g = torch.Generator(device=dev).manual_seed(5)
        x = torch.randn(tokens, hidden, device=dev, generator=g).to(torch.bfloat16)
        shards = list(x.chunk(tp, 0))
        for it in range(3):  # repeated launches: sequence numbers, parities and counters advance
            y = mlp.forward(shards)
            mlp.check_error()
            want = reference_forward_fp32(x, *_full_weights(mlp))
            got = torch.cat(y, 0).float()
            torch.testing.assert_close(got, want, rtol=3e-2, atol=3e-2)
        # the gathered buffer of every rank holds every shard
        for i in range(mlp.n_local):
            assert torch.equal(mlp.ws.x_full(i), x)
    finally:
        mlp.close()
    _loaded_native()


def test_tp_mlp_end_to_end_from_pinned_host(dev):
    from xccl_b200.models.tp_mlp import TpMlp
    mlp = TpMlp(512, 256, 512, tp=1)
    try:
        x = torch.randn(512, 256).to(torch.bfloat16).pin_memory()
        m = mlp.forward_from_host([x])
        mlp.check_error()
        assert m.device.type == "cpu" and torch.isfinite(m)
    finally:
        mlp.close()


@pytest.mark.parametrize("tp,phases", [(1, False), (2, False), (4, False), (4, True), (8, False), (8, True)])
def test_tp_mlp_input_arriving_from_host_overlaps_first_kernel(dev, tp, phases, monkeypatch):
    """The chunked host->device copy with stream-ordered flags: the kernel starts before the rows are there and
    must produce the same output as the plain copy-then-launch path, step after step. With copy CTAs (4 and 8
    ranks) and H2D_PHASES every rank reports its rows block by block and the tiles are walked in phases over all shards."""
    from xccl_b200.models.tp_mlp import TpMlp, reference_forward_fp32
    monkeypatch.setenv("XCCL_TP_H2D_OVERLAP", "1")
    monkeypatch.setenv("XCCL_TP_H2D_PHASES", "y" if phases else "n")
    tokens, hidden, ffn = (1024, 512, 1024) if tp <= 2 else (4096, 512, 1024)
    mlp = TpMlp(tokens, hidden, ffn, tp=tp, emulate=(tp > 1))
    try:
        assert mlp.overlap_h2d
        for it in range(3):
            x = torch.randn(tokens, hidden, generator=torch.Generator().manual_seed(it)).to(torch.bfloat16)
            pinned = [c.contiguous().pin_memory() for c in x.chunk(tp, 0)]
            mlp.forward_from_host(pinned)
            mlp.check_error()
            want = reference_forward_fp32(x.to(dev), *_full_weights(mlp))
            torch.testing.assert_close(torch.cat(mlp.y, 0).float(), want, rtol=3e-2, atol=3e-2)
    finally:
        mlp.close()


def test_tp_mlp_full_output_read_back_is_pipelined_and_exact(dev):
    """forward_from_host_full: input from pinned memory (kernels launched first, rows follow), the whole output shard
    copied back on a copy stream while the next step runs; every step's host copy must hold that step's output."""
    from xccl_b200.models.tp_mlp import TpMlp, reference_forward_fp32
    tokens, hidden, ffn = 1024, 512, 1024
    mlp = TpMlp(tokens, hidden, ffn, tp=1)
    try:
        y_pinned = [[torch.empty(tokens, hidden, dtype=torch.bfloat16).pin_memory()] for _ in range(2)]
        xs = [torch.randn(tokens, hidden, generator=torch.Generator().manual_seed(40 + it)).to(torch.bfloat16) for it in range(4)]
        pinned = [[x.pin_memory()] for x in xs]
        wants = [reference_forward_fp32(x.to(dev), *_full_weights(mlp)) for x in xs]
        for it in range(4):   # no host wait between the steps
            mlp.forward_from_host_full(pinned[it], y_pinned)
        mlp.wait_outputs()
        mlp.check_error()
        # the two host buffers hold the outputs of the last two steps (parity 0: step 2, parity 1: step 3)
        torch.testing.assert_close(y_pinned[0][0].float().to(dev), wants[2], rtol=3e-2, atol=3e-2)
        torch.testing.assert_close(y_pinned[1][0].float().to(dev), wants[3], rtol=3e-2, atol=3e-2)
    finally:
        mlp.close()


# ----------------------------------------------------------------------------- fused MoE all-to-all
@pytest.mark.parametrize("ranks", [1, 2, 4])
def test_moe_dispatch_combine_matches_reference(dev, ranks):
    """Routing, grouping by (expert, source) and the weighted combine, ranks emulated in one launch."""
    from xccl_b200.ops.moe import MoeWorkspace
    T, H, E, Kk = 96, 256, 8 * ranks, 4
    EL = E // ranks
    ws = MoeWorkspace(T, H, E, Kk, emu_ranks=ranks)
    try:
        g = torch.Generator(device="cpu").manual_seed(ranks)
        xs = [torch.randn(T, H, generator=g).to(torch.bfloat16).to(dev) for _ in range(ranks)]
        ids = [torch.stack([torch.randperm(E, generator=g)[:Kk] for _ in range(T)]).to(torch.int32).to(dev) for _ in range(ranks)]
        ws_ = [torch.softmax(torch.randn(T, Kk, generator=g), -1).to(dev) for _ in range(ranks)]
        for it in range(2):
            ws.dispatch(xs, ids)
            assert ws.error() == 0
            # every rank holds, per local expert, exactly the rows routed to it, grouped by source
            for r in range(ranks):
                rows = ws.expert_rows(r).cpu().tolist()
                recv, src = ws.recv(r), ws.row_source(r).cpu()
                row = 0
                for le in range(EL):
                    e = r * EL + le
                    want_n = sum(int((ids[s] == e).sum()) for s in range(ranks))
                    assert rows[le] == want_n
                    last_src = -1
                    for i in range(rows[le]):
                        s, t = divmod(int(src[row + i]), T)
                        assert s >= last_src          # sources appear in rank order inside an expert
                        last_src = s
                        assert bool((ids[s][t] == e).any())
                        assert torch.equal(recv[row + i], xs[s][t])
                    row += rows[le]
                assert rows[EL] == row
                # "experts": scale each row by (1 + global expert id)
                scale = torch.cat([torch.full((rows[le],), 1.0 + r * EL + le) for le in range(EL)]).to(dev)
                ws.expert_out(r)[:row] = (recv[:row].float() * scale[:, None]).to(torch.bfloat16)
            outs = [torch.zeros(T, H, dtype=torch.bfloat16, device=dev) for _ in range(ranks)]
            ws.combine(ids, ws_, outs)
            assert ws.error() == 0
            for r in range(ranks):
                y = (xs[r].float()[:, None, :] * (1.0 + ids[r].float())[:, :, None]).to(torch.bfloat16).float()
                want = (y * ws_[r][:, :, None]).sum(1)
                torch.testing.assert_close(outs[r].float(), want, rtol=2e-2, atol=2e-2)
    finally:
        ws.close()


@pytest.mark.parametrize("ranks,T,H,E,Kk", [
    (1, 96, 8, 16, 1), (2, 64, 264, 16, 4),          # a row of one pack; a second, ragged piece of one pack
    (1, 50, 1032, 64, 9), (2, 30, 520, 64, 33),      # more than eight entries per token in combine, more than 32 in dispatch
    (4, 20, 7168, 16, 4), (1, 300, 2048, 1024, 8),   # 28 pieces of a row; as many experts as there are
    (1, 6400, 1032, 16, 2), (1, 9500, 1032, 16, 2),  # pieces of 64 and of 128 packs (two and four loads per lane), ragged
])
def test_moe_row_pieces_many_entries_and_dropped_ids(dev, ranks, T, H, E, Kk):
    """Sizes at which dispatch and combine cut rows and entries differently, with ids outside the experts among them."""
    from xccl_b200.ops.moe import MoeWorkspace
    EL = E // ranks
    ws = MoeWorkspace(T, H, E, Kk, emu_ranks=ranks)
    try:
        g = torch.Generator(device=dev).manual_seed(T + H)
        xs = [torch.randn(T, H, device=dev, generator=g).to(torch.bfloat16) for _ in range(ranks)]
        ids = [torch.rand(T, E, device=dev, generator=g).topk(Kk, -1).indices.to(torch.int32) for _ in range(ranks)]
        for i in ids:                                 # dropped entries, a whole token among them
            drop = torch.rand(T, Kk, device=dev, generator=g) < 0.1
            i[drop] = -1
            i[T // 2] = E
        gates = [torch.rand(T, Kk, device=dev, generator=g) for _ in range(ranks)]
        x_all, ids_all = torch.stack(xs), torch.stack(ids).long()
        ws.dispatch(xs, ids)
        assert ws.error() == 0
        for r in range(ranks):
            rows = ws.expert_rows(r).long()
            n = int(rows[EL])
            want = torch.stack([(ids_all == e).sum() for e in range(r * EL, (r + 1) * EL)])
            assert torch.equal(rows[:EL], want) and n == int(want.sum())
            src = ws.row_source(r)[:n].long()
            e = torch.repeat_interleave(torch.arange(r * EL, (r + 1) * EL, device=dev), rows[:EL])
            assert torch.equal(ws.recv(r)[:n], x_all[src // T, src % T])
            # every (expert, source, token) that was asked for exactly once, sources in order inside an expert
            s_, t_, k_ = torch.nonzero((ids_all >= r * EL) & (ids_all < (r + 1) * EL), as_tuple=True)
            asked = (ids_all[s_, t_, k_] * ranks + s_) * T + t_
            assert torch.equal(((e * ranks + src // T) * T + src % T).sort().values, asked.sort().values)
            key = e * ranks + src // T
            assert bool((key[1:] >= key[:-1]).all())
            ws.expert_out(r)[:n] = (ws.recv(r)[:n].float() * (1.0 + (e % 7)[:, None])).to(torch.bfloat16)
        outs = [torch.full((T, H), 5.0, dtype=torch.bfloat16, device=dev) for _ in range(ranks)]
        ws.combine(ids, gates, outs)
        assert ws.error() == 0
        for r in range(ranks):
            want, size = torch.zeros(T, H, device=dev), torch.zeros(T, H, device=dev)
            for k in range(Kk):
                valid = ((ids[r][:, k] >= 0) & (ids[r][:, k] < E)).float()[:, None]
                y = (xs[r].float() * (1.0 + (ids[r][:, k] % 7).float()[:, None])).to(torch.bfloat16).float()
                want += valid * gates[r][:, k:k + 1] * y
                size += valid * gates[r][:, k:k + 1] * y.abs()
            # for every eight entries one bf16 rounding (half of its spacing: 2^-8) of a sum no larger than `size` and the
            # roundings before it (3 %); fp32 sums beside it
            assert bool(((outs[r].float() - want).abs() <= (-(-Kk // 8) * 1.03 * 2.0 ** -8 + 1e-5) * size).all())
            assert not bool(outs[r][T // 2].any())    # a token without experts
    finally:
        ws.close()


@pytest.mark.parametrize("T,H,E,Kk", [
    (1, 8, 4, 3), (1, 4104, 16, 8),                  # more blocks than pieces of the one row, and fewer
    (40, 1032, 8, 6), (147, 264, 16, 5),             # several blocks and one block per token
    (149, 264, 1024, 8), (700, 520, 16, 4),          # a few tokens per block
    (6000, 8, 64, 64), (300, 16, 8, 1000),           # more entries than a block routes at a time
    (5, 16, 8, 1500),                                # more entries per token than that: the kernel of several ranks
])
def test_moe_one_rank_with_repeated_experts(dev, T, H, E, Kk):
    """One rank alone, entries of a token that name the same expert again and again: rows grouped by expert, each entry with
    a row of its own, and the row that dispatch wrote is the one that combine reads."""
    from xccl_b200.ops.moe import MoeWorkspace
    ws = MoeWorkspace(T, H, E, Kk)
    try:
        g = torch.Generator(device=dev).manual_seed(T * 7 + Kk)
        x = torch.randn(T, H, device=dev, generator=g).to(torch.bfloat16)
        ids = torch.randint(-1, E + 1, (T, Kk), device=dev, generator=g).to(torch.int32)   # -1 and E: dropped
        gates = torch.rand(T, Kk, device=dev, generator=g) / Kk
        for _ in range(2):
            ws.dispatch([x], [ids])
        assert ws.error() == 0
        valid = (ids >= 0) & (ids < E)
        rows = ws.expert_rows().long()
        n = int(valid.sum())
        assert torch.equal(rows[:E], torch.bincount(ids[valid].long(), minlength=E)) and int(rows[E]) == n
        src = ws.row_source()[:n].long()
        e = torch.repeat_interleave(torch.arange(E, device=dev), rows[:E])
        assert torch.equal(ws.recv()[:n], x[src])
        asked = (ids.long() * T + torch.arange(T, device=dev)[:, None])[valid]
        assert torch.equal((e * T + src).sort().values, asked.sort().values)
        # experts: multiples of the row by a power of two, exact in bf16
        mult = torch.tensor([1.0, 0.5, 2.0, 0.25], device=dev)
        ws.expert_out()[:n] = (ws.recv()[:n].float() * mult[e % 4][:, None]).to(torch.bfloat16)
        out = torch.full((T, H), 5.0, dtype=torch.bfloat16, device=dev)
        ws.combine([ids], [gates], [out])
        assert ws.error() == 0
        f = (gates.double() * mult[ids.long() % 4].double() * valid).sum(-1, keepdim=True)
        # every eight entries the running sum is rounded to bf16: half of its spacing (2^-8) of a sum that only grows
        bound = (-(-Kk // 8) * 1.03 * 2.0 ** -8 + 1e-5) * (f * x.double().abs())
        assert bool(((out.double() - f * x.double()).abs() <= bound).all())
    finally:
        ws.close()


@pytest.mark.parametrize("ranks", [1, 2, 4])
def test_moe_receive_buffer_too_small(dev, ranks):
    """One rank's receive buffer is a row too small: every rank reports it, nobody writes a row, and the ranks meet at the
    end of every dispatch all the same, so that none runs ahead into its next one (rows or not: two barriers each)."""
    import ctypes as C
    from xccl_b200.ops.moe import MoeWorkspace
    T, H, E, Kk = 40, 64, 8, 2
    ws = MoeWorkspace(T, H, E, Kk, emu_ranks=ranks, cap_rows=ranks * T * Kk - 1)
    fn = K.load().xccl_moe_ws_meetings
    fn.restype, fn.argtypes = C.c_uint32, [C.c_void_p, C.c_int]
    meetings = lambda: [fn(ws.h, r) for r in range(ranks)]
    per = 2 if ranks > 1 else 0                       # one rank has nobody to meet
    try:
        xs = [torch.randn(T, H, device=dev).to(torch.bfloat16) for _ in range(ranks)]
        spread = [torch.randint(0, E, (T, Kk), dtype=torch.int32, device=dev) for _ in range(ranks)]
        fits = [(s + torch.arange(T, device=dev)[:, None]).remainder(E).to(torch.int32) for s in spread]
        full = [torch.zeros(T, Kk, dtype=torch.int32, device=dev) for _ in range(ranks)]   # all rows to expert 0
        if ranks > 1:
            ws.dispatch(xs, fits)
            assert ws.error() == 0 and meetings() == [per] * ranks
        else:
            per = 0
        for r in range(ranks):
            ws.recv(r).fill_(7.0)
            ws.row_source(r).fill_(-9)
        base = meetings()
        for it in range(1, 4):
            ws.dispatch(xs, full)
            assert all(bool((ws.recv(r) == 7.0).all()) and bool((ws.row_source(r) == -9).all()) for r in range(ranks))
            assert ws.error() == 0x400
            assert meetings() == [b + it * per for b in base]
        outs = [torch.full((T, H), 3.0, dtype=torch.bfloat16, device=dev) for _ in range(ranks)]
        ws.combine(full, [torch.ones(T, Kk, device=dev) for _ in range(ranks)], outs)
        assert ws.error() == 0x400 and all(bool((o == 3.0).all()) for o in outs)
        assert meetings() == [b + 4 * per for b in base]
    finally:
        ws.close()


def test_moe_views_outlive_the_workspace(dev):
    """A tensor on workspace memory keeps that memory after close(); without views close() frees it."""
    from xccl_b200.ops.moe import MoeWorkspace
    ws = MoeWorkspace(16, 64, 8, 2)
    x = torch.randn(16, 64, device=dev).to(torch.bfloat16)
    ids = torch.stack([torch.arange(16) % 8, (torch.arange(16) + 1) % 8], 1).to(torch.int32).to(dev)
    ws.dispatch([x], [ids])
    rows, recv = ws.expert_rows(), ws.recv()
    ws.close()
    assert rows.cpu().tolist() == [4] * 8 + [32]
    assert float(recv.float().abs().sum()) == pytest.approx(2 * float(x.float().abs().sum()), rel=1e-3)
    del rows, recv
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    big = MoeWorkspace(4096, 4096, 8, 4)          # 256 MB and more
    assert torch.cuda.mem_get_info()[0] < free - (200 << 20)
    big.close()
    assert torch.cuda.mem_get_info()[0] > free - (64 << 20)


# ----------------------------------------------------------------------------- block-scaled fp8 GEMM
@pytest.mark.parametrize("M,N,K_", [(128, 128, 128), (256, 384, 512), (1000, 256, 1024), (2048, 1024, 2048)])
def test_gemm_fp8_blockscaled_matches_dequantised_reference(dev, M, N, K_):
    from xccl_b200.ops import gemm
    a = torch.randn(M, K_, device=dev) * torch.rand(M, 1, device=dev) * 3
    b = torch.randn(N, K_, device=dev) * 0.05
    a8, sa = gemm.quantize_act_1x128(a)
    b8, sb = gemm.quantize_weight_128x128(b)
    out = gemm.gemm_fp8_blockscaled(a8, sa, b8, sb)
    assert gemm.last_error() == 0
    want = gemm.dequantize(a8, sa, 1) @ gemm.dequantize(b8, sb, 128).t()
    torch.testing.assert_close(out.float(), want, rtol=2e-2, atol=2e-2 * float(want.abs().max()))


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("M,N,K_", [(1409, 1792, 128), (1290, 1920, 256), (2047, 1280, 384), (513, 4096, 512), (2049, 1408, 640), (1300, 1920, 1152)])
def test_gemm_fp8_blockscaled_scale_groups(dev, M, N, K_, off):
    """Scales reach the kernel four K blocks at a time, 16 bytes per row where the rows are aligned: numbers of K blocks
    around the groups, scales that do not start on 16 bytes, a last tile half outside N. (Sizes of the large kernel.)"""
    from xccl_b200.ops import gemm
    a = torch.randn(M, K_, device=dev) * torch.rand(M, 1, device=dev) * 3
    b = torch.randn(N, K_, device=dev) * 0.05 * torch.rand(N // 128, device=dev).repeat_interleave(128)[:, None]
    a8, sa = gemm.quantize_act_1x128(a)
    b8, sb = gemm.quantize_weight_128x128(b)
    moved = torch.full((sa.numel() + 8,), float("nan"), device=dev)[off:off + sa.numel()].view_as(sa)
    moved.copy_(sa)
    out = gemm.gemm_fp8_blockscaled(a8, moved, b8, sb)
    assert gemm.last_error() == 0
    want = gemm.dequantize(a8, sa, 1).double() @ gemm.dequantize(b8, sb, 128).double().t()
    # half a unit in the last place of bf16 (2^-9), and 32-bit sums of K products far below the largest value
    torch.testing.assert_close(out.double(), want, rtol=2 ** -8, atol=1e-5 * float(want.abs().max()))


@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64, 65, 127, 128, 129])
@pytest.mark.parametrize("N,K_", [(8, 8), (264, 520), (1024, 4104)])
def test_gemm_few_rows_matches_fp32_reference(dev, M, N, K_):
    """Row counts around the edges of the few-rows kernel (its MMA takes 16-row steps up to 128), one CTA per weight
    tile and several that share K, ragged last tiles in N and K."""
    from xccl_b200.ops import gemm
    a = torch.randn(M, K_, device=dev).to(torch.bfloat16)
    b = torch.randn(N, K_, device=dev).to(torch.bfloat16)
    guard = torch.full((M + 2, N), 7.0, device=dev, dtype=torch.bfloat16)
    gemm.gemm_bf16(a, b, guard[1:M + 1])
    assert gemm.last_error() == 0
    want = a.float() @ b.float().t()
    # bf16 rounding of the result (2^-9 of it) and of fp32 sums of K products of size 1: far below 1e-2 of sqrt(K)
    torch.testing.assert_close(guard[1:M + 1].float(), want, rtol=1e-2, atol=1e-2 * K_ ** 0.5)
    assert bool((guard[0] == 7).all()) and bool((guard[M + 1] == 7).all())


@pytest.mark.parametrize("M", [1, 33, 100, 128])
@pytest.mark.parametrize("F,K_", [(128, 64), (384, 1000), (2048, 4096)])
def test_gemm_swiglu_few_rows_matches_fp32_reference(dev, M, F, K_):
    from xccl_b200.ops import gemm
    a = torch.randn(M, K_, device=dev).to(torch.bfloat16)
    wg = (torch.randn(F, K_, device=dev) / K_ ** 0.5).to(torch.bfloat16)
    wu = (torch.randn(F, K_, device=dev) / K_ ** 0.5).to(torch.bfloat16)
    out = gemm.gemm_swiglu(a, wg, wu)
    assert gemm.last_error() == 0
    want = torch.nn.functional.silu(a.float() @ wg.float().t()) * (a.float() @ wu.float().t())
    torch.testing.assert_close(out.float(), want, rtol=1e-2, atol=1e-2)   # values of size 1, one bf16 rounding


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("M,N,K_", [(129, 384, 2048), (255, 1024, 4096), (256, 512, 1536), (257, 128, 8192), (700, 256, 4224),
                                    (1300, 384, 1664)])
def test_gemm_blocks_of_few_rows(dev, fp8, M, N, K_):
    """More rows than one MMA in the few-rows kernel: whole and ragged blocks of rows, CTAs that share K and that do not,
    nothing written outside the output."""
    from xccl_b200.ops import gemm
    a = torch.randn(M, K_, device=dev) * (0.2 + torch.rand(M, 1, device=dev))
    b = torch.randn(N, K_, device=dev) * 0.05
    guard = torch.full((M + 2, N), 7.0, device=dev, dtype=torch.bfloat16)
    if fp8:
        a8, sa = gemm.quantize_act_1x128(a)
        b8, sb = gemm.quantize_weight_128x128(b)
        gemm.gemm_fp8_blockscaled(a8, sa, b8, sb, guard[1:M + 1])
        a, b = gemm.dequantize(a8, sa, 1), gemm.dequantize(b8, sb, 128)
    else:
        a, b = a.to(torch.bfloat16), b.to(torch.bfloat16)
        gemm.gemm_bf16(a, b, guard[1:M + 1])
    assert gemm.last_error() == 0
    want = a.double() @ b.double().t()
    # half a unit in the last place of bf16 (2^-9), and 32-bit sums of K products far below the largest value
    torch.testing.assert_close(guard[1:M + 1].double(), want, rtol=2 ** -8, atol=1e-5 * float(want.abs().max()))
    assert bool((guard[0] == 7).all()) and bool((guard[M + 1] == 7).all())


@pytest.mark.parametrize("tokens", [256, 384])
def test_tp_mlp_fp8_blocks_of_few_rows(dev, tokens):
    """The fp8 block on one rank with more rows than one MMA: SwiGLU with its quantised output and the down projection in
    blocks of rows, against the dequantised block with the same rounding steps in between."""
    from xccl_b200.models.tp_mlp import TpMlpFp8
    from xccl_b200.ops import gemm
    mlp = TpMlpFp8(tokens, 1024, 1536)
    try:
        x = torch.randn(tokens, 1024, device=dev).to(torch.bfloat16)
        y = mlp.forward([x])[0]
        mlp.check_error()
        deq = lambda q, s: gemm.dequantize(q, s, 128).double()
        xq = gemm.dequantize(mlp.x8[0], mlp.sx[0], 1).double()
        g, u = xq @ deq(mlp.w_gate8[0], mlp.s_gate[0]).t(), xq @ deq(mlp.w_up8[0], mlp.s_up[0]).t()
        h = g / (1 + torch.exp(-g)) * u
        hq = gemm.dequantize(mlp.h8[0], mlp.sh[0], 1).double()
        # the intermediate: half of an e4m3 spacing (2^-4 of a value; below the smallest normal 2^-10 in units of a 448th of the
        # block's largest value, which is less than 2^-17 of it)
        block = h.view(tokens, -1, 128).abs().amax(-1, keepdim=True).expand(-1, -1, 128).reshape(tokens, -1)
        assert bool(((hq - h).abs() <= (2 ** -4 + 1e-3) * h.abs() + block * 2 ** -17).all())
        want = hq @ deq(mlp.w_down8[0], mlp.s_down[0]).t()
        torch.testing.assert_close(y.double(), want, rtol=2 ** -8, atol=1e-5 * float(want.abs().max()))
    finally:
        mlp.close()


@pytest.mark.parametrize("M", [64, 300])
def test_gemm_swiglu_over_the_range_of_the_gate(dev, M):
    """Gates from far below the range of exp to far above it, and infinities: silu tends to 0 and to the gate."""
    from xccl_b200.ops import gemm
    F = 1024
    a = torch.zeros(M, 128, device=dev, dtype=torch.bfloat16)
    a[:, 0] = 1
    gate = torch.linspace(-130, 130, F, device=dev).to(torch.bfloat16)
    gate[0], gate[-1] = -3e38, float("inf")
    wg = torch.zeros(F, 128, device=dev, dtype=torch.bfloat16)
    wg[:, 0] = gate
    wu = torch.zeros_like(wg)
    wu[:, 0] = 1
    out = gemm.gemm_swiglu(a, wg, wu).double()
    assert gemm.last_error() == 0
    g = gate.double()
    want = g / (1 + torch.exp(-g))
    got, want = out[:, 1:-1], want[1:-1].expand(M, -1)
    # half a unit of bf16 and what exp loses at 130 (2^-21 per unit of the exponent); below 2^-126 bf16 has steps of 2^-133
    torch.testing.assert_close(got, want, rtol=2 ** -8, atol=2 ** -133)
    assert bool((out[:, 0] == 0).all()) and bool((out[:, -1] == float("inf")).all())   # the gate is 1 x the weight


@pytest.mark.parametrize("M", [1, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("N,K_", [(128, 128), (384, 1152), (1024, 8192)])
def test_gemm_fp8_few_rows_matches_dequantised_reference(dev, M, N, K_):
    from xccl_b200.ops import gemm
    a = torch.randn(M, K_, device=dev) * torch.rand(M, 1, device=dev) * 3
    b = torch.randn(N, K_, device=dev) * 0.05
    a8, sa = gemm.quantize_act_1x128(a)
    b8, sb = gemm.quantize_weight_128x128(b)
    out = gemm.gemm_fp8_blockscaled(a8, sa, b8, sb)
    assert gemm.last_error() == 0
    want = gemm.dequantize(a8, sa, 1) @ gemm.dequantize(b8, sb, 128).t()
    torch.testing.assert_close(out.float(), want, rtol=1e-2, atol=1e-2 * float(want.abs().max()))


@pytest.mark.parametrize("fp8", [False, True])
def test_tp_mlp_one_block_of_rows_matches_reference(dev, fp8):
    """The block with 128 tokens on one rank: both products run in the few-rows kernel, in fp8 with the intermediate
    quantised by it."""
    from xccl_b200.models.tp_mlp import TpMlp, TpMlpFp8, reference_forward_fp32
    mlp = (TpMlpFp8 if fp8 else TpMlp)(128, 1024, 2048, tp=1)
    try:
        x = torch.randn(128, 1024, device=dev).to(torch.bfloat16)
        for _ in range(2):
            got = mlp.forward([x])[0].float()
            mlp.check_error()
        want = reference_forward_fp32(x, *_full_weights(mlp))
        # bf16: two roundings of 2^-9; fp8: 2^-4 per quantised operand, averaged over the sums
        tol = 0.08 if fp8 else 0.02
        assert float((got - want).abs().max()) <= tol * float(want.abs().max()) + 1e-3
    finally:
        mlp.close()


_TILE_SCRIPT = r"""
import torch
from xccl_b200.ops import gemm
from xccl_b200.models.tp_mlp import TpMlp, reference_forward_fp32
dev = torch.device("cuda:0")
g = torch.Generator(device=dev).manual_seed(1)
R = lambda *s, scale=1.0: (torch.randn(*s, device=dev, generator=g) * scale).to(torch.bfloat16)
for M, N, K in ((129, 8, 64), (257, 264, 136), (400, 1000, 520), (640, 232, 4104)):
    a, b = R(M, K), R(N, K)
    out = torch.full((M + 2, N), 7.0, device=dev, dtype=torch.bfloat16)
    gemm.gemm_bf16(a, b, out[1:M + 1])
    # bf16 rounding of the result (2^-8 of it) and fp32 sums of K products of size 1
    torch.testing.assert_close(out[1:M + 1].float(), a.float() @ b.float().t(), rtol=1e-2, atol=1e-2 * K ** 0.5)
    assert bool((out[0] == 7).all()) and bool((out[M + 1] == 7).all())
for M, F, K in ((129, 128, 64), (300, 384, 1000)):
    a, wg, wu = R(M, K), R(F, K, scale=K ** -0.5), R(F, K, scale=K ** -0.5)
    out = torch.full((M + 2, F), 7.0, device=dev, dtype=torch.bfloat16)
    gemm.gemm_swiglu(a, wg, wu, out[1:M + 1])
    want = torch.nn.functional.silu(a.float() @ wg.float().t()) * (a.float() @ wu.float().t())
    torch.testing.assert_close(out[1:M + 1].float(), want, rtol=1e-2, atol=1e-2)
    assert bool((out[0] == 7).all()) and bool((out[M + 1] == 7).all())
assert gemm.last_error() == 0
for tokens, tp in ((512, 2), (768, 2), (384, 3)):      # shards of whole 256-row tiles and of single 128-row blocks
    mlp = TpMlp(tokens, 264, 384 * tp, tp=tp)
    x = R(tokens, 264)
    for _ in range(2):
        y = torch.cat(mlp.forward(list(x.chunk(tp, 0))), 0).float()
        mlp.check_error()
    want = reference_forward_fp32(x, torch.cat(mlp.w_gate, 0), torch.cat(mlp.w_up, 0), torch.cat(mlp.w_down, 1))
    # two bf16 roundings and one of every rank's partial sum
    assert float((y - want).abs().max()) <= 0.02 * float(want.abs().max()) + 1e-3, (tokens, tp)
    mlp.close()
print("tiles ok")
"""


@pytest.mark.parametrize("cols,pair", [(32, "y"), (32, "n"), (64, "n"), (160, "y"), (224, "y"), (224, "n")])
def test_gemm_tiles_of_every_kind_of_width(dev, cols, pair):
    """Tiles of a width that is asked for, as CTA pairs and as single CTAs (whose second half of B follows the first at
    half a tile), over ragged rows and columns and through the allgather and reduce-scatter forms. The options are read
    once per process."""
    import subprocess
    import sys
    from pathlib import Path
    env = dict(os.environ, PYTHONPATH=str(Path(__file__).resolve().parent.parent), XCCL_TP_GEMM_BN=str(cols), XCCL_TP_GEMM_PAIR=pair)
    r = subprocess.run([sys.executable, "-c", _TILE_SCRIPT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "tiles ok" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]


def test_quantize_rows_kernel_matches_torch(dev):
    from xccl_b200.ops import gemm
    from xccl_b200.ops.tp import quantize_rows
    x = (torch.randn(300, 512, device=dev) * torch.rand(300, 1, device=dev) * 5).to(torch.bfloat16)
    x[7, 128:256] = 0  # an all-zero block keeps a finite scale
    out8 = torch.empty(300, 512, dtype=torch.float8_e4m3fn, device=dev)
    s = torch.empty(300, 4, dtype=torch.float32, device=dev)
    quantize_rows(x, out8, s)
    torch.cuda.synchronize()
    q_ref, s_ref = gemm.quantize_act_1x128(x.float())
    torch.testing.assert_close(s, s_ref, rtol=1e-6, atol=0)
    # x / s and x * (1 / s) may round differently by one e4m3 step: compare the dequantised values
    got, want = gemm.dequantize(out8, s, 1), gemm.dequantize(q_ref, s_ref, 1)
    assert float((got - want).abs().max()) <= float(s.max()) * 32 + 1e-6   # one step at the top binade of e4m3
    torch.testing.assert_close(got, x.float(), rtol=0.07, atol=1e-3)
    _loaded_native()


@pytest.mark.parametrize("rows,shift", [(1, 0), (1, 4), (9, 0), (63, 4), (64, 8), (65, 0)])
def test_quantize_rows_edges_of_the_grid_and_alignments(dev, rows, shift):
    """Block counts around a thread block's 64, an input that is only 8-byte aligned, and bytes behind the output."""
    from xccl_b200.ops import gemm
    from xccl_b200.ops.tp import quantize_rows
    flat = (torch.randn(rows * 128 + 16, device=dev) * 3).to(torch.bfloat16)
    x = flat[shift: shift + rows * 128].view(rows, 128)
    out = torch.zeros(rows * 128 + 64, dtype=torch.uint8, device=dev)
    s = torch.full((rows + 1,), -1.0, device=dev)
    quantize_rows(x, out[: rows * 128].view(torch.float8_e4m3fn).view(rows, 128), s[:rows].view(rows, 1))
    scale = x.float().abs().amax(-1, keepdim=True).clamp_min(1e-12) / gemm.FP8_MAX
    torch.testing.assert_close(s[:rows, None], scale, rtol=1e-6, atol=0)
    want = (x.float() * (1.0 / s[:rows, None])).to(torch.float8_e4m3fn)   # the same product, rounded once
    assert torch.equal(out[: rows * 128].view(torch.float8_e4m3fn).view(rows, 128).float(), want.float())
    assert float(s[rows]) == -1.0 and int(out[rows * 128:].sum()) == 0


@pytest.mark.parametrize("tp,fuse_quant", [(1, True), (2, True), (4, True), (2, False)])
def test_tp_mlp_fp8_fused_matches_dequantised_reference(dev, tp, fuse_quant):
    """fp8 allgather->GEMM+SwiGLU and GEMM->reduce-scatter (ranks emulated in one launch) against fp32
    products of exactly the quantised operands the kernels consumed."""
    from xccl_b200.models.tp_mlp import TpMlpFp8
    from xccl_b200.ops import gemm
    tokens, hidden, ffn = 1024, 512, 1024
    mlp = TpMlpFp8(tokens, hidden, ffn, tp=tp, emulate=True, fuse_quant=fuse_quant)
    try:
        g = torch.Generator(device=dev).manual_seed(6)
        x = torch.randn(tokens, hidden, device=dev, generator=g).to(torch.bfloat16)
        shards = list(x.chunk(tp, 0))
        for it in range(3):
            y = mlp.forward(shards)
            mlp.check_error()
            xq = gemm.dequantize(torch.cat(mlp.x8, 0), torch.cat(mlp.sx, 0), 1)
            y_want = torch.zeros(tokens, hidden, device=dev)
            for r in range(tp):
                wg = gemm.dequantize(mlp.w_gate8[r], mlp.s_gate[r], 128)
                wu = gemm.dequantize(mlp.w_up8[r], mlp.s_up[r], 128)
                wd = gemm.dequantize(mlp.w_down8[r], mlp.s_down[r], 128)
                h_want = torch.nn.functional.silu(xq @ wg.t()) * (xq @ wu.t())
                if fuse_quant:
                    # the intermediate exists only as e4m3 with 1 x 128 scales: one e4m3 step (2^-3 relative) of the
                    # block maximum at most, and scales that are the block maxima over 448
                    h_got = gemm.dequantize(mlp.h8[r], mlp.sh[r], 1)
                    blk = h_want.view(tokens, -1, 128).abs().amax(-1)
                    torch.testing.assert_close(mlp.sh[r] * 448.0, blk.clamp_min(1e-12 * 448), rtol=3e-2, atol=1e-6)
                    assert float(((h_got - h_want).abs().view(tokens, -1, 128).amax(-1) / blk.clamp_min(1e-6)).max()) <= 0.07
                else:
                    torch.testing.assert_close(mlp.h[r].float(), h_want, rtol=2e-2, atol=2e-2 * float(h_want.abs().max()))
                y_want += gemm.dequantize(mlp.h8[r], mlp.sh[r], 1) @ wd.t()
            got = torch.cat(y, 0).float()
            torch.testing.assert_close(got, y_want, rtol=2e-2, atol=2e-2 * float(y_want.abs().max()))
            # and the whole block stays close to the unquantised fp32 block
            from xccl_b200.models.tp_mlp import reference_forward_fp32
            full = reference_forward_fp32(x, *_full_weights(mlp))
            assert float((got - full).abs().max()) <= 0.08 * float(full.abs().max()) + 1e-3
    finally:
        mlp.close()
    _loaded_native()


def test_silu_is_as_exact_as_a_rounded_division(dev):
    """silu in 32 bits against 64: what the fast exponential is documented to lose (2 + 1.173 |x| units of 2^-23, of which the
    quotient keeps the share e^-x / (1 + e^-x)), half a unit for the sum and half for a rounded division (1e-9 for the
    squares of these). A quotient that is good to two units only lies outside."""
    import ctypes as C
    n = 1 << 21
    g = torch.Generator(device=dev).manual_seed(3)
    x = torch.cat([torch.randn(n, device=dev, generator=g) * 4, torch.rand(n, device=dev, generator=g) * 200 - 100,
                   torch.tensor([0.0, -0.0, 1e-30, -1e-30, 16.7, 88.8, -86.99, -87.0, -87.01, -88.7, 3e38], device=dev)])
    y = torch.empty_like(x)
    fn = K.load().xccl_tp_silu
    fn.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p]
    assert fn(x.data_ptr(), y.data_ptr(), x.numel(), torch.cuda.current_stream().cuda_stream) == K.OK
    xd = x.double()
    want = xd / (1 + torch.exp(-xd))
    lost = (2 + 1.173 * xd.abs()) * 2.0 ** -23 * torch.sigmoid(-xd) + 2.0 ** -23 + 1e-9
    assert bool(((y.double() - want).abs() <= lost * want.abs() + 2.0 ** -149).all())
    ends = torch.tensor([float("inf"), float("-inf"), float("nan"), -3e38], device=dev)
    out = torch.empty_like(ends)
    assert fn(ends.data_ptr(), out.data_ptr(), 4, torch.cuda.current_stream().cuda_stream) == K.OK
    out = out.tolist()
    assert out[0] == float("inf") and out[1] != out[1] and out[2] != out[2] and out[3] == 0


@pytest.mark.parametrize("tp,tokens,hidden,ffn", [(2, 2048, 1152, 3840), (2, 2048, 2048, 4096), (4, 2048, 1152, 4608), (4, 2048, 2048, 4096),
                                                   (2, 1024, 1280, 2816), (4, 1024, 1408, 3072), (2, 256, 1664, 2048)])
def test_tp_mlp_fp8_walkers_of_local_and_gathered_tiles(dev, tp, tokens, hidden, ffn):
    """The fp8 block over emulated ranks with three to four tiles for every walker, local rows first and gathered rows after
    them: scales that differ strongly from row to row and from K block to K block reach the right tile, and those of gathered
    rows are read when they have arrived. K in groups of four blocks (16-byte scale loads) and every remainder; the last three
    sizes have a tile or two per walker, of single CTAs in the very last."""
    from xccl_b200.models.tp_mlp import TpMlpFp8
    from xccl_b200.ops import gemm
    mlp = TpMlpFp8(tokens, hidden, ffn, tp=tp, emulate=True, fuse_quant=False)
    g = torch.Generator(device=dev).manual_seed(11)
    # powers of two, one per block of 128
    steps = lambda n, lo, hi: torch.exp2(torch.randint(lo, hi + 1, (n // 128,), device=dev, generator=g).float()).repeat_interleave(128)
    try:
        for r in range(tp):
            for name, w, q, s in (("gate", mlp.w_gate, mlp.w_gate8, mlp.s_gate), ("up", mlp.w_up, mlp.w_up8, mlp.s_up),
                                  ("down", mlp.w_down, mlp.w_down8, mlp.s_down)):
                rows, cols = w[r].shape
                v = torch.randn(rows, cols, device=dev, generator=g) * 0.02 * steps(rows, -2, 2)[:, None] * steps(cols, -2, 2)
                w[r].copy_(v)
                q8, sc = gemm.quantize_weight_128x128(w[r])
                q[r].copy_(q8)
                s[r].copy_(sc)
        deq = lambda q, s, b: gemm.dequantize(q, s, b).double()
        for it in range(3):
            x = torch.randn(tokens, hidden, device=dev, generator=g) * steps(hidden, -2, 2)
            x = (x * torch.exp2(torch.randint(-3, 3, (tokens, 1), device=dev, generator=g).float())).to(torch.bfloat16)
            y = mlp.forward(list(x.chunk(tp, 0)))
            mlp.check_error()
            xq = deq(torch.cat(mlp.x8, 0), torch.cat(mlp.sx, 0), 1)
            want, lost = torch.zeros(tokens, hidden, dtype=torch.float64, device=dev), 0.0
            for r in range(tp):
                gate, up = xq @ deq(mlp.w_gate8[r], mlp.s_gate[r], 128).t(), xq @ deq(mlp.w_up8[r], mlp.s_up[r], 128).t()
                h = gate / (1 + torch.exp(-gate)) * up
                # half a unit of bf16 (2^-9), and 32-bit sums: far below 2e-5 of the row's largest gate and up values, of which
                # silu (slope at most 1.1) passes on both products
                sums = 2.1 * 2e-5 * gate.abs().amax(-1, keepdim=True) * up.abs().amax(-1, keepdim=True)
                assert bool(((mlp.h[r].double() - h).abs() <= 2 ** -8 * h.abs() + sums).all())
                part = deq(mlp.h8[r], mlp.sh[r], 1) @ deq(mlp.w_down8[r], mlp.s_down[r], 128).t()
                want += part
                lost = lost + 2 ** -8 * part.abs() + 2e-5 * part.abs().amax(-1, keepdim=True)   # every partial tile travels as bf16
            assert bool(((torch.cat(y, 0).double() - want).abs() <= lost + 2 ** -8 * want.abs()).all())
    finally:
        mlp.close()


@pytest.mark.parametrize("n,blocks", [(2, 0), (4, 3), (8, 0), (8, 18)])
@pytest.mark.parametrize("packs", [1, 31, 513, 2047, 2049, 18 * 2048 + 33, 40000])
def test_emu_direct_turns_of_the_blocks(dev, n, blocks, packs):
    """Zero-copy collectives whose segments give a block a part of one tile, a whole one and several: every pack arrives, and
    nothing behind a destination is written."""
    from xccl_b200.ops.emu import EmuWorld
    w = EmuWorld(n, 8 << 20)
    D, per = K.NVLINK_ALG_DIRECT, packs * 4          # fp32 values of a segment
    tail = lambda size: [torch.full((size + 64,), -7.0, device=dev) for _ in range(n)]
    try:
        src = _ints(n, per * n, torch.float32, dev, seed=packs)
        run = lambda op, ins, size, **kw: (lambda full: (getattr(w, op)(ins, [f[:size] for f in full], alg=D, **kw), full)[1])(tail(size))
        total = torch.stack(src).sum(0)
        want = {"allreduce": [total] * n, "reduce_scatter": list(total.chunk(n)),
                "allgather": [torch.cat([s[:per] for s in src])] * n,
                "alltoall": [torch.cat([s[r * per:(r + 1) * per] for s in src]) for r in range(n)]}
        for op, expected in want.items():
            ins = [s[:per] for s in src] if op == "allgather" else src
            kw = {"blocks": blocks} if op == "allreduce" else {}
            for got, e in zip(run(op, ins, e_size := expected[0].numel(), **kw), expected):
                assert torch.equal(got[:e_size], e), op
                assert bool((got[e_size:] == -7).all()), op
    finally:
        w.close()


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("M,N,K_", [(4096, 4096, 1024), (4096, 4096, 1152), (4000, 4224, 1280), (4096, 4096, 1408), (4096, 6144, 128), (3968, 4096, 2048)])
def test_gemm_fp8_blockscaled_many_tiles_per_walker(dev, M, N, K_, off):
    """Three to four tiles for every CTA pair of the large kernel: the scale ring, its phases and the scales loaded ahead go over
    from tile to tile, for every remainder of the K blocks by four and for scales that do not start on 16 bytes. Scales differ by
    powers of two from row to row and from K block to K block, so one that is a block off shows."""
    from xccl_b200.ops import gemm
    assert K.load().xccl_tp_skinny_plan_rows(M, N, K_, 1, 0, 148, (C.c_int * 11)()) == 0     # the large kernel's
    g = torch.Generator(device=dev).manual_seed(M + N + K_)
    steps = lambda n: torch.exp2(torch.randint(-3, 4, (n // 128,), device=dev, generator=g).float()).repeat_interleave(128)
    a = torch.randn(M, K_, device=dev, generator=g) * torch.exp2(torch.randint(-3, 4, (M, 1), device=dev, generator=g).float()) * steps(K_)
    b = torch.randn(N, K_, device=dev, generator=g) * 0.05 * steps(N)[:, None] * steps(K_)
    a8, sa = gemm.quantize_act_1x128(a)
    b8, sb = gemm.quantize_weight_128x128(b)
    moved = torch.full((sa.numel() + 8,), float("nan"), device=dev)[off:off + sa.numel()].view_as(sa)
    moved.copy_(sa)
    guard = torch.full((M + 2, N), 7.0, device=dev, dtype=torch.bfloat16)
    for _ in range(2):
        gemm.gemm_fp8_blockscaled(a8, moved, b8, sb, guard[1:M + 1])
    assert gemm.last_error() == 0
    want = gemm.dequantize(a8, sa, 1).double() @ gemm.dequantize(b8, sb, 128).double().t()
    # half a unit in the last place of bf16 (2^-9), and 32-bit sums of K products far below the largest value of the row
    assert bool(((guard[1:M + 1].double() - want).abs() <= 2 ** -8 * want.abs() + 2e-5 * want.abs().amax(-1, keepdim=True)).all())
    assert bool((guard[0] == 7).all()) and bool((guard[M + 1] == 7).all())


_COPIER_SCRIPT = r"""
import torch
from xccl_b200.models.tp_mlp import TpMlp, TpMlpFp8, reference_forward_fp32
from xccl_b200.ops import gemm
g = torch.Generator(device="cuda").manual_seed(4)
for fp8, hidden in ((False, 8), (False, 136), (False, 2056), (True, 128), (True, 384), (True, 2176)):
    for tp, tokens in ((2, 256), (2, 1280), (4, 1536), (3, 384)):
        mlp = (TpMlpFp8 if fp8 else TpMlp)(tokens, hidden, 256 * tp, tp=tp)
        x = torch.randn(tokens, hidden, device="cuda", generator=g).to(torch.bfloat16)
        for _ in range(2):
            x = x.roll(1, 0)
            y = torch.cat(mlp.forward(list(x.chunk(tp, 0))), 0).float()
            mlp.check_error()
        want = reference_forward_fp32(x, torch.cat(mlp.w_gate, 0), torch.cat(mlp.w_up, 0), torch.cat(mlp.w_down, 1))
        # bf16: two roundings and one of every rank's partial sum; fp8: 2^-4 per quantised operand, averaged over the sums
        assert float((y - want).abs().max()) <= (0.08 if fp8 else 0.02) * float(want.abs().max()) + 1e-3, (fp8, hidden, tp, tokens)
        mlp.close()
print("copiers ok")
"""


def test_tp_mlp_copier_warps_over_blocks_and_shards(dev):
    """Copier warps (asked for on more ranks than they are chosen for): shares of a row block from none and one pack to several
    batches, several row blocks and shards, a last batch that is not full."""
    import subprocess
    import sys
    from pathlib import Path
    env = dict(os.environ, PYTHONPATH=str(Path(__file__).resolve().parent.parent), XCCL_TP_COPY_MODE="1")
    r = subprocess.run([sys.executable, "-c", _COPIER_SCRIPT], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "copiers ok" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]
