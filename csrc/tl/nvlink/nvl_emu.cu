// Single-GPU emulation of an N-rank NVLink world (see nvl_world.h).
#include <algorithm>
#include <cstring>

#include "../../cuda/cuda_common.h"
#include "nvl_world.h"

namespace xccl {
namespace nvl {

EmuWorld::~EmuWorld()
{
    for (void *p : allocs_) cudaFree(p);
    if (status_host_ != nullptr) cudaFreeHost(status_host_);
}

xccl_status_t EmuWorld::create(int nranks, size_t ws_bytes, EmuWorld **out)
{
    if (nranks < 1 || nranks > kMaxRanks || ws_bytes < (1u << 16)) return XCCL_ERR_INVALID_PARAM;
    if (!cuda_available()) return XCCL_ERR_NO_RESOURCE;
    auto *e = new EmuWorld;
    ws_bytes &= ~(size_t)511;
    World &w      = e->world;
    w.size        = nranks;
    w.rank_base   = 0;
    w.n_local     = nranks;
    w.mc_ws       = nullptr;
    w.ws_bytes    = ws_bytes;
    w.wait_budget_ns = e->budget_ns;
    cudaError_t err = cudaHostAlloc((void **)&e->status_host_, sizeof(HostStatus) * kMaxRanks, cudaHostAllocMapped);
    if (err != cudaSuccess) {
        delete e;
        return cuda_status(err);
    }
    std::memset(e->status_host_, 0, sizeof(HostStatus) * kMaxRanks);
    HostStatus *sdev = nullptr;
    cudaHostGetDevicePointer((void **)&sdev, e->status_host_, 0);
    for (int r = 0; r < nranks; r++) {
        void *pad = nullptr, *ws = nullptr;
        if (cudaMalloc(&pad, kPadBytes) != cudaSuccess || cudaMalloc(&ws, ws_bytes) != cudaSuccess) {
            (void)cudaGetLastError();
            if (pad != nullptr) cudaFree(pad);
            delete e;
            return XCCL_ERR_NO_MEMORY;
        }
        e->allocs_.push_back(pad);
        e->allocs_.push_back(ws);
        cudaMemset(pad, 0, kPadBytes);
        w.pad[r]    = (uint32_t *)pad;
        w.ws[r]     = (char *)ws;
        w.status[r] = (uint32_t *)(sdev + r);
    }
    cudaDeviceSynchronize();
    *out = e;
    return XCCL_OK;
}

HostStatus EmuWorld::status(int i) const { return status_host_[i]; }

void EmuWorld::clear_status() { std::memset(status_host_, 0, sizeof(HostStatus) * kMaxRanks); }

int chunks_used(const World &w, xccl_collective_type_t coll, size_t count, size_t len, xccl_dt_t dt, bool multicast)
{
    const size_t half = w.ws_bytes / 2, cap = half / 16;
    const size_t es   = std::max<size_t>(xccl_dt_size(dt), 1);
    size_t       packs = 0, div = 1;
    switch (coll) {
    case XCCL_ALLREDUCE:
    case XCCL_REDUCE: packs = (count * es + 15) / 16; break;
    case XCCL_REDUCE_SCATTER:
        packs = (count * es + 15) / 16;
        div   = (size_t)w.size;
        break;
    case XCCL_BCAST: packs = (len + 15) / 16; break;
    case XCCL_ALLGATHER: packs = (len / (size_t)w.size + 15) / 16; break;
    case XCCL_ALLTOALL:
        packs = (len + 15) / 16;
        div   = (size_t)w.size;
        break;
    default: return 1;
    }
    size_t c = std::max<size_t>(cap / div, 1);
    if (coll == XCCL_BCAST && multicast && w.mc_bcast_cap != 0) c = std::min(c, w.mc_bcast_cap);  // as in mover_kernel
    return (int)std::max<size_t>((packs + c - 1) / c, 1);
}

}  // namespace nvl
}  // namespace xccl

using namespace xccl;
using namespace xccl::nvl;

namespace {

// Whether a collective for which no algorithm was named runs zero-copy on the user buffers (they are all on this device).
// The staged kernels pass every byte through the workspaces, which costs little while that traffic stays in L2 and
// doubles the DRAM traffic beyond it; the zero-copy kernels have one barrier more. Measured on one B200 per call (warm buffers),
// staged / zero-copy in us, by the bytes of all ranks together, on both sides of the limits: allreduce fp32 8 ranks 6 MB 34.2 / 29.8, 10 MB
// 37.5 / 29.8, 4 ranks 6 MB 32.3 / 27.2, 10 MB 34.4 / 28.7, 2 ranks 14 MB 34.4 / 29.0, 20 MB 38.5 / 30.7; reduce-scatter fp32 2 ranks 28 MB
// 33.6 / 28.6, 36 MB 43.7 / 29.3, 4 ranks 28 MB 35.8 / 27.7, 36 MB 43.7 / 28.0, 8 ranks 12 MB 29.3 / 28.1, 20 MB 33.1 / 28.9, bf16 4 ranks 12 MB
// 28.1 / 27.1, 20 MB 32.5 / 28.0; allgather 2 ranks 90 MB 69.6 / 52.6, 112 MB 81.8 / 57.5, 4 ranks 90 MB 56.5 / 51.6, 112 MB 63.7 / 56.8, 6 ranks
// 112 MB 59.2 / 59.6, 128 MB 70.3 / 60.5, 8 ranks 144 MB 65.7 / 60.8, 192 MB 97.0 / 70.6; alltoall 4 ranks 28 MB 41.8 / 36.0, 36 MB 53.6 / 37.5, 8 ranks
// 44 MB 58.7 / 41.4, 64 MB 86.3 / 48.7. Zero-copy is not slower anywhere above its limit. Most limits were drawn for zero-copy kernels
// that were slower and lie above the crossover: it is at or below 2 MB for allreduce, at 12 MB for reduce-scatter, 24 to 28 MB for alltoall,
// and for allgather at 48 MB (2 ranks), 64 MB (4), 80 MB (6) and 96 MB (8).
bool direct_pays(const World &w, const Call &c, int coll, xccl_dt_t dt, xccl_dt_t out_dt)
{
    if (out_dt == XCCL_DT_UNSUPPORTED || out_dt == XCCL_DT_LAST_PREDEFINED) out_dt = dt;
    const size_t n = (size_t)w.size, es = xccl_dt_size(dt);
    const bool   typed = (dt == XCCL_DT_FLOAT32 && (out_dt == XCCL_DT_FLOAT32 || out_dt == XCCL_DT_BFLOAT16)) ||
                         ((dt == XCCL_DT_BFLOAT16 || dt == XCCL_DT_FLOAT16) && out_dt == dt);
    size_t src_bytes = 0, dst_bytes = 0, least = 0;
    switch (coll) {
    case XCCL_ALLREDUCE:
        if (!typed) return false;
        src_bytes = c.count * es;
        dst_bytes = c.count * xccl_dt_size(out_dt);
        least     = n >= 4 ? (size_t)8 << 20 : (size_t)16 << 20;
        break;
    case XCCL_REDUCE_SCATTER:
        if (!typed) return false;
        src_bytes = c.count * es * n;
        dst_bytes = c.count * xccl_dt_size(out_dt);
        least     = (size_t)(es >= 4 && n < 8 ? 32 : 16) << 20;
        break;
    case XCCL_ALLGATHER:
        src_bytes = c.len / n;
        dst_bytes = c.len;
        least     = (size_t)(n >= 8 ? 160 : n >= 6 ? 120 : 100) << 20;
        break;
    case XCCL_ALLTOALL:
        src_bytes = dst_bytes = c.len * n;
        least     = (size_t)(n >= 8 ? 48 : 32) << 20;
        break;
    default: return false;
    }
    if (std::max(src_bytes, dst_bytes) * n < least || !direct_shape_ok(coll, c, dt, w.size)) return false;
    // Nobody may write where another rank still reads: a destination is apart from every source, or it is the rank's own
    // source in place (allreduce: a pack is read and written by one thread; allgather: its own segment).
    for (size_t r = 0; r < n; r++) {
        const char *d = (const char *)c.dst[r];
        if (d == nullptr || ((uintptr_t)d & 15) != 0) return false;
        for (size_t q = 0; q < n; q++) {
            const char *s = (const char *)c.src[q];
            if (d + dst_bytes <= s || s + src_bytes <= d) continue;
            const bool in_place = r == q && ((coll == XCCL_ALLREDUCE && s == d && src_bytes == dst_bytes) ||
                                             (coll == XCCL_ALLGATHER && s == d + r * src_bytes));
            if (!in_place) return false;
        }
    }
    return true;
}

}  // namespace

extern "C" {

xccl_status_t xccl_nvlink_emu_create(int nranks, size_t ws_bytes, void **world)
{
    EmuWorld     *e  = nullptr;
    xccl_status_t st = EmuWorld::create(nranks, ws_bytes, &e);
    if (st == XCCL_OK) *world = e;
    return st;
}

void xccl_nvlink_emu_destroy(void *world) { delete (EmuWorld *)world; }

xccl_status_t xccl_nvlink_emu_collective(void *world, int coll_type, const void *const *srcs, void *const *dsts,
                                         size_t count, size_t len, int dt, int out_dt, int op, int root, float scale,
                                         int alg, const uint32_t *const *vmeta, size_t max_src_bytes, int es,
                                         int blocks, void *stream)
{
    auto *e = (EmuWorld *)world;
    World w = e->world;
    Call  c{};
    for (int r = 0; r < w.size; r++) {
        c.src[r]   = srcs != nullptr ? srcs[r] : nullptr;
        c.dst[r]   = dsts != nullptr ? dsts[r] : nullptr;
        c.vmeta[r] = vmeta != nullptr ? vmeta[r] : nullptr;
    }
    c.count    = count;
    c.len      = len;
    c.op       = op;
    c.root     = root;
    c.scale    = scale;
    c.do_scale = (scale != 1.0f);
    c.parity   = e->parity & 1;
    c.src_es = c.dst_es = es;
    c.push   = (alg == ALG_ONE_SHOT && (coll_type == XCCL_ALLGATHER || coll_type == XCCL_ALLTOALL) && push_fits(w, coll_type, len)) ? 1 : 0;
    LaunchCfg cfg;
    cfg.cooperative = true;
    cfg.blocks      = blocks;
    cudaStream_t  s = (cudaStream_t)stream;
    xccl_status_t st;
    // emulated ranks share one address space: the "registered" peer buffers are the buffers themselves (in the zero-copy
    // call alone: a staged kernel has no business in a peer's buffer, and the bounds-checking build holds it to that)
    Call direct = c;
    for (int r = 0; r < w.size; r++) {
        direct.peer_src[r] = c.src[r];
        direct.peer_dst[r] = c.dst[r];
    }
    if (alg == ALG_AUTO && direct_pays(w, direct, coll_type, (xccl_dt_t)dt, (xccl_dt_t)out_dt)) alg = ALG_DIRECT;
    if (alg == ALG_DIRECT) {
        st = launch_direct(w, direct, coll_type, (xccl_dt_t)dt, (xccl_dt_t)out_dt, cfg, s);
        if (st != XCCL_OK) return st;
        XCCL_CUDA_CHECK(cudaStreamSynchronize(s));
        for (int r = 0; r < w.size; r++) {
            if (e->status(r).code == NVL_TIMEOUT) return XCCL_ERR_TIMED_OUT;
            if (e->status(r).code != NVL_OK) return XCCL_ERR_NO_MESSAGE;
        }
        return XCCL_OK;
    }
    switch (coll_type) {
    case XCCL_ALLREDUCE: {
        Alg a = (Alg)alg;
        if (a == ALG_AUTO) a = (count * xccl_dt_size((xccl_dt_t)dt) <= one_shot_limit(w) / 4) ? ALG_ONE_SHOT : ALG_TWO_SHOT;
        st = launch_allreduce(w, c, (xccl_dt_t)dt, (xccl_dt_t)out_dt, a, cfg, s);
        e->parity += (a == ALG_ONE_SHOT) ? 1 : chunks_used(w, XCCL_ALLREDUCE, count, len, (xccl_dt_t)dt);
        break;
    }
    case XCCL_REDUCE:
        st = launch_reduce(w, c, (xccl_dt_t)dt, (xccl_dt_t)out_dt, cfg, s);
        e->parity += chunks_used(w, XCCL_REDUCE, count, len, (xccl_dt_t)dt);
        break;
    case XCCL_REDUCE_SCATTER:
        st = launch_reduce_scatter(w, c, (xccl_dt_t)dt, (xccl_dt_t)out_dt, cfg, s);
        e->parity += chunks_used(w, XCCL_REDUCE_SCATTER, count, len, (xccl_dt_t)dt);
        break;
    case XCCL_BCAST:
        st = launch_bcast(w, c, cfg, s);
        e->parity += chunks_used(w, XCCL_BCAST, count, len, (xccl_dt_t)dt);
        break;
    case XCCL_ALLGATHER:
        st = launch_allgather(w, c, cfg, s);
        e->parity += chunks_used(w, XCCL_ALLGATHER, count, len, (xccl_dt_t)dt);
        break;
    case XCCL_ALLTOALL:
        st = launch_alltoall(w, c, cfg, s);
        e->parity += chunks_used(w, XCCL_ALLTOALL, count, len, (xccl_dt_t)dt);
        break;
    case XCCL_ALLTOALLV:
        st = launch_alltoallv(w, c, max_src_bytes, cfg, s);
        e->parity += 1;
        break;
    case XCCL_BARRIER:
    case XCCL_FANIN:
    case XCCL_FANOUT: st = launch_sync(w, c, coll_type, cfg, s); break;
    default: st = XCCL_ERR_UNSUPPORTED;
    }
    if (st != XCCL_OK) return st;
    XCCL_CUDA_CHECK(cudaStreamSynchronize(s));
    for (int r = 0; r < w.size; r++) {
        if (e->status(r).code == NVL_TIMEOUT) return XCCL_ERR_TIMED_OUT;
        if (e->status(r).code != NVL_OK) return XCCL_ERR_NO_MESSAGE;
    }
    return XCCL_OK;
}

// Whether a collective on these buffers runs zero-copy when no algorithm is named (tests; the buffers are not touched).
int xccl_nvlink_emu_direct_pays(int nranks, int coll_type, const void *const *srcs, void *const *dsts, size_t count, size_t len,
                                int dt, int out_dt)
{
    World w{};
    Call  c{};
    w.size = nranks;
    for (int r = 0; r < nranks; r++) {
        c.src[r] = c.peer_src[r] = srcs[r];
        c.dst[r] = c.peer_dst[r] = dsts[r];
    }
    c.count = count;
    c.len   = len;
    return direct_pays(w, c, coll_type, (xccl_dt_t)dt, (xccl_dt_t)out_dt) ? 1 : 0;
}

xccl_status_t xccl_nvlink_emu_timeout_probe(void *world, int budget_ms, float *elapsed_ms, uint32_t *status4)
{
    auto *e = (EmuWorld *)world;
    e->clear_status();
    cudaEvent_t e0, e1;
    XCCL_CUDA_CHECK(cudaEventCreate(&e0));
    XCCL_CUDA_CHECK(cudaEventCreate(&e1));
    XCCL_CUDA_CHECK(cudaEventRecord(e0, nullptr));
    World w   = e->world;
    w.n_local = 1;  // only rank 0 probes
    xccl_status_t st = launch_timeout_probe(w, (unsigned long long)budget_ms * 1000000ull, nullptr);
    if (st != XCCL_OK) return st;
    XCCL_CUDA_CHECK(cudaEventRecord(e1, nullptr));
    XCCL_CUDA_CHECK(cudaEventSynchronize(e1));
    if (elapsed_ms != nullptr) cudaEventElapsedTime(elapsed_ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    HostStatus hs = e->status(0);
    if (status4 != nullptr) {
        status4[0] = hs.code;
        status4[1] = hs.rank;
        status4[2] = hs.peer;
        status4[3] = hs.epoch;
    }
    e->clear_status();
    return hs.code == NVL_TIMEOUT ? XCCL_ERR_TIMED_OUT : XCCL_OK;
}

}  // extern "C"
