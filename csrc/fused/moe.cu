// MoE expert dispatch / combine fused with the all-to-all (extension; the reference only has
// alltoallv call sites: src/team_lib/nccl/xccl_nccl_collective.c:125-163).
//
// dispatch (ONE kernel; one rank alone has its own, without the exchange): count tokens per expert,
//   exchange the counts with every rank through peer memory, turn them into receive offsets, and
//   copy every routed token row straight into its slot of the destination rank's receive buffer -
//   rows arrive grouped by (local expert, source rank), ready for a grouped GEMM. No host round
//   trip, no intermediate permuted copy.
// combine (ONE kernel): every token pulls its top-k expert outputs from the owners' buffers and
//   adds them up with its gate weights in fp32.
// Ranks are real (one process per GPU) or emulated (blockIdx.y = rank in one cooperative launch).
// Waits are bounded; a timeout sets the workspace's error word and the kernel drains.
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "../core/core.h"
#include "../cuda/cuda_common.h"
#include "../tl/nvlink/nvl_device.cuh"
#include "../tl/nvlink/nvl_shm.h"
#include "moe.h"

namespace xccl {
namespace moe {

constexpr int kMaxRanks   = 8;
constexpr int kMaxExperts = 1024;

struct MoeParams {
    int T, H, E, K, tp, rank_base, n_local;
    int cap_rows;
    int seg_packs;                    // 16-byte packs of a row that one warp handles at a time
    unsigned long long budget_ns;
    // per TEAM rank (as mapped here)
    uint32_t      *pad[kMaxRanks];
    uint32_t      *cnt[kMaxRanks];    // [tp][E] tokens of each source rank for each expert of the team
    __nv_bfloat16 *recv[kMaxRanks];   // [cap_rows][H]
    __nv_bfloat16 *yout[kMaxRanks];   // [cap_rows][H] expert outputs, same row numbering
    int32_t       *rsrc[kMaxRanks];   // [cap_rows] source rank * T + token
    // per LOCAL rank
    uint32_t *ctl[kMaxRanks];         // launch control: [0] go word of the offsets, [1] blocks that have finished
    uint32_t *send_base[kMaxRanks];   // [E] first row at the destination for my tokens of expert e
    uint32_t *pos[kMaxRanks];         // [T*K] position among my tokens of the same expert
    uint32_t *slot[kMaxRanks];        // [T*K] row at the destination (kept for combine)
    uint32_t *expert_rows[kMaxRanks]; // [E_local + 1] rows per local expert, total last
    uint32_t *error[kMaxRanks];
    const __nv_bfloat16 *x[kMaxRanks];
    const int32_t       *ids[kMaxRanks];
    const float         *w[kMaxRanks];
    __nv_bfloat16       *out[kMaxRanks];
};

namespace {

// Barrier among the blocks with this index of every rank (flag row `row` of the pads), bounded. All threads call it.
__device__ bool cross_rank_barrier(const MoeParams &p, int rank, int row, uint32_t &epoch)
{
    epoch++;
    __syncthreads();
    int bad = 0;
    if ((int)threadIdx.x < p.tp) {
        const int q = threadIdx.x;
        nvl::st_release_sys(p.pad[q] + (size_t)row * nvl::kMaxRanks + rank, epoch);
        if (!nvl::wait_flag(p.pad[rank] + (size_t)row * nvl::kMaxRanks + q, epoch, p.budget_ns)) bad = 1;
    }
    return __syncthreads_or(bad) == 0;
}

__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(uint32_t *p, uint32_t v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Predicated 16-byte load that bypasses L1 (zeros when !on). A branch around the load instead makes the warp wait for
// each load before it issues the next one.
// kAlone: the memory is this GPU's and nobody writes it during the kernel.
template <bool kAlone> __device__ __forceinline__ uint4 ld16_if(const void *p, bool on)
{
    uint4 v = make_uint4(0, 0, 0, 0);
    if (kAlone) {
        asm volatile(
            "{\n"
            ".reg .pred q;\n"
            "setp.ne.u32 q, %5, 0;\n"
            "@q ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n"
            "}\n"
            : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
            : "l"(p), "r"((uint32_t)on));
        return v;
    }
    asm volatile(
        "{\n"
        ".reg .pred q;\n"
        "setp.ne.u32 q, %5, 0;\n"
        "@q ld.relaxed.sys.global.v4.u32 {%0,%1,%2,%3}, [%4];\n"
        "}\n"
        : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
        : "l"(p), "r"((uint32_t)on)
        : "memory");
    return v;
}

// Go words of the offsets (ctl[0]); 0 between launches. kGoMeet: nothing is copied (a receive buffer is too small, or this
// rank has failed before), but the ranks have met and meet again at the end. kGoSkip: they have not met.
constexpr uint32_t kGoRun = 1, kGoSkip = 2, kGoMeet = 3;

// Block 0 of each rank routes: it counts its entries per expert in shared memory (the atomic's return value is the
// entry's position among its expert's), sends the E counts to every rank, and after one barrier every rank knows the
// whole [tp][E] matrix and derives all offsets itself, so nobody reads a peer's offsets back. The other blocks wait for
// its go word; the block that finishes last holds the closing barrier and clears the words for the next launch. The
// closing barrier follows every opening one that was met, rows or none: a rank that ran ahead into its next dispatch would
// overwrite the counts a peer is still adding up, and the peer, one epoch behind, would take the wrong flags for its own.
// Returns the go word.
// The routing is a serial chain that every row waits for: with the offsets added up by one thread over E loads and
// three grid-wide barriers around it, 128 tokens x 7168, 256 experts, top 8, took 102 us for a 5 us copy.
__device__ uint32_t route_block0(const MoeParams &p, int local, int rank)
{
    __shared__ uint32_t s_cnt[kMaxExperts];
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_first[kMaxRanks + 1];
    const int      EL = p.E / p.tp, nent = p.T * p.K;
    const int32_t *ids = p.ids[local];
    const int      lane = threadIdx.x % 32, wid = threadIdx.x / 32;
    const uint32_t failed = *(volatile uint32_t *)p.error[local];   // by an earlier launch; asked here, where nobody waits for it
    for (int e = threadIdx.x; e < kMaxExperts; e += blockDim.x) s_cnt[e] = 0;
    __syncthreads();
    // eight entries per thread in flight: the ids are the only memory latency of the count
    for (int i0 = threadIdx.x; i0 < nent; i0 += 8 * blockDim.x) {
        int e[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int i = i0 + u * (int)blockDim.x;
            e[u]        = i < nent ? ids[i] : -1;
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if (e[u] >= 0 && e[u] < p.E) p.pos[local][i0 + u * (int)blockDim.x] = atomicAdd(&s_cnt[e[u]], 1u);
        }
    }
    __syncthreads();
    bool     ok    = true;
    uint32_t epoch = 0;
    if (p.tp > 1) {
        epoch = p.pad[rank][nvl::kPadEpochOff];
        for (int j = threadIdx.x; j < p.E * p.tp; j += blockDim.x) {
            const int q = j / p.E, e = j % p.E;
            asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p.cnt[q] + (size_t)rank * p.E + e), "r"(s_cnt[e]) : "memory");
        }
        __threadfence_system();
        ok = cross_rank_barrier(p, rank, 0, epoch);
        if (threadIdx.x == 0) p.pad[rank][nvl::kPadEpochOff] = epoch;
    }
    // thread e: rows of expert e from all ranks, and those of the ranks before mine; kMaxExperts = threads of the block
    const bool met = ok;
    const int  e   = threadIdx.x;
    uint32_t  tot = 0, before = 0;
    if (e < p.E && ok) {
        for (int s = 0; s < p.tp; s++) {
            const uint32_t c = p.tp > 1 ? nvl::ld_relaxed_sys(p.cnt[rank] + (size_t)s * p.E + e) : s_cnt[e];
            tot += c;
            if (s < rank) before += c;
        }
    }
    uint32_t incl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        uint32_t v = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        s_warp[lane] = v;
    }
    __syncthreads();
    const uint32_t excl = incl - tot + (wid > 0 ? s_warp[wid - 1] : 0);   // rows of all experts before e
    if (e < p.E && e % EL == 0) s_first[e / EL] = excl;
    if (e == p.E - 1) s_first[p.tp] = excl + tot;
    __syncthreads();
    // every rank sees every receive buffer's fill: when one is too small, nobody writes
    for (int d = 0; d < p.tp && ok; d++) {
        if (s_first[d + 1] - s_first[d] > (uint32_t)p.cap_rows) {
            if (threadIdx.x == 0) atomicExch(p.error[local], 0x400u);
            ok = false;
        }
    }
    if (e < p.E && met) {
        p.send_base[local][e] = excl - s_first[e / EL] + before;
        if (e / EL == rank) p.expert_rows[local][e % EL] = tot;
    }
    if (threadIdx.x == 0) {
        if (met) p.expert_rows[local][EL] = s_first[rank + 1] - s_first[rank];
        else atomicExch(p.error[local], 0x401u);
    }
    __threadfence();
    __syncthreads();
    return !met ? kGoSkip : ok && failed == 0 ? kGoRun : kGoMeet;
}

__global__ void __launch_bounds__(kMaxExperts, 1) moe_dispatch_kernel(MoeParams p)
{
    const int      local = blockIdx.y, rank = p.rank_base + local;
    const int      EL    = p.E / p.tp;
    const int32_t *ids   = p.ids[local];
    uint32_t      *ctl   = p.ctl[local];
    __shared__ uint32_t s_go;

    if (blockIdx.x == 0) {
        const uint32_t go = route_block0(p, local, rank);
        if (threadIdx.x == 0) {
            s_go = go;
            st_release_gpu(ctl, go);
        }
    } else if (threadIdx.x == 0) {
        const unsigned long long t0 = nvl::global_ns();
        uint32_t                 go;
        // block 0 itself waits up to one budget for its peers
        while ((go = ld_acquire_gpu(ctl)) == 0 && nvl::global_ns() - t0 < 2 * p.budget_ns) {}
        if (go == 0) {
            atomicCAS(p.error[local], 0u, 0x405u);
            go = kGoSkip;
        }
        s_go = go;
    }
    __syncthreads();
    // every row goes straight to its slots at the owners. A warp takes seg_packs packs of a token's row, reads them
    // once and stores them to all K destinations, four packs per lane in flight: the stores (K x the input) are what
    // the copy is bound by. 4096 x 7168 tokens, top 8, 470 MB of stores: 355 us with a warp per (token, expert) that
    // waited for each load before its store.
    if (s_go == kGoRun) {
        const int    lane = threadIdx.x % 32;
        const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 32, nwarps = (size_t)gridDim.x * blockDim.x / 32;
        const int    packs = p.H * 2 / 16, nseg = (packs + p.seg_packs - 1) / p.seg_packs;
        const size_t items = (size_t)p.T * nseg;
        for (size_t it = warp; it < items; it += nwarps) {
            const int    t  = (int)(it / nseg), seg = (int)(it % nseg);
            const int    lo = seg * p.seg_packs, hi = min(lo + p.seg_packs, packs);
            const uint4 *src = reinterpret_cast<const uint4 *>(p.x[local] + (size_t)t * p.H);
            for (int kb = 0; kb < p.K; kb += 32) {
                // lane k: where the token's entry kb + k goes
                const int          kn  = min(32, p.K - kb);
                unsigned long long my  = 0;
                if (lane < kn) {
                    const size_t i = (size_t)t * p.K + kb + lane;
                    const int    e = ids[i];
                    if (e >= 0 && e < p.E) {
                        const int      d   = e / EL;
                        const uint32_t row = __ldcg(p.send_base[local] + e) + __ldcg(p.pos[local] + i);
                        my = (unsigned long long)(p.recv[d] + (size_t)row * p.H);
                        if (seg == 0) {
                            p.slot[local][i] = row;
                            p.rsrc[d][row]   = rank * p.T + t;
                        }
                    }
                }
                for (int b0 = lo; b0 < hi; b0 += 128) {
                    const int k0 = b0 + lane;
                    uint4     v[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        if (k0 + 32 * u < hi) v[u] = __ldg(src + k0 + 32 * u);
                    }
                    for (int k = 0; k < kn; k++) {
                        uint4 *dst = reinterpret_cast<uint4 *>(__shfl_sync(0xffffffffu, my, k));
                        if (dst == nullptr) continue;
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            if (k0 + 32 * u < hi) nvl::st_16(dst + k0 + 32 * u, v[u]);
                        }
                    }
                }
            }
        }
    }
    __threadfence_system();
    __syncthreads();
    __shared__ int s_last;
    if (threadIdx.x == 0) {
        s_last = atomicAdd(ctl + 1, 1u) == gridDim.x - 1;
        // block 0's word, also where this block gave up waiting for it (one rank alone has no barrier to decide on)
        if (s_last != 0 && p.tp > 1) s_go = *(volatile uint32_t *)ctl;
    }
    __syncthreads();
    if (s_last == 0) return;
    // the last block of this rank: everything has landed everywhere before anyone returns
    __threadfence_system();
    if (threadIdx.x == 0) ctl[0] = ctl[1] = 0;
    if (s_go != kGoSkip && p.tp > 1) {
        uint32_t epoch = *(volatile uint32_t *)(p.pad[rank] + nvl::kPadEpochOff);
        bool     ok    = cross_rank_barrier(p, rank, 0, epoch);
        if (threadIdx.x == 0) {
            p.pad[rank][nvl::kPadEpochOff] = epoch;
            if (!ok) atomicExch(p.error[local], 0x402u);
        }
    }
}

// Exclusive prefix sum over the threads of a block of kMaxExperts; every thread calls it. *total: the sum of all.
__device__ uint32_t block_prefix(uint32_t v, uint32_t *total)
{
    __shared__ uint32_t s_warp[32];
    const int lane = threadIdx.x % 32, wid = threadIdx.x / 32;
    uint32_t  incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    uint32_t w = s_warp[lane];   // every warp adds the warps' sums up for itself
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += u;
    }
    *total = __shfl_sync(0xffffffffu, w, 31);
    const uint32_t before = __shfl_sync(0xffffffffu, w, wid > 0 ? wid - 1 : 0);
    return incl - v + (wid > 0 ? before : 0);
}

// Dispatch of one rank alone. Every block routes for itself: it counts all entries per expert, those before its own tokens
// apart, so that the first row of its entries of expert e is the prefix sum over the experts plus the entries of e before it.
// No block waits for another (and the launch need not be cooperative); what every block reads besides its rows are the T x K
// ids, from L2. Blocks own whole tokens; where there are fewer tokens than blocks, `parts` blocks share a token's row and
// each derives the same rows for its entries. The first rows of x are on their way while the block counts.
// One block that routed for all while the others waited: 128 tokens x 7168, 256 experts, top 8, 16.5 us, now 7.7; 16 tokens x
// 2048 13.0 and 5.1; 4096 x 7168 (bound by 470 MB of stores) 112 and 104. With several ranks the counts have to be exchanged
// anyway, and one block does it (moe_dispatch_kernel).
constexpr int kOwnEntries = 1024;   // entries that a block routes at a time (callers: K <= kOwnEntries)

__global__ void __launch_bounds__(kMaxExperts, 1) moe_dispatch_alone_kernel(MoeParams p)
{
    __shared__ uint32_t s_before[kMaxExperts], s_rest[kMaxExperts], s_row[kOwnEntries];
    __shared__ int32_t  s_id[kOwnEntries];
    const int      tid = threadIdx.x, lane = tid % 32, wid = tid / 32, nwarps = kMaxExperts / 32;
    const int32_t *ids = p.ids[0];
    const int      nent = p.T * p.K, blocks = gridDim.x;
    const int      parts = max(1, blocks / p.T);
    const int      part  = blocks >= p.T ? (int)blockIdx.x % parts : 0;
    const int      t_lo  = blocks >= p.T ? min((int)blockIdx.x / parts, p.T) : (int)((long long)blockIdx.x * p.T / blocks);
    const int      t_hi  = blocks >= p.T ? min(t_lo + 1, p.T) : (int)((long long)(blockIdx.x + 1) * p.T / blocks);
    const uint32_t failed = *(volatile uint32_t *)p.error[0];   // by an earlier launch
    // a warp takes seg_packs packs of a token's row at a time
    const int      packs = p.H * 2 / 16, nseg = (packs + p.seg_packs - 1) / p.seg_packs;
    const int      seg_lo = nseg * part / parts, segs = nseg * (part + 1) / parts - seg_lo;
    auto load = [&](int t0, int it, uint4 (&v)[4]) {
        const int    lo  = (seg_lo + it % segs) * p.seg_packs + lane, hi = min((seg_lo + it % segs + 1) * p.seg_packs, packs);
        const uint4 *src = reinterpret_cast<const uint4 *>(p.x[0] + (size_t)(t0 + it / segs) * p.H);
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (lo + 32 * u < hi) v[u] = __ldg(src + lo + 32 * u);
        }
    };
    const int batch = max(1, kOwnEntries / p.K);   // tokens that are routed at a time
    uint4     v[4];
    if (wid < segs * min(batch, t_hi - t_lo)) load(t_lo, wid, v);

    s_before[tid] = s_rest[tid] = 0;
    __syncthreads();
    // eight entries per thread in flight
    for (int i0 = tid; i0 < nent; i0 += 8 * kMaxExperts) {
        int e[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int i = i0 + u * kMaxExperts;
            e[u]        = i < nent ? __ldg(ids + i) : -1;
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if (e[u] >= 0 && e[u] < p.E) atomicAdd((i0 + u * kMaxExperts < t_lo * p.K ? s_before : s_rest) + e[u], 1u);
        }
    }
    __syncthreads();
    const uint32_t before = s_before[tid], tot = before + s_rest[tid];
    uint32_t       total;
    const uint32_t first = block_prefix(tot, &total);
    s_before[tid]        = first + before;   // the row of my next entry of expert tid
    if (blockIdx.x == 0) {
        if (tid < p.E) p.expert_rows[0][tid] = tot;
        if (tid == 0) p.expert_rows[0][p.E] = total;
        if (tid == 0 && total > (uint32_t)p.cap_rows) atomicExch(p.error[0], 0x400u);
    }
    if (total > (uint32_t)p.cap_rows || failed != 0) return;   // the same in every block: nobody writes
    for (int t0 = t_lo; t0 < t_hi; t0 += batch) {
        const int nt = min(batch, t_hi - t0), n = nt * p.K;
        __syncthreads();
        if (tid < n) s_id[tid] = __ldg(ids + (size_t)t0 * p.K + tid);
        __syncthreads();
        if (tid < n) {
            const int32_t e   = s_id[tid];
            uint32_t      row = 0xffffffffu;
            if (e >= 0 && e < p.E) {
                if (parts > 1) {   // one token: its earlier entries of the same expert, alike in every block
                    row = s_before[e];
                    for (int k = 0; k < tid; k++) row += s_id[k] == e;
                } else {
                    row = atomicAdd(s_before + e, 1u);
                }
                if (part == 0) {
                    p.slot[0][(size_t)t0 * p.K + tid] = row;
                    p.rsrc[0][row]                    = t0 + tid / p.K;
                }
            }
            s_row[tid] = row;
        }
        __syncthreads();
        for (int it = wid; it < nt * segs; it += nwarps) {
            const int lo = (seg_lo + it % segs) * p.seg_packs + lane, hi = min((seg_lo + it % segs + 1) * p.seg_packs, packs);
            const uint32_t *rows = s_row + it / segs * p.K;
            uint4           next[4];
            const int       nit = it + nwarps;
            if (nit < nt * segs) load(t0, nit, next);
            else if (t0 + batch < t_hi && wid < segs * min(batch, t_hi - t0 - batch)) load(t0 + batch, wid, next);
            for (int k = 0; k < p.K; k++) {
                const uint32_t row = rows[k];
                if (row == 0xffffffffu) continue;
                uint4 *dst = reinterpret_cast<uint4 *>(p.recv[0] + (size_t)row * p.H) + lo;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    if (lo + 32 * u < hi) dst[32 * u] = v[u];
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = next[u];
        }
        // (a warp without an item in this batch has no load of the next one's on its way yet)
        if (wid >= nt * segs && t0 + batch < t_hi && wid < segs * min(batch, t_hi - t0 - batch)) load(t0 + batch, wid, v);
    }
}

// Block b meets block b of every rank before its first load (the peers' expert outputs are complete) and after its last
// one (nobody's buffer is reused while a peer may still read it); the launch ends when all blocks have. One rank alone
// has nobody to meet.
template <bool kAlone> __global__ void __launch_bounds__(1024, 1) moe_combine_kernel(MoeParams p)
{
    const int local = blockIdx.y, rank = p.rank_base + local;
    const int EL    = p.E / p.tp;
    uint32_t  epoch = 0;
    bool      ok    = true;
    if (p.tp > 1) {
        epoch = p.pad[rank][nvl::kPadEpochOff + blockIdx.x];
        ok    = cross_rank_barrier(p, rank, blockIdx.x, epoch);
        if (!ok && threadIdx.x == 0) atomicExch(p.error[local], 0x403u);
    }
    // a warp adds up seg_packs packs of one token: lane k holds routing entry k, the warp shares the rows' addresses, and all
    // (up to eight) expert rows of a pack are in flight at once. 4096 x 7168, top 8 (530 MB): 244 us with a warp per whole
    // token and a branch per load, which made the eight loads wait for one another. One rank alone loads the entries of a warp's
    // next piece beside the rows of this one and reads without system scope and past L1: 104 us, now 97 (the last costs where the
    // same rows are read from L2 again and again, 512 x 4096 9.6 and 12.6 us, and nothing behind the kernel that writes them). With
    // several ranks the early entries only spill: 2048 x 4096, top 4, two ranks 43.6 us, so 45.2, 1024 x 2048, top 10, 27.3 and 29.2.
    const int    lane = threadIdx.x % 32;
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 32, nwarps = (size_t)gridDim.x * blockDim.x / 32;
    const int    packs = p.H * 2 / 16, nseg = (packs + p.seg_packs - 1) / p.seg_packs;
    const size_t items = ok ? (size_t)p.T * nseg : 0;
    // entry kb + lane of a token (lanes 0-7): expert (-1: none), gate, row
    auto entry = [&](size_t t, int kb, int &e, float &g, uint32_t &row) {
        e   = -1;
        g   = 0.0f;
        row = 0;
        if (lane < min(8, p.K - kb)) {
            const size_t i = t * p.K + kb + lane;
            e   = __ldg(p.ids[local] + i);
            g   = __ldg(p.w[local] + i);
            row = __ldg(p.slot[local] + i);
        }
    };
    const uint32_t failed = *(volatile uint32_t *)p.error[local];
    int      e_next = -1;
    float    g_next = 0.0f;
    uint32_t r_next = 0;
    if (kAlone && warp < items) entry(warp / nseg, 0, e_next, g_next, r_next);
    for (size_t it = warp; it < items && failed == 0; it += nwarps) {
        const size_t t  = it / nseg;
        const int    lo = (int)(it % nseg) * p.seg_packs, hi = min(lo + p.seg_packs, packs);
        // (with more than eight entries the running sum passes through bf16 between groups)
        for (int kb = 0; kb < p.K; kb += 8) {
            if (!kAlone) entry(t, kb, e_next, g_next, r_next);
            const bool     on     = e_next >= 0 && e_next < p.E;
            const float    my_g   = on ? g_next : 0.0f;
            const unsigned long long my_row = on ? (unsigned long long)(p.yout[kAlone ? 0 : e_next / EL] + (size_t)r_next * p.H) : 0ull;
            if (kAlone && kb + 8 < p.K) entry(t, kb + 8, e_next, g_next, r_next);
            else if (kAlone && it + nwarps < items) entry((it + nwarps) / nseg, 0, e_next, g_next, r_next);
            const uint4 *rows[8];
            float        gs[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                rows[k] = reinterpret_cast<const uint4 *>(__shfl_sync(0xffffffffu, my_row, k));
                gs[k]   = __shfl_sync(0xffffffffu, my_g, k);
            }
            for (int k0 = lo + lane; k0 < hi; k0 += 32) {
                uint4 raw[8];
#pragma unroll
                for (int k = 0; k < 8; k++) raw[k] = ld16_if<kAlone>(rows[k] + k0, rows[k] != nullptr);
                float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                uint4 *dst = reinterpret_cast<uint4 *>(p.out[local] + t * p.H) + k0;
                if (kb > 0) {
                    const uint4 prev = *dst;
                    const __nv_bfloat162 *ph = reinterpret_cast<const __nv_bfloat162 *>(&prev);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        float2 f = __bfloat1622float2(ph[j]);
                        acc[2 * j] = f.x;
                        acc[2 * j + 1] = f.y;
                    }
                }
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw[k]);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        float2 f = __bfloat1622float2(h[j]);
                        acc[2 * j] += gs[k] * f.x;
                        acc[2 * j + 1] += gs[k] * f.y;
                    }
                }
                uint4 o;
                __nv_bfloat162 *oh = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
                for (int j = 0; j < 4; j++) oh[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
                *dst = o;
            }
        }
    }
    if (p.tp > 1) {
        const bool done = ok && cross_rank_barrier(p, rank, blockIdx.x, epoch);
        if (threadIdx.x == 0) {
            p.pad[rank][nvl::kPadEpochOff + blockIdx.x] = epoch;
            if (ok && !done) atomicExch(p.error[local], 0x404u);
        }
    }
}

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

}  // namespace

struct MoeWorkspace {
    MoeParams             p{};
    bool                  emulated = false;
    nvl::SymmetricRegion *region   = nullptr;
    std::vector<void *>   allocs;
    char                 *sym[kMaxRanks] = {nullptr};
    size_t                off_cnt = 0, off_rsrc = 0, off_recv = 0, off_yout = 0, total = 0;
    int                   blocks = 0;   // per local rank: one per SM, all of them resident
};

}  // namespace moe
}  // namespace xccl

using namespace xccl;
using namespace xccl::moe;

extern "C" {

xccl_status_t xccl_moe_ws_create(const xccl_oob_collectives_t *oob, int emu_ranks, int T, int H, int E, int K,
                                 int cap_rows, xccl_moe_ws_h *out)
{
    if (out == nullptr || T <= 0 || H <= 0 || (H * 2) % 16 != 0 || E <= 0 || E > kMaxExperts || K <= 0) return XCCL_ERR_INVALID_PARAM;
    if (!cuda_available()) return XCCL_ERR_NO_RESOURCE;
    auto *w      = new MoeWorkspace;
    MoeParams &p = w->p;
    p.T = T; p.H = H; p.E = E; p.K = K;
    p.budget_ns = 4000000000ull;
    w->emulated = (oob == nullptr);
    p.tp        = w->emulated ? std::max(emu_ranks, 1) : oob->size;
    p.n_local   = w->emulated ? p.tp : 1;
    p.rank_base = w->emulated ? 0 : oob->rank;
    if (p.tp > kMaxRanks || E % p.tp != 0) {
        delete w;
        return XCCL_ERR_INVALID_PARAM;
    }
    const int EL = E / p.tp;
    p.cap_rows   = cap_rows > 0 ? cap_rows : p.tp * T * K;
    w->off_cnt   = align_up(nvl::kPadBytes, 4096);
    w->off_rsrc  = align_up(w->off_cnt + (size_t)p.tp * E * 4, 4096);
    w->off_recv  = align_up(w->off_rsrc + (size_t)p.cap_rows * 4, 4096);
    w->off_yout  = align_up(w->off_recv + (size_t)p.cap_rows * H * 2, 4096);
    w->total     = align_up(w->off_yout + (size_t)p.cap_rows * H * 2, 4096);
    xccl_status_t st = XCCL_OK;
    if (w->emulated) {
        for (int r = 0; r < p.tp && st == XCCL_OK; r++) {
            void *q = nullptr;
            if (cudaMalloc(&q, w->total) != cudaSuccess) {
                (void)cudaGetLastError();
                st = XCCL_ERR_NO_MEMORY;
                break;
            }
            w->allocs.push_back(q);
            cudaMemset(q, 0, w->off_recv);
            w->sym[r] = (char *)q;
        }
    } else {
        OobGroup g;
        g.oob = *oob; g.range.type = XCCL_EP_RANGE_UNDEFINED; g.rank = oob->rank; g.size = oob->size;
        st = nvl::SymmetricRegion::create(g, w->total, false, &w->region);
        if (st == XCCL_OK) {
            for (int r = 0; r < p.tp; r++) w->sym[r] = w->region->base[(size_t)r];
        }
    }
    for (int r = 0; r < p.tp && st == XCCL_OK; r++) {
        p.pad[r]  = (uint32_t *)w->sym[r];
        p.cnt[r]  = (uint32_t *)(w->sym[r] + w->off_cnt);
        p.rsrc[r] = (int32_t *)(w->sym[r] + w->off_rsrc);
        p.recv[r] = (__nv_bfloat16 *)(w->sym[r] + w->off_recv);
        p.yout[r] = (__nv_bfloat16 *)(w->sym[r] + w->off_yout);
    }
    auto dev_alloc = [&](size_t bytes) -> void * {
        void *q = nullptr;
        if (cudaMalloc(&q, bytes) != cudaSuccess) {
            st = XCCL_ERR_NO_MEMORY;
            return nullptr;
        }
        cudaMemset(q, 0, bytes);
        w->allocs.push_back(q);
        return q;
    };
    for (int l = 0; l < p.n_local && st == XCCL_OK; l++) {
        p.ctl[l]         = (uint32_t *)dev_alloc(8);
        p.send_base[l]   = (uint32_t *)dev_alloc((size_t)E * 4);
        p.pos[l]         = (uint32_t *)dev_alloc((size_t)T * K * 4);
        p.slot[l]        = (uint32_t *)dev_alloc((size_t)T * K * 4);
        p.expert_rows[l] = (uint32_t *)dev_alloc((size_t)(EL + 1) * 4);
        p.error[l]       = (uint32_t *)dev_alloc(4);
    }
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    w->blocks = std::max(1, sms / p.n_local);
    // Packs of a row per warp: as long as possible (the routing entries are read once per piece) while every warp of the
    // grid still gets a few pieces; a batch of 128 tokens is cut into pieces of 512 bytes.
    const size_t packs = (size_t)H * 2 / 16, warps = (size_t)w->blocks * (kMaxExperts / 32);
    p.seg_packs = 32;
    while (p.seg_packs < 128 && (size_t)T * ((packs + 2 * p.seg_packs - 1) / (2 * p.seg_packs)) >= 4 * warps) p.seg_packs *= 2;
    cudaDeviceSynchronize();
    if (st != XCCL_OK) {
        xccl_moe_ws_destroy(w);
        return st;
    }
    *out = w;
    return XCCL_OK;
}

void xccl_moe_ws_destroy(xccl_moe_ws_h w)
{
    if (w == nullptr) return;
    cudaDeviceSynchronize();
    for (void *q : w->allocs) cudaFree(q);
    delete w->region;
    delete w;
}

// Blocks of one launch wait on one another (dispatch: for block 0; with several ranks: for the peers), hence cooperative.
// The combine of one rank alone has no waits and starts without that.
static xccl_status_t launch(void (*kernel)(MoeParams), MoeWorkspace *w, int blocks, bool cooperative, cudaStream_t s)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim  = dim3((unsigned)blocks, (unsigned)w->p.n_local);
    cfg.blockDim = dim3(kMaxExperts);
    cfg.stream   = s;
    cudaLaunchAttribute attr[1];
    attr[0].id              = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = cooperative ? 1 : 0;
    cfg.attrs               = attr;
    cfg.numAttrs            = 1;
    XCCL_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, w->p));
    return XCCL_OK;
}

xccl_status_t xccl_moe_dispatch(xccl_moe_ws_h w, const void *const *x, const int32_t *const *ids, void *stream)
{
    if (w == nullptr || x == nullptr || ids == nullptr) return XCCL_ERR_INVALID_PARAM;
    for (int l = 0; l < w->p.n_local; l++) {
        w->p.x[l]   = (const __nv_bfloat16 *)x[l];
        w->p.ids[l] = ids[l];
    }
    if (w->p.tp == 1 && w->p.K <= kOwnEntries) return launch(moe_dispatch_alone_kernel, w, w->blocks, false, (cudaStream_t)stream);
    return launch(moe_dispatch_kernel, w, w->blocks, true, (cudaStream_t)stream);
}

xccl_status_t xccl_moe_combine(xccl_moe_ws_h w, const int32_t *const *ids, const float *const *weights, void *const *out,
                               void *stream)
{
    if (w == nullptr || ids == nullptr || weights == nullptr || out == nullptr) return XCCL_ERR_INVALID_PARAM;
    for (int l = 0; l < w->p.n_local; l++) {
        w->p.ids[l] = ids[l];
        w->p.w[l]   = weights[l];
        w->p.out[l] = (__nv_bfloat16 *)out[l];
    }
    // several ranks: a row of barrier flags per block
    const int blocks = w->p.tp > 1 ? std::min(w->blocks, nvl::kMaxBlocks) : w->blocks;
    return launch(w->p.tp > 1 ? moe_combine_kernel<false> : moe_combine_kernel<true>, w, blocks, w->p.tp > 1, (cudaStream_t)stream);
}

void *xccl_moe_ws_buffer(xccl_moe_ws_h w, int local_rank, int which)
{
    if (w == nullptr || local_rank < 0 || local_rank >= w->p.n_local) return nullptr;
    const int r = w->p.rank_base + local_rank;
    switch (which) {
    case XCCL_MOE_BUF_RECV: return w->p.recv[r];
    case XCCL_MOE_BUF_EXPERT_OUT: return w->p.yout[r];
    case XCCL_MOE_BUF_EXPERT_ROWS: return w->p.expert_rows[local_rank];
    case XCCL_MOE_BUF_ROW_SOURCE: return w->p.rsrc[r];
    default: return nullptr;
    }
}

int xccl_moe_ws_cap_rows(xccl_moe_ws_h w) { return w != nullptr ? w->p.cap_rows : 0; }

uint32_t xccl_moe_ws_error(xccl_moe_ws_h w)
{
    if (w == nullptr) return 0xffffffffu;
    uint32_t worst = 0;
    for (int l = 0; l < w->p.n_local; l++) {
        uint32_t v = 0;
        cudaMemcpy(&v, w->p.error[l], 4, cudaMemcpyDeviceToHost);
        if (v != 0) worst = v;
    }
    return worst;
}

// Barriers that a local rank has held on flag row 0 (dispatch: two, also when it copies nothing; combine: two of its
// block 0), for tests. Synchronises.
uint32_t xccl_moe_ws_meetings(xccl_moe_ws_h w, int local_rank)
{
    uint32_t v = 0;
    if (w == nullptr || local_rank < 0 || local_rank >= w->p.n_local) return 0xffffffffu;
    cudaMemcpy(&v, w->p.pad[w->p.rank_base + local_rank] + nvl::kPadEpochOff, 4, cudaMemcpyDeviceToHost);
    return v;
}

}  // extern "C"
