// Host side of the fused tensor-parallel MLP operations: owns the symmetric buffers the
// allgather->GEMM and GEMM->reduce-scatter kernels communicate through, builds the TMA
// descriptors and launches tp_gemm_kernel in the matching mode.
//
// Buffers per rank (all in one symmetric region, or plain device memory when emulated):
//   pad    signal pad: barrier flags for the copy CTAs, arrival counters for reduce-scatter
//   xg     [M, K]  gathered activations; rows [r*M/tp, (r+1)*M/tp) are rank r's own shard and are
//          the only rows other ranks ever read
//   part   [2][tp][M/tp][N_rs]  partial output tiles written by every rank, two parities
#include <cuda_fp8.h>

#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "../core/core.h"
#include "../cuda/cuda_common.h"
#include "../tl/nvlink/nvl_shm.h"
#include "tp_gemm.cuh"
#include "tp_mlp.h"
#include "tp_skinny.cuh"

namespace xccl {
namespace tp {

struct TpWorkspace {
    int  tp = 1, n_local = 1, rank_base = 0;
    int  M = 0, K = 0, N_rs = 0;
    bool emulated = false;
    nvl::SymmetricRegion *region = nullptr;
    std::vector<void *>   allocs;     // emulated buffers
    char     *base[kMaxTpRanks]  = {nullptr};  // per TEAM rank: start of that rank's buffers as mapped here
    uint32_t *ready[kMaxTpRanks] = {nullptr};  // per LOCAL rank
    uint32_t *error = nullptr;
    size_t    off_xg = 0, off_part = 0, total = 0;
    uint32_t  seq_ag = 0, seq_rs = 0, rs_count[2] = {0, 0};
    bool      copy_ctas_auto = true;
    int       copy_ctas = 0;      // CTAs of the allgather->GEMM kernel that pull the remote shards; 0 = by team size
    int       copy_mode = 1;      // 1: copier warps in every CTA, 0: whole copy CTAs
    bool      rs_debug_local = false;
    bool      rs_fused  = true;   // XCCL_TP_RS_FUSED=0: separate reduce phase after the last tile
    // input rows arriving from the host while the allgather->GEMM kernel already runs
    uint32_t   *in_flags[kMaxTpRanks] = {nullptr};  // per LOCAL rank: one word per chunk of in_rows rows
    uint32_t    in_seq = 0;
    bool        in_active = false;
    int         in_ramp   = 0;      // 1: walk the local rows in growing groups (the kernel starts before the rows are there); 2: phases over all shards
    int         in_rows = 256;
    cudaEvent_t in_consumed = nullptr;

    uint32_t      *pad(int r) const { return (uint32_t *)base[r]; }
    __nv_bfloat16 *xg(int r) const { return (__nv_bfloat16 *)(base[r] + off_xg); }
    __nv_bfloat16 *part(int r) const { return (__nv_bfloat16 *)(base[r] + off_part); }
    // fp8 view of the gathered buffer: [M, K] e4m3 rows, then their [M, K/128] fp32 scales
    float *sx(int r) const { return (float *)(base[r] + off_xg + (size_t)M * K); }
};

namespace {

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Block of 128 columns b of the matrix (rows are contiguous and K is a multiple of 128, so blocks and their scales are
// simply numbered through): amax by shuffles, one scale, e4m3 bytes. kV values per lane, 128 / kV lanes per block, eight
// blocks per warp with their loads all in flight. What it costs is the traffic (3 bytes per value); with one block per
// warp, 8-byte loads and nothing in flight beside them 4096 x 8192 (100 MB) took 43.8 us, now 20.3 us.
// kV = 8 needs 16-byte aligned input and 8-byte aligned output, kV = 4 half of that.
template <int kV> __global__ void __launch_bounds__(256) quantize_rows_1x128_kernel(const __nv_bfloat16 *x, size_t blocks,
                                                                                  uint8_t *out, float *scales)
{
    constexpr int kLanes = 128 / kV, kPer = 32 / kLanes, kU = 8 / kPer;  // lanes per block, blocks per warp at a time, times
    const size_t  warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int     lane = threadIdx.x % 32, l = lane % kLanes;
    const size_t  b0   = warp * 8 + lane / kLanes;
    using Raw = typename std::conditional<kV == 8, uint4, uint2>::type;
    Raw raw[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
        // (a warp past the end repeats the last block and stores nothing)
        const size_t b = min(b0 + (size_t)u * kPer, blocks - 1);
        raw[u] = __ldg(reinterpret_cast<const Raw *>(x + b * 128 + l * kV));
    }
#pragma unroll
    for (int u = 0; u < kU; u++) {
        const size_t          b = b0 + (size_t)u * kPer;
        const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw[u]);
        float2 v[kV / 2];
        float  amax = 0.0f;
#pragma unroll
        for (int e = 0; e < kV / 2; e++) {
            v[e] = __bfloat1622float2(h[e]);
            amax = fmaxf(amax, fmaxf(fabsf(v[e].x), fabsf(v[e].y)));
        }
#pragma unroll
        for (int o = kLanes / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        const float s = fmaxf(amax, 1e-12f) / 448.0f, inv = 1.0f / s;
        uint32_t q[kV / 4];
#pragma unroll
        for (int e = 0; e < kV / 4; e++) {
            q[e] = (uint32_t)__nv_cvt_float_to_fp8(v[2 * e].x * inv, __NV_SATFINITE, __NV_E4M3) |
                   ((uint32_t)__nv_cvt_float_to_fp8(v[2 * e].y * inv, __NV_SATFINITE, __NV_E4M3) << 8) |
                   ((uint32_t)__nv_cvt_float_to_fp8(v[2 * e + 1].x * inv, __NV_SATFINITE, __NV_E4M3) << 16) |
                   ((uint32_t)__nv_cvt_float_to_fp8(v[2 * e + 1].y * inv, __NV_SATFINITE, __NV_E4M3) << 24);
        }
        if (b < blocks) {
            if (kV == 8) {
                *reinterpret_cast<uint2 *>(out + b * 128 + l * kV) = make_uint2(q[0], q[kV / 4 - 1]);
            } else {
                *reinterpret_cast<uint32_t *>(out + b * 128 + l * kV) = q[0];
            }
            if (l == 0) scales[b] = s;
        }
    }
}

// CTAs per rank that pull the remote shards (copy mode 0): `want`, or with `emulated_auto` fewer where that pays. Emulated
// ranks share one GPU's SMs (37 CTAs per rank with four) and copy inside its memory, and what the copy has to keep up with is
// the tile walk, whose time per byte of A grows with the columns of B. Four ranks, 2048 x 4096 x 14336 (7168 columns per
// rank), block step with 10 / 6 / 4 / 2 copy CTAs: 689 / 658 / 645 / 790 us, fp8 723 / 654 / 629 / 631; 1024 x 2048 x 4096 (2048
// columns): 142 / 151 / 161 / 209. Shards of a single 128-row block want the shard sooner than the walk of one block covers:
// three ranks, 384 x 4096 x 14208, 12 / 6 / 4 copy CTAs 243 / 257 / 260 us, fp8 190 / 202 / 204; there all copy that may.
// (3, 4 and 8 ranks, 134 sizes, against 16 everywhere: 1 to 2 % less with 256 rows and more per shard, up to 11 %.)
int copy_ctas(int tp, int copy_mode, int want, bool emulated_auto, int shard_rows, int columns, int ctas)
{
    if (tp <= 1 || copy_mode != 0) return 0;
    if (emulated_auto && shard_rows >= 2 * kBM) want = std::min(want, std::max(2, (28672 + columns - 1) / columns));
    return std::max(1, std::min(want, ctas / 4));
}
int copy_ctas_of(const TpWorkspace *w, int columns, int ctas)
{
    return copy_ctas(w->tp, w->copy_mode, w->copy_ctas, w->emulated && w->copy_ctas_auto, w->M / w->tp, columns, ctas);
}

void layout(TpWorkspace *w)
{
    w->off_xg   = align_up(nvl::kPadBytes, 4096);
    w->off_part = align_up(w->off_xg + (size_t)w->M * w->K * 2, 4096);
    w->total    = align_up(w->off_part + (size_t)2 * w->M * w->N_rs * 2, 4096);
}

}  // namespace

}  // namespace tp
}  // namespace xccl

using namespace xccl;
using namespace xccl::tp;

extern "C" {

xccl_status_t xccl_tp_ws_create(const xccl_oob_collectives_t *oob, int emu_ranks, int M, int K, int N_rs,
                                xccl_tp_ws_h *out)
{
    if (out == nullptr || M <= 0 || K <= 0 || N_rs <= 0) return XCCL_ERR_INVALID_PARAM;
    if (!cuda_available()) return XCCL_ERR_NO_RESOURCE;
    auto *w = new TpWorkspace;
    w->M = M;
    w->K = K;
    w->N_rs = N_rs;
    w->copy_ctas = (int)tp_options().num("COPY_CTAS");
    w->copy_mode = (int)tp_options().num("COPY_MODE");
    w->rs_debug_local = tp_options().flag("RS_DEBUG_LOCAL");
    w->rs_fused  = tp_options().flag("RS_FUSED");
    w->in_rows   = std::max(1, (int)tp_options().num("H2D_CHUNK_ROWS"));
    layout(w);
    xccl_status_t st = XCCL_OK;
    if (oob == nullptr) {
        w->emulated  = true;
        w->tp        = std::max(emu_ranks, 1);
        w->n_local   = w->tp;
        w->rank_base = 0;
        if (w->tp > kMaxTpRanks) st = XCCL_ERR_INVALID_PARAM;
        for (int r = 0; r < w->tp && st == XCCL_OK; r++) {
            void *p = nullptr;
            if (cudaMalloc(&p, w->total) != cudaSuccess) {
                (void)cudaGetLastError();
                st = XCCL_ERR_NO_MEMORY;
                break;
            }
            w->allocs.push_back(p);
            cudaMemset(p, 0, nvl::kPadBytes);
            w->base[r] = (char *)p;
        }
    } else {
        w->tp        = oob->size;
        w->n_local   = 1;
        w->rank_base = oob->rank;
        if (w->tp > kMaxTpRanks) {
            st = XCCL_ERR_INVALID_PARAM;
        } else {
            OobGroup g;
            g.oob        = *oob;
            g.range.type = XCCL_EP_RANGE_UNDEFINED;
            g.rank       = oob->rank;
            g.size       = oob->size;
            st           = nvl::SymmetricRegion::create(g, w->total, false, &w->region);
            if (st == XCCL_OK) {
                for (int r = 0; r < w->tp; r++) w->base[r] = w->region->base[(size_t)r];
            }
        }
    }
    // Copy mode 0 (whole copy CTAs, bulk copies through shared memory): one SM pulls only 16-20 GB/s over NVLink
    // (measured on 8 GPUs: 4 copy CTAs 1.52 ms, 8: 0.92 ms, 16: 0.76 ms for the 8192 x 7168 x 8192 projection whose MMAs
    // take 0.68 ms), so 16 of them are needed to stay ahead of the tile walk, and each costs tensor throughput.
    // Copy mode 1 (copier warps in every CTA, plain loads) costs no tensor throughput but moves only about
    // 120 GB/s per GPU however many loads it keeps in flight (8 GPUs: 1.12 ms), enough for two ranks (67 MB in 2.5 ms:
    // 4.16 ms per block step against 4.41 ms with copy CTAs), not for eight.
    w->copy_ctas_auto = w->copy_ctas <= 0;
    if (w->copy_ctas <= 0) w->copy_ctas = 16;
    if (w->copy_mode < 0) w->copy_mode = w->tp <= 2 ? 1 : 0;
    int tiles_m = (M + kBM - 1) / kBM;
    if (st == XCCL_OK && (M % kBM != 0 || tiles_m % w->tp != 0)) st = XCCL_ERR_INVALID_PARAM;
    for (int l = 0; l < w->n_local && st == XCCL_OK; l++) {
        void *p = nullptr;
        if (cudaMalloc(&p, (size_t)tiles_m * 4) != cudaSuccess) {
            st = XCCL_ERR_NO_MEMORY;
            break;
        }
        cudaMemset(p, 0, (size_t)tiles_m * 4);
        w->allocs.push_back(p);
        w->ready[l] = (uint32_t *)p;
        void  *f = nullptr;
        size_t chunks = (size_t)(M / w->tp + w->in_rows - 1) / w->in_rows;
        if (cudaMalloc(&f, chunks * 4) != cudaSuccess) {
            st = XCCL_ERR_NO_MEMORY;
            break;
        }
        cudaMemset(f, 0, chunks * 4);
        w->allocs.push_back(f);
        w->in_flags[l] = (uint32_t *)f;
    }
    if (st == XCCL_OK) {
        void *p = nullptr;
        if (cudaMalloc(&p, 4) != cudaSuccess) {
            st = XCCL_ERR_NO_MEMORY;
        } else {
            cudaMemset(p, 0, 4);
            w->allocs.push_back(p);
            w->error = (uint32_t *)p;
        }
    }
    cudaDeviceSynchronize();
    if (st != XCCL_OK) {
        xccl_tp_ws_destroy(w);
        return st;
    }
    *out = w;
    return XCCL_OK;
}

void xccl_tp_ws_destroy(xccl_tp_ws_h w)
{
    if (w == nullptr) return;
    cudaDeviceSynchronize();
    for (void *p : w->allocs) cudaFree(p);
    if (w->in_consumed != nullptr) cudaEventDestroy(w->in_consumed);
    delete w->region;
    delete w;
}

void *xccl_tp_ws_x_shard(xccl_tp_ws_h w, int local_rank)
{
    if (w == nullptr || local_rank < 0 || local_rank >= w->n_local) return nullptr;
    int r = w->rank_base + local_rank;
    return w->xg(r) + (size_t)r * (w->M / w->tp) * w->K;
}

void *xccl_tp_ws_x_full(xccl_tp_ws_h w, int local_rank)
{
    if (w == nullptr || local_rank < 0 || local_rank >= w->n_local) return nullptr;
    return w->xg(w->rank_base + local_rank);
}

uint32_t xccl_tp_ws_error(xccl_tp_ws_h w)
{
    uint32_t v = 0;
    if (w == nullptr) return 0xffffffffu;
    cudaMemcpy(&v, w->error, 4, cudaMemcpyDeviceToHost);
    return v;
}

xccl_status_t xccl_tp_ag_gemm_swiglu(xccl_tp_ws_h w, const void *const *Wg, const void *const *Wu, void *const *Hout,
                                     int F_local, void *stream)
{
    if (w == nullptr || Wg == nullptr || Wu == nullptr || Hout == nullptr || F_local % (kBN / 2) != 0) {
        return XCCL_ERR_INVALID_PARAM;
    }
    if (w->tp == 1 && !w->in_active) {  // one rank, the rows are there
        SkinnyArgs    sk{};
        xccl_status_t sst;
        sk.M = w->M; sk.N = F_local; sk.K = w->K; sk.swiglu = true;
        sk.A = w->xg(0); sk.B0 = Wg[0]; sk.B1 = Wu[0]; sk.C = Hout[0]; sk.ldc = F_local; sk.error = w->error;
        if (try_skinny(sk, (cudaStream_t)stream, &sst)) return sst;
    }
    GemmParams p{};
    GemmLaunch l{};
    p.M = w->M;
    p.N = 2 * F_local;
    p.K = w->K;
    p.epilogue  = EPI_SWIGLU;
    p.comm      = w->tp > 1 ? COMM_ALLGATHER_A : COMM_NONE;
    p.tp_size   = w->tp;
    p.rank_base = w->rank_base;
    p.seq       = ++w->seq_ag;
    p.error     = w->error;
    p.ldc       = F_local;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int ctas      = sms / w->n_local;
    int copy_ctas = copy_ctas_of(w, p.N, ctas);
    l.n_local     = w->n_local;
    l.ctas        = ctas;
    l.cooperative = w->tp > 1;
    p.n_gemm_ctas = ctas - copy_ctas;
    p.copy_mode   = w->copy_mode;
    p.bn          = gemm_tile_cols(p.M, p.N, p.K, true, tile_walk(p, l));
    for (int r = 0; r < w->tp; r++) {
        p.xg[r]  = w->xg(r);
        p.pad[r] = w->pad(r);
    }
    for (int i = 0; i < w->n_local; i++) {
        p.C[i]     = (__nv_bfloat16 *)Hout[i];
        p.ready[i] = w->ready[i];
        xccl_status_t st = make_tensor_map_2d(&l.tmA[i], w->xg(w->rank_base + i), (uint64_t)w->M, (uint64_t)w->K,
                                              (uint64_t)w->K, kBM);
        if (st != XCCL_OK) return st;
        st = make_tensor_map_2d(&l.tmB0[i], Wg[i], (uint64_t)F_local, (uint64_t)w->K, (uint64_t)w->K, (uint32_t)p.bn / 2);
        if (st != XCCL_OK) return st;
        st = make_tensor_map_2d(&l.tmB1[i], Wu[i], (uint64_t)F_local, (uint64_t)w->K, (uint64_t)w->K, (uint32_t)p.bn / 2);
        if (st != XCCL_OK) return st;
        if (w->in_active) p.in_ready[i] = w->in_flags[i];
    }
    if (w->in_active) {
        p.in_target        = w->in_seq;
        p.in_rows_per_flag = w->in_rows;
        // H2D_PHASES (with copy CTAs; every rank of the team must run with the same setting): every rank reports its
        // rows block by block and the walk takes row block c of every shard before c + 1. Otherwise the peers' shards
        // are read whole and only the local rows ramp.
        const bool phases  = w->tp > 1 && w->copy_mode == 0 && w->in_ramp == 2;
        p.group_ramp       = w->in_ramp == 0 ? 0 : phases ? 2 : 1;
    }
    xccl_status_t lst = launch_gemm(p, l, (cudaStream_t)stream);
    if (w->in_active && lst == XCCL_OK) {
        // the next host->device copy into the shard may start once this kernel has consumed it
        if (w->in_consumed == nullptr) XCCL_CUDA_CHECK(cudaEventCreateWithFlags(&w->in_consumed, cudaEventDisableTiming));
        XCCL_CUDA_CHECK(cudaEventRecord(w->in_consumed, (cudaStream_t)stream));
    }
    w->in_active = false;
    return lst;
}

// The overlapped input copy in two halves, so that the caller can launch the consuming kernel BETWEEN them: the kernel
// then starts at once and waits for rows, and the host time of issuing the chunks (two driver calls per chunk) is spent
// while the GPU already works. `expect` fixes the sequence number the next allgather->GEMM waits for and orders the copy
// stream after the kernel that read the shard last; `issue` enqueues the chunks and their flag writes. ramp != 0: the
// kernel walks the local rows in groups of 1, 1, 2, 4, ... row blocks, so its first wave needs the first chunk only
// (for a step that starts with an idle GPU; a pipelined caller, whose copy runs under the previous step's second
// kernel, passes 0 and keeps the full groups). ramp == 2 (or the option H2D_PHASES): with copy CTAs, phases over all
// shards as described at GemmParams::group_ramp; every rank of the team must ask for the same.
xccl_status_t xccl_tp_h2d_expect(xccl_tp_ws_h w, void *copy_stream, int ramp)
{
    if (w == nullptr) return XCCL_ERR_INVALID_PARAM;
    if (w->in_active) return XCCL_ERR_NO_RESOURCE;  // one copy per allgather->GEMM
    if (w->in_consumed != nullptr) XCCL_CUDA_CHECK(cudaStreamWaitEvent((cudaStream_t)copy_stream, w->in_consumed, 0));
    w->in_seq++;
    w->in_active = true;
    w->in_ramp   = (ramp == 0 || !tp_options().flag("H2D_RAMP")) ? 0 : (ramp == 2 || tp_options().flag("H2D_PHASES")) ? 2 : 1;
    return XCCL_OK;
}

xccl_status_t xccl_tp_h2d_issue(xccl_tp_ws_h w, const void *const *host_x, void *copy_stream)
{
    if (w == nullptr || host_x == nullptr) return XCCL_ERR_INVALID_PARAM;
    XCCL_DRIVER_FN(cuStreamWriteValue32);
    cudaStream_t cs = (cudaStream_t)copy_stream;
    const size_t rows = (size_t)w->M / w->tp, row_bytes = (size_t)w->K * 2;
    for (int i = 0; i < w->n_local; i++) {
        char       *dst = (char *)xccl_tp_ws_x_shard(w, i);
        const char *src = (const char *)host_x[i];
        size_t      c   = 0;
        for (size_t r0 = 0; r0 < rows; r0 += (size_t)w->in_rows, c++) {
            const size_t n = std::min((size_t)w->in_rows, rows - r0);
            XCCL_CUDA_CHECK(cudaMemcpyAsync(dst + r0 * row_bytes, src + r0 * row_bytes, n * row_bytes, cudaMemcpyHostToDevice, cs));
            XCCL_CU_CHECK(cuStreamWriteValue32((CUstream)cs, (CUdeviceptr)(w->in_flags[i] + c), w->in_seq, 0));
        }
    }
    return XCCL_OK;
}

xccl_status_t xccl_tp_h2d_begin(xccl_tp_ws_h w, const void *const *host_x, void *copy_stream)
{
    xccl_status_t st = xccl_tp_h2d_expect(w, copy_stream, 1);
    return st != XCCL_OK ? st : xccl_tp_h2d_issue(w, host_x, copy_stream);
}

// Host-side view of the number of copy CTAs (tests).
int xccl_tp_copy_ctas(int tp, int copy_mode, int want, int emulated_auto, int shard_rows, int columns, int ctas)
{
    return copy_ctas(tp, copy_mode, want, emulated_auto != 0, shard_rows, columns, ctas);
}

xccl_status_t xccl_tp_gemm_rs(xccl_tp_ws_h w, const void *const *Hin, const void *const *Wd, void *const *Yout,
                              int F_local, void *stream)
{
    if (w == nullptr || Hin == nullptr || Wd == nullptr || Yout == nullptr || F_local % 8 != 0) return XCCL_ERR_INVALID_PARAM;
    if (w->tp == 1) {
        SkinnyArgs    sk{};
        xccl_status_t sst;
        sk.M = w->M; sk.N = w->N_rs; sk.K = F_local;
        sk.A = Hin[0]; sk.B0 = Wd[0]; sk.C = Yout[0]; sk.ldc = w->N_rs; sk.error = w->error;
        if (try_skinny(sk, (cudaStream_t)stream, &sst)) return sst;
    }
    GemmParams p{};
    GemmLaunch l{};
    p.M = w->M;
    p.N = w->N_rs;
    p.K = F_local;
    p.epilogue  = EPI_STORE;
    p.comm      = w->tp > 1 ? COMM_REDUCE_SCATTER_C : COMM_NONE;
    p.tp_size   = w->tp;
    p.rank_base = w->rank_base;
    p.seq       = ++w->seq_rs;
    p.error     = w->error;
    p.ldc       = w->N_rs;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    l.n_local     = w->n_local;
    l.ctas        = sms / w->n_local;
    p.n_gemm_ctas = l.ctas;
    p.bn          = gemm_tile_cols(p.M, p.N, p.K, false, tile_walk(p, l));
    w->rs_count[p.seq & 1] += rs_arrivals_total(p.N);
    p.rs_target = w->rs_count[p.seq & 1];
    p.rs_fused  = w->rs_fused ? 1 : 0;
    p.rs_debug_local = w->rs_debug_local ? 1 : 0;
    l.cooperative = w->emulated && w->tp > 1;  // emulated ranks wait on one another inside one launch
    for (int r = 0; r < w->tp; r++) {
        p.part[r] = w->part(r);
        p.pad[r]  = w->pad(r);
    }
    for (int i = 0; i < w->n_local; i++) {
        p.C[i] = (__nv_bfloat16 *)Yout[i];
        xccl_status_t st = make_tensor_map_2d(&l.tmA[i], Hin[i], (uint64_t)w->M, (uint64_t)F_local, (uint64_t)F_local, kBM);
        if (st != XCCL_OK) return st;
        st = make_tensor_map_2d(&l.tmB0[i], Wd[i], (uint64_t)w->N_rs, (uint64_t)F_local, (uint64_t)F_local, (uint32_t)p.bn / 2);
        if (st != XCCL_OK) return st;
        l.tmB1[i] = l.tmB0[i];
    }
    return launch_gemm(p, l, (cudaStream_t)stream);
}


xccl_status_t xccl_tp_quantize_rows(const void *x_bf16, int rows, int K, void *out8, float *scales, void *stream)
{
    if (x_bf16 == nullptr || out8 == nullptr || scales == nullptr || rows <= 0 || K <= 0 || K % 128 != 0) {
        return XCCL_ERR_INVALID_PARAM;
    }
    const size_t   blocks = (size_t)rows * (K / 128);
    const unsigned grid   = (unsigned)((blocks + 63) / 64);   // eight warps of eight blocks
    const bool     wide   = ((uintptr_t)x_bf16 & 15) == 0 && ((uintptr_t)out8 & 7) == 0;
    auto           k      = wide ? quantize_rows_1x128_kernel<8> : quantize_rows_1x128_kernel<4>;
    k<<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16 *)x_bf16, blocks, (uint8_t *)out8, scales);
    XCCL_CUDA_CHECK(cudaGetLastError());
    return XCCL_OK;
}

void *xccl_tp_ws_x8_shard(xccl_tp_ws_h w, int local_rank)
{
    if (w == nullptr || local_rank < 0 || local_rank >= w->n_local) return nullptr;
    int r = w->rank_base + local_rank;
    return (uint8_t *)w->xg(r) + (size_t)r * (w->M / w->tp) * w->K;
}

float *xccl_tp_ws_sx_shard(xccl_tp_ws_h w, int local_rank)
{
    if (w == nullptr || local_rank < 0 || local_rank >= w->n_local || w->K % 128 != 0) return nullptr;
    int r = w->rank_base + local_rank;
    return w->sx(r) + (size_t)r * (w->M / w->tp) * (w->K / 128);
}

xccl_status_t xccl_tp_ag_gemm_swiglu_fp8(xccl_tp_ws_h w, const void *const *Wg8, const float *const *sWg,
                                         const void *const *Wu8, const float *const *sWu, void *const *Hout, int F_local,
                                         void *stream)
{
    return xccl_tp_ag_gemm_swiglu_fp8q(w, Wg8, sWg, Wu8, sWu, Hout, nullptr, F_local, stream);
}

xccl_status_t xccl_tp_ag_gemm_swiglu_fp8q(xccl_tp_ws_h w, const void *const *Wg8, const float *const *sWg,
                                          const void *const *Wu8, const float *const *sWu, void *const *Hout,
                                          float *const *out_scales, int F_local, void *stream)
{
    if (w == nullptr || Wg8 == nullptr || sWg == nullptr || Wu8 == nullptr || sWu == nullptr || Hout == nullptr ||
        F_local % 128 != 0 || w->K % 128 != 0) {
        return XCCL_ERR_INVALID_PARAM;
    }
    if (w->tp == 1) {
        SkinnyArgs    sk{};
        xccl_status_t sst;
        sk.M = w->M; sk.N = F_local; sk.K = w->K; sk.fp8 = true; sk.swiglu = true;
        sk.A = w->xg(0); sk.B0 = Wg8[0]; sk.B1 = Wu8[0]; sk.C = Hout[0]; sk.ldc = F_local; sk.error = w->error;
        sk.sa = w->sx(0); sk.sb0 = sWg[0]; sk.sb1 = sWu[0]; sk.out_scale = out_scales != nullptr ? out_scales[0] : nullptr;
        if (try_skinny(sk, (cudaStream_t)stream, &sst)) return sst;
    }
    GemmParams p{};
    GemmLaunch l{};
    p.M = w->M;
    p.N = 2 * F_local;
    p.K = w->K;
    p.epilogue  = EPI_SWIGLU;
    p.comm      = w->tp > 1 ? COMM_ALLGATHER_A : COMM_NONE;
    p.tp_size   = w->tp;
    p.rank_base = w->rank_base;
    p.seq       = ++w->seq_ag;
    p.error     = w->error;
    p.ldc       = F_local;   // elements of the output row: bf16 values, or e4m3 bytes with out_scales
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int ctas      = sms / w->n_local;
    int copy_ctas = copy_ctas_of(w, p.N, ctas);
    l.n_local     = w->n_local;
    l.ctas        = ctas;
    l.cooperative = w->tp > 1;
    p.n_gemm_ctas = ctas - copy_ctas;
    p.copy_mode   = w->copy_mode;
    if (out_scales != nullptr) p.out_fp8 = 1;
    for (int r = 0; r < w->tp; r++) {
        p.xg[r]  = w->xg(r);
        p.sg[r]  = w->sx(r);
        p.pad[r] = w->pad(r);
    }
    for (int i = 0; i < w->n_local; i++) {
        p.C[i]     = (__nv_bfloat16 *)Hout[i];
        p.ready[i] = w->ready[i];
        p.sb0[i]   = sWg[i];
        p.sb1[i]   = sWu[i];
        xccl_status_t st = make_tensor_map_u8(&l.tmA[i], w->xg(w->rank_base + i), (uint64_t)w->M, (uint64_t)w->K, 128);
        if (st != XCCL_OK) return st;
        st = make_tensor_map_u8(&l.tmB0[i], Wg8[i], (uint64_t)F_local, (uint64_t)w->K, kBN / 2);
        if (st != XCCL_OK) return st;
        st = make_tensor_map_u8(&l.tmB1[i], Wu8[i], (uint64_t)F_local, (uint64_t)w->K, kBN / 2);
        if (st != XCCL_OK) return st;
        if (out_scales != nullptr) p.out_scale[i] = out_scales[i];
    }
    return launch_gemm_fp8(p, l, (cudaStream_t)stream);
}

xccl_status_t xccl_tp_gemm_rs_fp8(xccl_tp_ws_h w, const void *const *H8, const float *const *sH, const void *const *Wd8,
                                  const float *const *sWd, void *const *Yout, int F_local, void *stream)
{
    if (w == nullptr || H8 == nullptr || sH == nullptr || Wd8 == nullptr || sWd == nullptr || Yout == nullptr ||
        F_local % 128 != 0 || w->N_rs % 128 != 0) {
        return XCCL_ERR_INVALID_PARAM;
    }
    if (w->tp == 1) {
        SkinnyArgs    sk{};
        xccl_status_t sst;
        sk.M = w->M; sk.N = w->N_rs; sk.K = F_local; sk.fp8 = true;
        sk.A = H8[0]; sk.B0 = Wd8[0]; sk.C = Yout[0]; sk.ldc = w->N_rs; sk.error = w->error;
        sk.sa = sH[0]; sk.sb0 = sWd[0];
        if (try_skinny(sk, (cudaStream_t)stream, &sst)) return sst;
    }
    GemmParams p{};
    GemmLaunch l{};
    p.M = w->M;
    p.N = w->N_rs;
    p.K = F_local;
    p.epilogue  = EPI_STORE;
    p.comm      = w->tp > 1 ? COMM_REDUCE_SCATTER_C : COMM_NONE;
    p.tp_size   = w->tp;
    p.rank_base = w->rank_base;
    p.seq       = ++w->seq_rs;
    p.error     = w->error;
    p.ldc       = w->N_rs;
    w->rs_count[p.seq & 1] += rs_arrivals_total(p.N);
    p.rs_target = w->rs_count[p.seq & 1];
    p.rs_fused  = w->rs_fused ? 1 : 0;
    p.rs_debug_local = w->rs_debug_local ? 1 : 0;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    l.n_local     = w->n_local;
    l.ctas        = sms / w->n_local;
    l.cooperative = w->emulated && w->tp > 1;
    p.n_gemm_ctas = l.ctas;
    for (int r = 0; r < w->tp; r++) {
        p.part[r] = w->part(r);
        p.pad[r]  = w->pad(r);
    }
    for (int i = 0; i < w->n_local; i++) {
        p.C[i]   = (__nv_bfloat16 *)Yout[i];
        p.sb0[i] = sWd[i];
        // activation scales are local here: the kernel reads them through the TEAM-rank slot of this local rank
        p.sg[w->rank_base + i] = const_cast<float *>(sH[i]);
        xccl_status_t st = make_tensor_map_u8(&l.tmA[i], H8[i], (uint64_t)w->M, (uint64_t)F_local, 128);
        if (st != XCCL_OK) return st;
        st = make_tensor_map_u8(&l.tmB0[i], Wd8[i], (uint64_t)w->N_rs, (uint64_t)F_local, kBN / 2);
        if (st != XCCL_OK) return st;
        l.tmB1[i] = l.tmB0[i];
    }
    return launch_gemm_fp8(p, l, (cudaStream_t)stream);
}

}  // extern "C"
