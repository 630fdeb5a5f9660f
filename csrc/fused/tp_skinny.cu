// GEMM kernels for few rows of activations (see tp_skinny.cuh).
//
// What bounds such a product is reading the weights once. A tile of the large kernel is 256 rows of A high, so with 16
// or 128 rows its grid is N / 256 CTA pairs that each walk all of K: 32 of 74 pairs for N = 8192, and half of the SMs'
// loads are never issued. Here the operands change places: 128 rows of the WEIGHTS are the M side of tcgen05.mma, the
// activations (rounded up to 16 rows) its N side, and the CTAs of a cluster share the K blocks of a tile, so that the
// grid fills the chip (up to two CTAs per SM, one in fp8 with more than 32 tokens or SwiGLU) and each keeps its whole ring
// of weight loads in flight. Measured on one B200, operands in DRAM, before (large kernel with 256-column tiles) and now: bf16
// 16 x 8192 x 8192 (134 MB of weights) 47.5 -> 26.5 us, 128 x 8192 x 8192 49.0 -> 34.2 us; SwiGLU 16 x 3584 x 8192 69.0 ->
// 26.2 us; fp8 64 x 7168 x 8192 49.2 -> 18.6 us.
// One MMA holds 128 rows; more of them come in several blocks where that pays (skinny_plan_rows). On both sides of the line at
// 128 rows, this kernel / the large one with the narrower tiles it now has, L2 flushed, event times in steps of 2 us: bf16 N 8192,
// K 8192 40.9 / 53.2, K 2048 20.5 / 20.7, K 512 15.7 / 14.6; N 2048, K 1024 16.3 / 14.5 (K up to 1024 is where the large one is level
// or up to 2 us ahead); SwiGLU N 8192, K 2048 37 / 50; fp8 N 8192, K 2048 19 / 26, N 28672, K 512 22.3 / 20.6.
//
//   warp 0     TMA producer: weights (streamed, evict first) and activations (kept in L2) of a K block per stage
//   warp 1     MMA issuer, accumulators in tensor memory: lane = weight row, column = token
//   warps 2..  bf16: four warps read the accumulator once. fp8: eight warps add every K block's product into fp32
//              registers with the scales that warp 10 has multiplied into shared memory
//   the end    every CTA of the cluster puts its fp32 partial sums into its own shared memory, token by token, and adds
//              up the tokens it owns over the cluster (distributed shared memory, in rank order: same bits every run),
//              applies the epilogue and writes rows of 128 outputs
#include <algorithm>
#include <atomic>
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "../cuda/cuda_common.h"
#include "sm100_ptx.cuh"
#include "tp_gemm.cuh"
#include "tp_device.cuh"
#include "tp_skinny.cuh"

namespace xccl {
namespace tp {

namespace {

constexpr uint32_t kWBytes      = 128 * 128;  // one block of weights: 128 rows x 128 bytes of K
constexpr int      kMaxStages   = 8;
constexpr int      kScaleSlots  = 8;
constexpr int      kScaleGroup  = 4;          // K blocks whose scales are loaded together
constexpr int      kMaxBuf      = 4;
constexpr int      kSkinnyThreads = 192, kSkinnyThreadsFp8 = 352;
constexpr uint32_t kBarBytes    = 512;

struct SkinnyParams {
    int M, N, K, ldc;
    SkinnyPlan plan;
    const float *sa, *sb0, *sb1;
    float       *out_scale;
    void        *C;
    uint32_t    *error;
    unsigned long long budget_ns;
};

struct SkinnyMaps {
    CUtensorMap a, b0, b1;
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// kCW: fp8, tokens per promotion warp (mn / 2); 0 in bf16. kOcc: CTAs per SM the registers are cut for.
template <bool kFp8, bool kSwi, int kCW, int kOcc>
__global__ void __launch_bounds__(kFp8 ? kSkinnyThreadsFp8 : kSkinnyThreads, kOcc)
skinny_kernel(SkinnyParams p, const __grid_constant__ SkinnyMaps maps)
{
    constexpr int kEpiWarps = kFp8 ? 8 : 4;
    constexpr int kMats     = kSwi ? 2 : 1;
    constexpr int kKE       = kFp8 ? 128 : 64;  // K elements of a block
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint32_t s_tmem, s_abort;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t       *gen  = smem_raw + (base - smem_u32(smem_raw));
    const int      mn = p.plan.mn, stages = p.plan.stages, nbuf = p.plan.nbuf;
    const uint32_t stage_bytes = kWBytes * kMats + (uint32_t)mn * 128;
    const uint32_t ring   = base;
    const uint32_t bars   = base + stages * stage_bytes;
    float         *scales = reinterpret_cast<float *>(gen + stages * stage_bytes + kBarBytes);  // [kScaleSlots][kMats][mn]
    float         *red    = reinterpret_cast<float *>(gen);                                     // [chunk][kMats][128], after the last K block
    auto full_bar       = [&](int s) { return bars + 8u * s; };
    auto empty_bar      = [&](int s) { return bars + 8u * (kMaxStages + s); };
    auto tmem_full_bar  = [&](int a) { return bars + 8u * (2 * kMaxStages + a); };
    auto tmem_empty_bar = [&](int a) { return bars + 8u * (2 * kMaxStages + kMaxBuf + a); };

    const int  warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int  split = blockIdx.x, tile = blockIdx.y;  // split = rank in the cluster
    const int  m0   = (int)blockIdx.z * mn;            // first token of this block of rows
    const int  rows = min(p.M - m0, mn);
    const int  kb_lo = (int)((long)split * p.plan.kblocks / p.plan.splits);
    const int  kb_hi = (int)((long)(split + 1) * p.plan.kblocks / p.plan.splits);
    AbortFlag  ab{&s_abort, p.error, p.budget_ns};

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < stages; s++) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < nbuf; a++) {
            mbar_init(tmem_full_bar(a), kFp8 ? 2 : 1);  // fp8: the product and its scales
            mbar_init(tmem_empty_bar(a), kEpiWarps);
        }
        mbar_fence_init();
        tma_prefetch_desc(&maps.a);
        tma_prefetch_desc(&maps.b0);
        if (kSwi) tma_prefetch_desc(&maps.b1);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&s_tmem), p.plan.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = s_tmem;

    float acc[kFp8 ? kMats * kCW : 1];  // fp8: running sums of this warp's tokens, [matrix][token]
    const int quarter = warp % 4;       // TMEM lanes a warp may read
    const int half    = (warp - 2) / 4; // fp8: which half of the tokens

    if (warp == 0) {
        if (elect_one()) {
            // (several blocks of rows read the same weights at about the same time)
            const uint64_t pol_a = l2_policy_evict_last(), pol_w = gridDim.z == 1 ? l2_policy_evict_first() : pol_a;
            int      s = 0;
            uint32_t phase = 0;
            int      issued = 0;
            bool     ok = true;
            for (int kb = kb_lo; kb < kb_hi; kb++) {
                if (!mbar_wait(empty_bar(s), phase ^ 1, ab, 2)) {
                    ok = false;
                    break;
                }
                const uint32_t st = ring + s * stage_bytes;
                mbar_arrive_expect_tx(full_bar(s), stage_bytes);
                tma_load_2d_hint(st, &maps.b0, kb * kKE, tile * 128, full_bar(s), pol_w);
                if (kSwi) tma_load_2d_hint(st + kWBytes, &maps.b1, kb * kKE, tile * 128, full_bar(s), pol_w);
                tma_load_2d_hint(st + kMats * kWBytes, &maps.a, kb * kKE, m0, full_bar(s), pol_a);
                issued++;
                if (++s == stages) {
                    s = 0;
                    phase ^= 1;
                }
            }
            if (!ok) {
                // let the copies that are still in flight land before the memory is reused: bounded wait per stage
                for (int i = 0; i < min(issued, stages); i++) {
                    const int      g = issued - 1 - i;  // the last load of each stage
                    for (int spin = 0; spin < (1 << 16); spin++) {
                        if (mbar_try_wait(full_bar(g % stages), (uint32_t)(g / stages) & 1u)) break;
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t idesc = kFp8 ? make_idesc(0, 0, 128, (uint32_t)mn) : make_idesc(1, 1, 128, (uint32_t)mn);
            int      s = 0, a = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool     ok = true;
            for (int kb = kb_lo; kb < kb_hi && ok; kb++) {
                if (!mbar_wait(full_bar(s), phase, ab, 4)) break;
                if (kFp8 && !mbar_wait(tmem_empty_bar(a), acc_phase ^ 1, ab, 3)) break;
                tc_fence_after();
                const uint32_t st = ring + s * stage_bytes;
                const uint64_t dt = make_desc_sw128(st + kMats * kWBytes);
#pragma unroll
                for (int m = 0; m < kMats; m++) {
                    const uint64_t dw = make_desc_sw128(st + m * kWBytes);
                    const uint32_t d  = tmem_base + (uint32_t)(a * p.plan.cols + m * (p.plan.cols / kMats));
#pragma unroll
                    for (int k = 0; k < 4; k++) {  // 32 bytes of K per instruction
                        if (kFp8) {
                            mma_f8(d, dw + (uint64_t)(k * 2), dt + (uint64_t)(k * 2), idesc, k != 0);
                        } else {
                            mma_f16(d, dw + (uint64_t)(k * 2), dt + (uint64_t)(k * 2), idesc, (kb > kb_lo || k != 0) ? 1u : 0u);
                        }
                    }
                }
                if (kFp8) {
                    mma_commit(tmem_full_bar(a));
                    if (++a == nbuf) {
                        a = 0;
                        acc_phase ^= 1;
                    }
                }
                mma_commit(empty_bar(s));
                if (++s == stages) {
                    s = 0;
                    phase ^= 1;
                }
            }
            if (!kFp8) mma_commit(tmem_full_bar(0));
        }
        __syncwarp();
    } else if (kFp8 && warp == 2 + kEpiWarps) {
        // activation scale x weight scale of every token for the K blocks ahead. The loads are unconditional (clamped) and
        // those of the next four K blocks are in flight while this group's products are handed over: their latency from
        // DRAM is about two K blocks' share of the time. A product buffer counts as full when its scales are there too, so the
        // promotion warps wait once per K block. Product n's scales are written when product n - nbuf and its scales are
        // complete: then everybody has emptied n - 2 nbuf, and the slot's last reader was n - kScaleSlots. After a wait that ran
        // out the K blocks go by unheeded, so that the lanes stay together (leaving by the flag: 64 x 7168 x 8192 18.6 us, so 20.0).
        static_assert(kScaleSlots >= 2 * kMaxBuf, "a slot's last reader has finished");
        constexpr int kNT = kCW > 0 ? kCW / 16 : 1;  // tokens per lane
        const int    kbn = p.plan.kblocks;
        const float *w0  = p.sb0 + (size_t)tile * kbn, *w1 = kSwi ? p.sb1 + (size_t)tile * kbn : w0;
        float x[2][kScaleGroup][kNT], u0[2][kScaleGroup], u1[2][kScaleGroup];
        auto load_group = [&](int g, float (&xx)[kScaleGroup][kNT], float (&uu0)[kScaleGroup], float (&uu1)[kScaleGroup]) {
#pragma unroll
            for (int i = 0; i < kScaleGroup; i++) {
                const int kb = min(g + i, kb_hi - 1);
                uu0[i] = __ldg(w0 + kb);
                uu1[i] = __ldg(w1 + kb);
#pragma unroll
                for (int j = 0; j < kNT; j++) xx[i][j] = __ldcg(p.sa + (size_t)(m0 + min(lane + 32 * j, rows - 1)) * kbn + kb);
            }
        };
        int      slot = 0, a = 0;
        uint32_t phase = 0;
        load_group(kb_lo, x[0], u0[0], u1[0]);
        for (int g = kb_lo; g < kb_hi; g += 2 * kScaleGroup) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                load_group(g + (h + 1) * kScaleGroup, x[1 - h], u0[1 - h], u1[1 - h]);
#pragma unroll
                for (int i = 0; i < kScaleGroup; i++) {
                    if (g + h * kScaleGroup + i >= kb_hi) continue;
                    (void)mbar_wait(tmem_full_bar(a), phase ^ 1, ab, 7);
                    float *dst = scales + slot * kMats * mn;
#pragma unroll
                    for (int j = 0; j < kNT; j++) {
                        dst[lane + 32 * j] = x[h][i][j] * u0[h][i];
                        if (kSwi) dst[mn + lane + 32 * j] = x[h][i][j] * u1[h][i];
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tmem_full_bar(a));
                    if (++slot == kScaleSlots) slot = 0;
                    if (++a == nbuf) {
                        a = 0;
                        phase ^= 1;
                    }
                }
            }
        }
    } else if (kFp8) {
        // What bounds the loop is its serial chain: all of a chunk's columns and scales are on their way before the first is
        // waited for, and there is one wait per K block (with one for the scales beside it and sixteen columns at a time 64 x 7168
        // x 8192 took 18.5 us, now 17.8, the block step of 128 tokens, 8192, 14336 115.7, now 110.3).
        constexpr int kB = kMats * kCW > 64 || kCW < 32 ? 16 : 32;   // columns (tokens) at a time
        int      a = 0, slot = 0;
        uint32_t acc_phase = 0;
#pragma unroll
        for (int j = 0; j < kMats * kCW; j++) acc[j] = 0.0f;
        for (int kb = kb_lo; kb < kb_hi; kb++) {
            // (as in the scale warp, the lanes stay together after a wait that ran out)
            (void)mbar_wait(tmem_full_bar(a), acc_phase, ab, 5);
            tc_fence_after();
            const float   *sc = scales + slot * kMats * mn + half * kCW;
            const uint32_t t0 = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(a * p.plan.cols + half * kCW);
#pragma unroll
            for (int m = 0; m < kMats; m++) {
#pragma unroll
                for (int c = 0; c < kCW; c += kB) {
                    uint32_t v[kB / 16][16];
                    float4   f[kB / 4];
#pragma unroll
                    for (int b = 0; b < kB / 16; b++) tmem_ld_32x16(t0 + m * (p.plan.cols / kMats) + c + 16 * b, v[b]);
#pragma unroll
                    for (int e = 0; e < kB / 4; e++) f[e] = *reinterpret_cast<const float4 *>(sc + m * mn + c + 4 * e);
#pragma unroll
                    for (int b = 0; b < kB / 16; b++) tmem_ld_wait_16(v[b]);
#pragma unroll
                    for (int e = 0; e < kB; e += 4) {
                        const uint32_t *x = v[e / 16] + e % 16;
                        float          *s = acc + m * kCW + c + e;
                        s[0] = fmaf(f[e / 4].x, __uint_as_float(x[0]), s[0]);
                        s[1] = fmaf(f[e / 4].y, __uint_as_float(x[1]), s[1]);
                        s[2] = fmaf(f[e / 4].z, __uint_as_float(x[2]), s[2]);
                        s[3] = fmaf(f[e / 4].w, __uint_as_float(x[3]), s[3]);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tmem_empty_bar(a));
            if (++a == nbuf) {
                a = 0;
                acc_phase ^= 1;
            }
            if (++slot == kScaleSlots) slot = 0;
        }
    } else {
        mbar_wait_warp(tmem_full_bar(0), 0, ab, 5);
        tc_fence_after();
    }

    // ---- reduction over the cluster, `chunk` tokens per round, through the memory of the ring: every load has landed
    // and every MMA has read its stage (the accumulator's or the last product's barrier says so)
    __syncthreads();
    const bool epi = warp >= 2 && warp < 2 + kEpiWarps;
    const int  row = quarter * 32 + lane;  // weight row of the tile
    for (int t0 = 0; t0 < mn; t0 += p.plan.chunk) {
        const int t1 = min(t0 + p.plan.chunk, mn);
        if (epi && kFp8) {
#pragma unroll
            for (int m = 0; m < kMats; m++) {
#pragma unroll
                for (int c = 0; c < kCW; c++) {
                    const int t = half * kCW + c;
                    if (t >= t0 && t < t1) red[((t - t0) * kMats + m) * 128 + row] = acc[m * kCW + c];
                }
            }
        } else if (epi) {
            for (int m = 0; m < kMats; m++) {
                for (int c = t0; c < t1; c += 16) {
                    uint32_t v[16];
                    tmem_ld_32x16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(m * (p.plan.cols / kMats) + c), v);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 16; e++) red[((c + e - t0) * kMats + m) * 128 + row] = __uint_as_float(v[e]);
                }
            }
        }
        __syncwarp();
        cluster_sync_all();  // every CTA's partial sums of the round can be read
        if (epi) {
            const int tid = threadIdx.x - 64, nthr = kEpiWarps * 32;
            const int tokens = min(t1, rows) - t0;
            const int mine   = tokens > split ? (tokens - split + p.plan.splits - 1) / p.plan.splits : 0;
            // sixteen lanes share a token of 128 outputs, eight outputs each
            for (int it = tid; it < mine * 16; it += nthr) {
                const int t = split + (it / 16) * p.plan.splits, q = it % 16;
                float     x[kMats][8];
#pragma unroll
                for (int m = 0; m < kMats; m++) {
                    const uint32_t at = smem_u32(red + (t * kMats + m) * 128 + q * 8);
                    float4 a0 = make_float4(0, 0, 0, 0), a1 = a0;
                    // in rank order; two peers' values in flight (registers), the last one read twice if they are odd
                    for (int s = 0; s < p.plan.splits; s += 2) {
                        const uint32_t r0 = map_to_cta(at, (uint32_t)s), r1 = map_to_cta(at, (uint32_t)min(s + 1, p.plan.splits - 1));
                        const float4   v0 = ld_cluster_f4(r0), v1 = ld_cluster_f4(r0 + 16), v2 = ld_cluster_f4(r1), v3 = ld_cluster_f4(r1 + 16);
                        a0.x += v0.x; a0.y += v0.y; a0.z += v0.z; a0.w += v0.w;
                        a1.x += v1.x; a1.y += v1.y; a1.z += v1.z; a1.w += v1.w;
                        if (s + 1 < p.plan.splits) {
                            a0.x += v2.x; a0.y += v2.y; a0.z += v2.z; a0.w += v2.w;
                            a1.x += v3.x; a1.y += v3.y; a1.z += v3.z; a1.w += v3.w;
                        }
                    }
                    x[m][0] = a0.x; x[m][1] = a0.y; x[m][2] = a0.z; x[m][3] = a0.w;
                    x[m][4] = a1.x; x[m][5] = a1.y; x[m][6] = a1.z; x[m][7] = a1.w;
                }
                if (kSwi) {
#pragma unroll
                    for (int e = 0; e < 8; e++) x[0][e] = silu(x[0][e]) * x[kMats - 1][e];
                }
                const int col = tile * 128 + q * 8;
                if (kFp8 && kSwi && p.out_scale != nullptr) {
                    // the 128 outputs of the token are one quantisation block; the sixteen lanes are half a warp and all
                    // of them are here (N is a multiple of 128)
                    float amax = 0.0f;
#pragma unroll
                    for (int e = 0; e < 8; e++) amax = fmaxf(amax, fabsf(x[0][e]));
                    const unsigned mask = (lane < 16) ? 0x0000ffffu : 0xffff0000u;
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(mask, amax, o));
                    const float sc = fmaxf(amax, 1e-12f) / 448.0f, inv = 1.0f / sc;
                    if (q == 0) p.out_scale[(size_t)(m0 + t0 + t) * (size_t)(p.N / 128) + tile] = sc;
                    uint32_t w2[2];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        w2[h] = (uint32_t)__nv_cvt_float_to_fp8(x[0][4 * h] * inv, __NV_SATFINITE, __NV_E4M3) |
                                ((uint32_t)__nv_cvt_float_to_fp8(x[0][4 * h + 1] * inv, __NV_SATFINITE, __NV_E4M3) << 8) |
                                ((uint32_t)__nv_cvt_float_to_fp8(x[0][4 * h + 2] * inv, __NV_SATFINITE, __NV_E4M3) << 16) |
                                ((uint32_t)__nv_cvt_float_to_fp8(x[0][4 * h + 3] * inv, __NV_SATFINITE, __NV_E4M3) << 24);
                    }
                    *reinterpret_cast<uint2 *>((uint8_t *)p.C + (size_t)(m0 + t0 + t) * p.ldc + col) = make_uint2(w2[0], w2[1]);
                } else if (col < p.N) {
                    *reinterpret_cast<uint4 *>((__nv_bfloat16 *)p.C + (size_t)(m0 + t0 + t) * p.ldc + col) =
                        make_uint4(pack_bf16x2(x[0][0], x[0][1]), pack_bf16x2(x[0][2], x[0][3]),
                                   pack_bf16x2(x[0][4], x[0][5]), pack_bf16x2(x[0][6], x[0][7]));
                }
            }
        }
        __syncwarp();
        cluster_sync_all();  // nobody's shared memory is overwritten or gone while a peer reads it
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, p.plan.tmem_cols);
    }
}

int pow2_at_least(int v, int lo)
{
    int p = lo;
    while (p < v) p *= 2;
    return p;
}

// CTAs per SM for which the kernel's registers are cut. fp8 keeps mn / 2 sums per thread and matrix: with more than 16 of
// them the 80 registers of two CTAs per SM spill (64 x 7168 x 8192: 30.2 us, one CTA with 168 registers 18.6 us).
int skinny_occupancy(int mn, bool fp8, bool swiglu) { return fp8 && mn * (swiglu ? 2 : 1) > 32 ? 1 : 2; }

using SkinnyKernel = void (*)(SkinnyParams, SkinnyMaps);
SkinnyKernel skinny_kernel_of(int mn, bool fp8, bool swiglu)
{
    if (!fp8) return swiglu ? skinny_kernel<false, true, 0, 2> : skinny_kernel<false, false, 0, 2>;
    switch (mn) {
    case 32: return swiglu ? skinny_kernel<true, true, 16, 1> : skinny_kernel<true, false, 16, 2>;
    case 64: return swiglu ? skinny_kernel<true, true, 32, 1> : skinny_kernel<true, false, 32, 1>;
    default: return swiglu ? skinny_kernel<true, true, 64, 1> : skinny_kernel<true, false, 64, 1>;
    }
}

int kernel_index(int mn, bool fp8, bool swiglu)
{
    return !fp8 ? (swiglu ? 1 : 0) : 2 + 2 * (mn == 32 ? 0 : mn == 64 ? 1 : 2) + (swiglu ? 1 : 0);
}

// Dynamic shared memory of a CTA when `occ` of them share an SM (228 KB, 1 KB of it taken by each CTA).
constexpr int skinny_smem_budget(int occ) { return (occ == 2 ? 113 : 226) * 1024 - 64; }

// The largest number of CTAs up to `splits` (halved where it does not fit) that the device places as one cluster.
template <typename F> int placeable(int splits, F &&fits)
{
    while (splits > 1 && !fits(splits)) splits = (splits + 1) / 2;
    return splits;
}

void launch_config(const SkinnyPlan &plan, bool fp8, cudaStream_t stream, cudaLaunchConfig_t *cfg, cudaLaunchAttribute *attr)
{
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim          = dim3((unsigned)plan.splits, (unsigned)plan.tiles, (unsigned)plan.blocks);
    cfg->blockDim         = dim3(fp8 ? kSkinnyThreadsFp8 : kSkinnyThreads);
    cfg->dynamicSmemBytes = (size_t)plan.smem_bytes;
    cfg->stream           = stream;
    attr->id               = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)plan.splits;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    cfg->attrs    = attr;
    cfg->numAttrs = 1;
}

// Sets the kernel up on this device and lowers plan->splits to a cluster that it places: a partitioned device may have no
// room for eight CTAs in one GPC. Asked once per device, kernel and cluster size (properties that do not change, and the
// kernel's largest shared memory stands for all of its plans).
xccl_status_t prepare_kernel(SkinnyKernel k, int dev, bool fp8, bool swiglu, SkinnyPlan *plan)
{
    static std::atomic<unsigned char> ready[64][8], fit[64][8][9];   // fit: 0 not asked, 1 yes, 2 no
    const int id = kernel_index(plan->mn, fp8, swiglu);
    if (ready[dev][id].load() == 0) {
        XCCL_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
        ready[dev][id].store(1);
    }
    plan->splits = placeable(plan->splits, [&](int s) {
        auto &f = fit[dev][id][s];
        if (f.load() == 0) {
            SkinnyPlan         q = *plan;
            cudaLaunchConfig_t cfg;
            cudaLaunchAttribute attr[1];
            q.splits     = s;
            q.smem_bytes = skinny_smem_budget(skinny_occupancy(plan->mn, fp8, swiglu));
            launch_config(q, fp8, nullptr, &cfg, attr);
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) != cudaSuccess) (void)cudaGetLastError();
            if (clusters < 1) xccl_warn("few-rows gemm: no room for a cluster of %d CTAs on device %d", s, dev);
            f.store(clusters >= 1 ? 1 : 2);
        }
        return f.load() == 1;
    });
    return XCCL_OK;
}

}  // namespace

namespace {

// CTAs that share the K blocks of a tile: as many as run in one wave, as long as each gets enough K blocks to be worth its
// launch and its part of the reduction. A cluster lies inside one GPC: a B200 with room for 296 of these CTAs (148 with one
// per SM) places 71 (33) clusters of four, 45 (22) of six and 33 (15) of eight, so clusters may take 7/8 of the room, those
// of eight 3/4; pairs always fit. How many K blocks are enough depends on who else is there: four while half of the SMs are
// free, eight while every CTA has an SM to itself (16 for the large clusters, whose reduction is longer), 32 where two share
// an SM and one more only splits its bandwidth; for pairs always four.
// us with 1 / 2 / 3 / 4 / 6 / 8 CTAs per tile, L2 flushed, event times in steps of 2 us, the large kernel last:
//   bf16  16 x 1024 x  8192   32.8 / 22.5 / 18.4 / 18.0 / 16.4 / 14.4   39.1
//   bf16 128 x 4096 x  2048   24.6 / 19.8 / 18.4 / 18.4 / 22.5 / 24.7   18.6
//   bf16 128 x 6144 x  2048   24.6 / 20.4 / 21.5 / 22.6 / 32.8 / 36.9   20.6
//   bf16 128 x 6144 x 28672    178 /  106 / 90.1 / 80.3 /  107 / 99.4    123
//   bf16 128 x 8192 x  8192   61.5 / 43.0 / 41.0 / 40.9 / 57.3 / 59.1   53.2
//   fp8   64 x 2048 x  8192   26.7 / 20.5 / 18.5 / 18.5 / 18.5 / 26.7   43.2
//   fp8  128 x 5120 x 28672    115 / 65.7 / 51.2 / 78.3 / 67.6 / 82.5    133
int skinny_share(int tiles, int kblocks, int occ, int sms)
{
    int best = 1;
    for (int s : {2, 3, 4, 6, 8}) {
        const int ctas = s * tiles, room = occ * sms;
        if (ctas > (s == 2 ? room : s == 8 ? room * 3 / 4 : room * 7 / 8)) continue;
        int least = 32;
        if (ctas <= sms / 2 || s == 2) least = 4;
        else if (ctas <= sms) least = s >= 6 ? 16 : 8;
        if (kblocks >= least * s) best = s;
    }
    return best;
}

}  // namespace

// A plan for `blocks` blocks of up to M rows.
static bool plan_blocks(int M, int blocks, int N, int K, bool fp8, bool swiglu, int sms, SkinnyPlan *out)
{
    if (M <= 0 || M > kSkinnyMaxM || N <= 0 || K <= 0) return false;
    SkinnyPlan  q{};
    const int   mats = swiglu ? 2 : 1;
    q.blocks  = blocks;
    q.mn      = fp8 ? (M <= 32 ? 32 : M <= 64 ? 64 : 128) : (M + 15) / 16 * 16;
    q.tiles   = (N + 127) / 128;
    q.kblocks = (K + (fp8 ? 127 : 63)) / (fp8 ? 128 : 64);
    if (q.tiles > 65535) return false;
    const int occ     = skinny_occupancy(q.mn, fp8, swiglu);
    const int stage   = (int)kWBytes * mats + q.mn * 128;
    const int fixed   = 1024 + (int)kBarBytes + (fp8 ? kScaleSlots * mats * q.mn * 4 : 0);
    const int budget  = skinny_smem_budget(occ);
    q.stages  = std::min(kMaxStages, (budget - fixed) / stage);
    q.cols    = mats * (fp8 ? q.mn : (q.mn + 31) / 32 * 32);
    q.nbuf    = fp8 ? std::max(1, std::min(kMaxBuf, 512 / occ / q.cols)) : 1;
    q.tmem_cols = pow2_at_least(q.nbuf * q.cols, 32);
    q.splits  = skinny_share(q.tiles * blocks, q.kblocks, occ, sms);
    q.chunk   = std::min(q.mn, q.stages * stage / (512 * mats) / 16 * 16);
    q.smem_bytes = fixed + q.stages * stage;
    if (q.stages < 2 || q.chunk < 16) return false;
    *out = q;
    return true;
}

bool skinny_plan(int M, int N, int K, bool fp8, bool swiglu, int sms, SkinnyPlan *out)
{
    return plan_blocks(M, 1, N, K, fp8, swiglu, sms, out);
}

// Rows beyond one MMA, in blocks of up to 128: where the tiles of the large kernel (256 x 256, in bf16 narrower ones too) leave
// most of the chip idle, small tiles whose K is shared by a cluster fill it, although each block of rows reads the weights
// again (from L2). fp8: as long as every CTA has an SM to itself (the large kernel's fp8 tiles are all 256 columns wide), with
// SwiGLU only where CTAs share K. bf16: where at least three CTAs share more than 32 K blocks (with fewer 0.95 to 1.04 of the
// large kernel's time) and the CTAs are nine tenths of the SMs at most: clusters do not fill every SM, so with more of them some
// SMs run two and the rest waits for those (135 to 225 CTAs: 0.80 to 1.28 of the large kernel's time, 1.00 on average). SwiGLU in
// bf16 stays with the large kernel (0.89 of its speed). Operands in DRAM, launches back to back, 83 drawn bf16 products within the
// rule: 0.81 of the time on average, 1.00 the worst; 110 fp8 products and blocks 0.76 on average, 1.00 the worst. Large / few-rows
// kernel in us: bf16 206 x 576 x 7160 33.5 / 18.8, 370 x 1280 x 7032 32.9 / 23.0, 1654 x 336 x 3016 18.6 / 18.6, outside 480 x 1528 x 1672
// 14.4 / 18.5 and 590 x 1816 x 8072 41.1 / 46.2. L2 flushed: fp8 212 x 768 x 7808 54.3 / 20.5, 502 x 1664 x 5376 37.9 / 22.5, 8192 x 256 x 512
// 17.3 / 12.3; fp8 block step (SwiGLU and down projection) 256 rows, 1152, 4352 64.5 / 44.0, 512 rows, 5376, 2944 76.8 (97.2 with
// unshared SwiGLU tiles).
bool skinny_plan_rows(int M, int N, int K, bool fp8, bool swiglu, int sms, SkinnyPlan *out)
{
    if (M <= kSkinnyMaxM) return skinny_plan(M, N, K, fp8, swiglu, sms, out);
    const int blocks = (M - 1) / kSkinnyMaxM + 1;
    if ((swiglu && !fp8) || blocks > sms) return false;
    SkinnyPlan q{};
    if (!plan_blocks((M - 1) / blocks + 1, blocks, N, K, fp8, swiglu, sms, &q)) return false;
    const int ctas = q.blocks * q.tiles * q.splits;
    if (fp8 ? ctas > sms || (swiglu && q.splits < 2) : q.splits < 3 || q.kblocks <= 32 || ctas * 10 > sms * 9) return false;
    *out = q;
    return true;
}

// Whether a product runs here: the rule above, unless it is one for tiles and the user asks for a kind of them.
static bool takes(int M, int N, int K, bool fp8, bool swiglu, int sms, SkinnyPlan *out)
{
    return (M <= kSkinnyMaxM || !tiles_asked_for(fp8)) && skinny_plan_rows(M, N, K, fp8, swiglu, sms, out);
}

bool try_skinny(const SkinnyArgs &a, cudaStream_t stream, xccl_status_t *st)
{
    // what the large kernels refuse is left to them to refuse
    if ((a.fp8 ? (a.K % 128 != 0 || a.N % 128 != 0) : (a.K % 8 != 0 || a.N % 8 != 0))) return false;
    int        dev = 0, sms = 0;
    SkinnyPlan plan;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return false;
    if (!takes(a.M, a.N, a.K, a.fp8, a.swiglu, sms, &plan)) return false;
    *st = launch_skinny(a, plan, stream);
    if (*st == XCCL_OK) return true;
    (void)cudaGetLastError();   // refused: the large kernel serves the call, or says why not
    return false;
}

xccl_status_t launch_skinny(const SkinnyArgs &a, const SkinnyPlan &plan, cudaStream_t stream)
{
    SkinnyMaps   maps{};
    SkinnyParams p{};
    p.M = a.M; p.N = a.N; p.K = a.K;
    p.ldc       = a.ldc;
    p.plan      = plan;
    p.sa        = a.sa;
    p.sb0       = a.sb0;
    p.sb1       = a.sb1;
    p.out_scale = a.out_scale;
    p.C         = a.C;
    p.error     = a.error != nullptr ? a.error : error_word();
    p.budget_ns = 4000000000ull;
    xccl_status_t st;
    auto map = [&](CUtensorMap *m, const void *base, int rows, int box) {
        return a.fp8 ? make_tensor_map_u8(m, base, (uint64_t)rows, (uint64_t)a.K, (uint32_t)box)
                     : make_tensor_map_2d(m, base, (uint64_t)rows, (uint64_t)a.K, (uint64_t)a.K, (uint32_t)box);
    };
    if ((st = map(&maps.a, a.A, a.M, plan.mn)) != XCCL_OK) return st;
    if ((st = map(&maps.b0, a.B0, a.N, 128)) != XCCL_OK) return st;
    if ((st = map(&maps.b1, a.swiglu ? a.B1 : a.B0, a.N, 128)) != XCCL_OK) return st;
    SkinnyKernel k = skinny_kernel_of(plan.mn, a.fp8, a.swiglu);
    int          dev = 0;
    XCCL_CUDA_CHECK(cudaGetDevice(&dev));
    if ((st = prepare_kernel(k, dev, a.fp8, a.swiglu, &p.plan)) != XCCL_OK) return st;
    cudaLaunchConfig_t  cfg;
    cudaLaunchAttribute attr[1];
    launch_config(p.plan, a.fp8, stream, &cfg, attr);
    XCCL_CUDA_CHECK(cudaLaunchKernelEx(&cfg, k, p, maps));
    return XCCL_OK;
}

}  // namespace tp
}  // namespace xccl

// Host-side view of the cluster that is launched (tests): `splits` CTAs are wanted, bit s of `fits` says that s are placed.
extern "C" int xccl_tp_skinny_cluster(int splits, unsigned fits)
{
    return xccl::tp::placeable(splits, [&](int s) { return (fits >> s & 1u) != 0; });
}

// Host-side view of the cut (tests): out = {mn, tiles, splits, kblocks, stages, nbuf, cols, tmem_cols, chunk, smem_bytes,
// CTAs per SM}. Returns the number of blocks of rows (here 1), 0 when the sizes are not for this kernel.
static int skinny_plan_out(bool rows, int M, int N, int K, bool fp8, bool swiglu, int sms, int *out)
{
    xccl::tp::SkinnyPlan q;
    if (out == nullptr || !(rows ? xccl::tp::skinny_plan_rows : xccl::tp::skinny_plan)(M, N, K, fp8, swiglu, sms, &q)) return 0;
    const int v[11] = {q.mn, q.tiles, q.splits, q.kblocks, q.stages, q.nbuf, q.cols, q.tmem_cols, q.chunk, q.smem_bytes,
                       xccl::tp::skinny_occupancy(q.mn, fp8, swiglu)};
    std::copy(v, v + 11, out);
    return q.blocks;
}
extern "C" int xccl_tp_skinny_plan(int M, int N, int K, int fp8, int swiglu, int sms, int *out)
{
    return skinny_plan_out(false, M, N, K, fp8 != 0, swiglu != 0, sms, out);
}
// The same for any number of rows: returns the number of blocks of rows, 0 when the large kernel serves the product.
extern "C" int xccl_tp_skinny_plan_rows(int M, int N, int K, int fp8, int swiglu, int sms, int *out)
{
    return skinny_plan_out(true, M, N, K, fp8 != 0, swiglu != 0, sms, out);
}
// Whether such a product runs in this kernel under the options of this process.
extern "C" int xccl_tp_skinny_takes(int M, int N, int K, int fp8, int swiglu, int sms)
{
    xccl::tp::SkinnyPlan q;
    return xccl::tp::takes(M, N, K, fp8 != 0, swiglu != 0, sms, &q) ? 1 : 0;
}
