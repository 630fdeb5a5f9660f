// GEMM for few rows of activations (decoding; more rows where the large kernel's tiles would leave the chip idle): C[M,N] =
// A[M,K] * B[N,K]^T in blocks of up to kSkinnyMaxM rows, plain or SwiGLU, bf16 or
// block-scaled fp8 (same operands, scales and rounding as the kernels of tp_gemm.cuh). Implemented in tp_skinny.cu.
#pragma once
#include <cuda_runtime.h>

#include "xccl/xccl.h"

namespace xccl {
namespace tp {

constexpr int kSkinnyMaxM = 128;

struct SkinnyArgs {
    int M, N, K;              // N: rows of B0 (and of B1 with SwiGLU) = output columns
    bool fp8, swiglu;
    const void *A, *B0, *B1;  // B1: the "up" weights
    void       *C;
    int         ldc;
    const float *sa, *sb0, *sb1;  // fp8: scales as in xccl_gemm_fp8_blockscaled
    float      *out_scale;    // fp8 SwiGLU: non-null = C is e4m3, quantised per row and 128 columns
    uint32_t   *error;        // device word, 0 = fine
};

// How a launch is cut up (a pure function of the sizes; the tests walk it on the CPU).
struct SkinnyPlan {
    int mn;        // columns of the MMA: rows of a block rounded up
    int blocks;    // blocks of rows (each up to kSkinnyMaxM)
    int tiles;     // blocks of 128 weight rows
    int splits;    // CTAs of a cluster that share the K blocks of a tile
    int kblocks;
    int stages;    // of the TMA ring
    int nbuf;      // fp8: product buffers in tensor memory
    int cols;      // tensor-memory columns of one accumulator or product (gate and up side by side)
    int tmem_cols;
    int chunk;     // tokens per round of the final reduction
    int smem_bytes;
};
// False when the sizes are not for this kernel (the callers then use launch_gemm / launch_gemm_fp8).
bool          skinny_plan(int M, int N, int K, bool fp8, bool swiglu, int sms, SkinnyPlan *plan);
// The same for any number of rows (blocks of them): false also where the large kernel is the faster one.
bool          skinny_plan_rows(int M, int N, int K, bool fp8, bool swiglu, int sms, SkinnyPlan *plan);
// Runs the product here when its sizes are for this kernel and the device takes the launch (true); otherwise nothing has
// been launched and the caller's large kernel serves it.
bool          try_skinny(const SkinnyArgs &a, cudaStream_t stream, xccl_status_t *st);
xccl_status_t launch_skinny(const SkinnyArgs &a, const SkinnyPlan &plan, cudaStream_t stream);

}  // namespace tp
}  // namespace xccl
