// Pieces shared by the warm-start network's GEMM kernels.
#pragma once

#include <cuda_bf16.h>

#include "pg_internal.cuh"

namespace pg {

// C[m, n] = A B + bias with element (m, k) of A at a[m * sam + k * sak],
// (k, n) of B at b[k * sbk + n * sbn].
struct GemmArgs {
    const __nv_bfloat16 *a;
    int64_t sam, sak;
    const __nv_bfloat16 *b;
    int64_t sbk, sbn;
    int m, n, k;
    const float *bias;         // [n] or nullptr
    int epilogue;              // PG_MLP_EPI_* flags
    const float *zin;          // pre-activations for the GELU backward, [m, ldz]
    float *zout;               // pre-activations written by the forward, [m, ldz]
    int64_t ldz;
    __nv_bfloat16 *c;          // bf16 output [m, ldc] or nullptr
    float *cf;                 // fp32 output [m, ldc] or nullptr
    int64_t ldc;
    float beta;                // fp32 output: cf = acc + beta * cf
};

// Launches the tensor-core tile GEMM (pg_mlp_train.cu); PG_ERR_UNSUPPORTED,
// with nothing launched, for operands it does not cover.
int launch_mlp_gemm_tile(const GemmArgs &g, cudaStream_t stream);

namespace {

__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 lo, __nv_bfloat16 hi) {
    uint32_t l = (uint32_t)__bfloat16_as_ushort(lo);
    uint32_t h = (uint32_t)__bfloat16_as_ushort(hi);
    return l | (h << 16);
}

__device__ __forceinline__ void mma_bf16(float d[4], const uint32_t a[4], const uint32_t b[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ float gelu(float x) {
    return 0.5f * x * (1.f + erff(x * 0.70710678118654752f));
}

__device__ __forceinline__ float gelu_grad(float x) {
    const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

}  // namespace
}  // namespace pg
