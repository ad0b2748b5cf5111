// The 32-bit product on the tensor cores, what its two kernels (gemm_split_tc.cu, gemm_split_rows.cu) and gemm_simt.cu share.
#pragma once

#include "common.cuh"

// Shorter sums stay on the CUDA cores (K 256, 3 and 300 tokens of 256 columns: 2.6 and 6.5 us there, 3.5 and 9.1 here; from
// 1024 on faster here but for one token, see gemm_split_rows.cu).  A property of K alone, as the order of a sum has to be.
#define GF_MIN_K 1024
#define GF_BK 64            // groups are multiples of it
#define GF_GROUPS 8

// Operands are multiplied by 2^24 before they are taken apart and sums by 2^-48 at the end, which changes no bit of either (a
// result below 2^-126 is rounded, once): a float's lowest bit lies 2^-23 below its first, under the smallest bfloat16 for floats
// below 2^-110 (relative error of the parts at 1e-34 and 1e-37: 3e-7 and 3e-4); scaled, all parts of all floats are bfloat16
// values, and normal ones but for those of floats that are subnormal themselves.  What the scale takes out of a float's range,
// operands from 2^104 and sums from 2^80 on, comes out as no finite number and is made by gf_plain.
#define GF_SCALE 16777216.f
#define GF_SCALE_BACK 3.552713678800501e-15f

struct GfArgs {
    const float *A, *W, *gate;
    float* C;
    int* status;
    int lda, ldw, ldc, ldg, M, N, K;
    long long a_batch, w_batch, c_batch, g_batch;
};

// (K from GF_MIN_K on: six to eight groups)
__host__ __device__ __forceinline__ int gf_group_length(int K) { return ((K + GF_GROUPS - 1) / GF_GROUPS + GF_BK - 1) / GF_BK * GF_BK; }

// (a, b) minus the pair of bfloat16 values packed in h
__device__ __forceinline__ void gf_less(float& a, float& b, uint32_t h) {
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tsub.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "+f"(a), "+f"(b) : "f"(__uint_as_float(h << 16)), "f"(__uint_as_float(h & 0xffff0000u)));
}

__device__ __forceinline__ void gf_scale(float& a, float& b) {
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %2};\n\tmul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "+f"(a), "+f"(b) : "f"(GF_SCALE));
}

// an output by itself, in the order of gemm_simt.cu
static __device__ __noinline__ float gf_plain(const float* a, const float* w, int K) {
    const int gl = ((K + 7) / 8 + 31) / 32 * 32;
    float g[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float s = 0.f;
        for (int k = i * gl; k < min(K, (i + 1) * gl); ++k) s = fmaf(a[k], w[k], s);
        g[i] = s;
    }
    return ((g[0] + g[1]) + (g[2] + g[3])) + ((g[4] + g[5]) + (g[6] + g[7]));
}

int gf_run(const GfArgs& p, bool pieces, int batches, int sms, cudaStream_t stream);
// the kernel for few tokens or few outputs, and whether it is the one for these
int gr_run(const GfArgs& p, bool pieces, int batches, int sms, cudaStream_t stream);
bool gr_takes(const GfArgs& p, int batches, int sms);
