// The inner loop of the bfloat16 products of a few rows (gemm_rows.cu, moe_rows.cu): a warp's chunks of 64 k, R octets of weight rows
// by H octets of tokens, in a ring in shared memory of which a lane reads what it brought itself.
#pragma once

#include "mma_tiles.cuh"

#define RR_WARPS 8          // of a block, each with an eighth of K

// A chunk holds two blocks of 32 k; of each the weights' octets, then the tokens', 512 bytes an octet, a lane's 16 bytes side by side.
template <int R, int H>
struct RrChunk {
    static constexpr int BYTES = 2 * (R + H) * 512;
    uint4 w[2][R], x[2][H];
    static __device__ __forceinline__ uint32_t weights_at(uint32_t lane_base, int b, int r) { return lane_base + (b * (R + H) + r) * 512; }
    static __device__ __forceinline__ uint32_t tokens_at(uint32_t lane_base, int b, int h) { return lane_base + (b * (R + H) + R + h) * 512; }
    __device__ __forceinline__ void read(uint32_t lane_base) {
        auto at = [](uint32_t src) {
            uint4 v;
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(src) : "memory");
            return v;
        };
#pragma unroll
        for (int b = 0; b < 2; ++b) {
#pragma unroll
            for (int r = 0; r < R; ++r) w[b][r] = at(weights_at(lane_base, b, r));
#pragma unroll
            for (int h = 0; h < H; ++h) x[b][h] = at(tokens_at(lane_base, b, h));
        }
    }
};

// The sums of a warp's rows and tokens, in two chains: of c[..][h], (row g, tokens 2 tq and the next), (row g + 8, the same).
template <int R, int H>
struct RrSums {
    float c[2][R / 2][H][4];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int a = 0; a < R / 2; ++a)
#pragma unroll
                for (int h = 0; h < H; ++h)
#pragma unroll
                    for (int i = 0; i < 4; ++i) c[j][a][h][i] = 0.f;
    }
    __device__ __forceinline__ void add(const RrChunk<R, H>& k) {
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int a = 0; a < R / 2; ++a) {
                const uint4 lo = k.w[b][2 * a], hi = k.w[b][2 * a + 1];
                const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
                for (int h = 0; h < H; ++h) {
                    mma_bf16(c[0][a][h], a0, k.x[b][h].x, k.x[b][h].y);
                    mma_bf16(c[1][a][h], a1, k.x[b][h].z, k.x[b][h].w);
                }
            }
    }
    // into the block's parts, [turn][warp][token][row]
    template <int STRIDE>
    __device__ __forceinline__ void leave(float (&part)[2][RR_WARPS][8 * H][STRIDE], int turn, int warp, int g, int tq) const {
#pragma unroll
        for (int h = 0; h < H; ++h)
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    part[turn][warp][h * 8 + 2 * tq + e][r * 8 + g] = c[0][r / 2][h][2 * (r & 1) + e] + c[1][r / 2][h][2 * (r & 1) + e];
    }
};

// the warps' sums of a token and a row
template <int TOKENS, int STRIDE>
__device__ __forceinline__ float rr_sum(const float (&part)[RR_WARPS][TOKENS][STRIDE], int m, int q) {
    float v = 0.f;
#pragma unroll
    for (int j = 0; j < RR_WARPS; ++j) v += part[j][m][q];
    return v;
}
