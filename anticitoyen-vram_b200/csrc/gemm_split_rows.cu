// The 32-bit product of gemm_split_tc.cu for up to 16 tokens: the same parts, the same products in the same order, on
// mma.sync, whose sums of 16 products are the tcgen05 unit's to the bit (the tests compare the two), so a row's result does not
// depend on how many rows there are.
//
// What bounds it is the weights' stream.  Every lane brings its own operands by 16-byte asynchronous copies into a ring of its
// own (four neighbouring k of a weight row; which k of a step of 16 a lane holds is the same for tokens and weights), so the
// ring's depth is under way at any time, no registers hold what is on its way and no barrier stands in the loop.  A warp takes
// one group of K (gf_group_length) for 8 R weight rows, which fill the tensor core's M; the groups of a row meet in shared
// memory.  A block goes on to its next rows with their first copies already under way.  Microseconds, multiply-adds on the
// CUDA cores (gemm_simt.cu) and now: 1, 3, 8 and 16 tokens 4096 x 1024 5.6, 6.3, 8.0, 9.8 -> 5.8, 5.9, 6.0, 7.7; 1024 x 3072 6.3,
// 7.8, 10.3, 12.6 -> 7.0, 7.0, 7.0, 10.9; 151936 x 1024 108, 124, 166, 235 -> 119, 119, 120 (5.2 TB/s of weights), 174.
#include "mma_tiles.cuh"
#include "gemm_split_tc.h"

#define GR_WARPS 8

// two floats into three pairs of bfloat16, each the rounding of what is left
__device__ __forceinline__ void gr_parts(float a, float b, uint32_t& h1, uint32_t& h2, uint32_t& h3) {
    gf_scale(a, b);
    h1 = pack_bf16(a, b);
    gf_less(a, b, h1);
    h2 = pack_bf16(a, b);
    gf_less(a, b, h2);
    h3 = pack_bf16(a, b);
}

// (not volatile: the products of one chunk may come between those of another)
__device__ __forceinline__ void gr_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// R: octets of weight rows of a warp (1 or 2); H: octets of tokens; DEPTH: chunks of 32 k in a warp's ring
template <int R, int H, int DEPTH, bool PIECES>
__global__ void __launch_bounds__(GR_WARPS * 32, 2)
gemm_split_rows_kernel(const GfArgs p, int groups, int slots) {
    constexpr int CHUNK = 2 * (R + H) * 512;        // bytes: two steps' rows, a lane's 16 bytes side by side
    extern __shared__ __align__(16) unsigned char ring[];
    __shared__ float part[2][GR_WARPS][8 * H][8 * R + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    // slots: `groups` rounded up to a power of two; GR_WARPS / slots rows' tiles side by side
    const int group = warp % slots, set = warp / slots, sets = GR_WARPS / slots, cols = sets * 8 * R, tokens = min(p.M, 8 * H);
    const float* A = p.A + (size_t)blockIdx.z * p.a_batch;
    const float* W = p.W + (size_t)blockIdx.z * p.w_batch;
    float* C = p.C + (size_t)blockIdx.z * p.c_batch;
    const float* gate = p.gate ? p.gate + (size_t)blockIdx.z * p.g_batch : nullptr;
    bool again = gate != nullptr;
    const int gl = gf_group_length(p.K), k_begin = group * gl, mine = group < groups ? min(gl, p.K - k_begin) : 0;
    const int chunks = (mine + 31) / 32, tiles = (p.N + cols - 1) / cols;
    const uint32_t own = smem_u32(ring) + warp * (DEPTH * CHUNK) + lane * 16;
    const float* wr[R];
    const float* ar[H];
    int next_tile = blockIdx.x, next = 0, into = 0;         // the chunk that is asked for next, and its place in the ring
    auto rows = [&]() {         // weight rows that do not exist: the last one that does (their outputs go nowhere); tokens: zeros
#pragma unroll
        for (int r = 0; r < R; ++r) wr[r] = W + (size_t)min(next_tile * cols + (set * R + r) * 8 + g, p.N - 1) * p.ldw + k_begin + tq * 4;
#pragma unroll
        for (int h = 0; h < H; ++h) ar[h] = A + (size_t)(h * 8 + g) * p.lda + k_begin + tq * 4;
    };
    auto copy = [&](uint32_t dst, const float* src, int left) {        // (zeros behind K's end)
        if constexpr (PIECES) {
            const int bytes = left >= 4 ? 16 : left > 0 ? left * 4 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(bytes ? src : W), "r"(bytes) : "memory");
        } else {            // (rows without 16-byte pieces: float by float)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * i), "l"(i < left ? src + i : W), "r"(i < left ? 4 : 0) : "memory");
        }
    };
    auto ask = [&]() {
        if (next_tile < tiles) {
            const uint32_t dst = own + into * CHUNK;
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int left = mine - next * 32 - e * 16 - tq * 4;
#pragma unroll
                for (int r = 0; r < R; ++r) copy(dst + (e * (R + H) + r) * 512, wr[r] + e * 16, left);
#pragma unroll
                for (int h = 0; h < H; ++h) copy(dst + (e * (R + H) + R + h) * 512, ar[h] + e * 16, h * 8 + g < p.M ? left : 0);
            }
            into = into + 1 == DEPTH ? 0 : into + 1;
            if (++next == chunks) {
                next = 0;
                next_tile += gridDim.x;
                rows();
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) wr[r] += 32;
#pragma unroll
                for (int h = 0; h < H; ++h) ar[h] += 32;
            }
        }
        cp_async_commit();
    };
    pdl_wait();
    if (chunks) {
        rows();
#pragma unroll
        for (int i = 0; i < DEPTH - 1; ++i) ask();
    }
    int from = 0;
    for (int tile = blockIdx.x, turn = 0; tile < tiles; tile += gridDim.x, turn ^= 1) {
        if (chunks) {
            float sum[H][4];
#pragma unroll
            for (int h = 0; h < H; ++h)
#pragma unroll
                for (int i = 0; i < 4; ++i) sum[h][i] = 0.f;
#pragma unroll 1
            for (int n = 0; n < chunks; ++n) {
                cp_async_wait<DEPTH - 2>();         // (a lane reads what it brought itself)
                const uint32_t src = own + from * CHUNK;
                from = from + 1 == DEPTH ? 0 : from + 1;
                auto read = [&](int at) {
                    float4 v;
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(src + at * 512) : "memory");
                    return v;
                };
                uint32_t w[2][3][4], t[2][3][H][2];             // weights: (g, low k) (g + 8, low) (g, high) (g + 8, high)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float4 v = read(e * (R + H) + r);
                        gr_parts(v.x, v.y, w[e][0][r], w[e][1][r], w[e][2][r]);
                        gr_parts(v.z, v.w, w[e][0][2 + r], w[e][1][2 + r], w[e][2][2 + r]);
                    }
                    if constexpr (R == 1) {
#pragma unroll
                        for (int q = 0; q < 3; ++q) w[e][q][1] = w[e][q][3] = 0;
                    }
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        const float4 v = read(e * (R + H) + R + h);
                        gr_parts(v.x, v.y, t[e][0][h][0], t[e][1][h][0], t[e][2][h][0]);
                        gr_parts(v.z, v.w, t[e][0][h][1], t[e][1][h][1], t[e][2][h][1]);
                    }
                }
                ask();                              // (into the place that was read in the turn before this one)
                float c[H][4];
#pragma unroll
                for (int h = 0; h < H; ++h)
#pragma unroll
                    for (int i = 0; i < 4; ++i) c[h][i] = 0.f;
                auto product = [&](int e, int pt, int pw) {
#pragma unroll
                    for (int h = 0; h < H; ++h) gr_mma(c[h], w[e][pw], t[e][pt][h][0], t[e][pt][h][1]);
                };
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    product(e, 1, 0);
                    product(e, 0, 1);
                    product(e, 2, 0);
                    product(e, 1, 1);
                    product(e, 0, 2);
                }
                product(0, 0, 0);
                product(1, 0, 0);
#pragma unroll
                for (int h = 0; h < H; ++h)
#pragma unroll
                    for (int i = 0; i < 4; ++i) sum[h][i] += c[h][i];
            }
            // c: (row g, tokens 2 tq and the next), (row g + 8, the same)
#pragma unroll
            for (int h = 0; h < H; ++h)
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int e = 0; e < 2; ++e) part[turn][warp][h * 8 + 2 * tq + e][r * 8 + g] = sum[h][2 * r + e];
        }
        __syncthreads();
        if (tile + (int)gridDim.x >= tiles) pdl_launch_dependents();
        // outputs: token by token, weight rows side by side
        for (int i = threadIdx.x; i < tokens * cols; i += GR_WARPS * 32) {
            const int m = i / cols, c = i - m * cols, q = c / (8 * R), gn = tile * cols + c;
            if (gn >= p.N) continue;
            float v[GF_GROUPS];
#pragma unroll
            for (int j = 0; j < GF_GROUPS; ++j) v[j] = j < groups ? part[turn][q * slots + j][m][c - q * 8 * R] : 0.f;
            float x = v[0];
#pragma unroll
            for (int j = 1; j < GF_GROUPS; ++j)
                if (j < groups) x = x + v[j];
            again |= !(fabsf(x) <= 3.402823466e38f);
            C[(size_t)m * p.ldc + gn] = x * GF_SCALE_BACK;
        }
    }
    cp_async_wait<0>();
    if (!again) return;
    // this thread's outputs once more: a gate, or one that is no finite number
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x)
        for (int i = threadIdx.x; i < tokens * cols; i += GR_WARPS * 32) {
            const int m = i / cols, gn = tile * cols + i - m * cols;
            if (gn >= p.N) continue;
            float x = C[(size_t)m * p.ldc + gn];
            if (!(fabsf(x) <= 3.402823466e38f)) x = gf_plain(A + (size_t)m * p.lda, W + (size_t)gn * p.ldw, p.K);
            if (gate) x /= 1.f + expf(-gate[(size_t)m * p.ldg + gn]);
            C[(size_t)m * p.ldc + gn] = x;
        }
}

template <int R, int H, int DEPTH, bool PIECES>
static int gr_launch(const GfArgs& p, int groups, int batches, int sms, cudaStream_t stream) {
    constexpr int smem = GR_WARPS * DEPTH * 2 * (R + H) * 512;
    static AcvSmemConfig cfg;
    auto kernel = gemm_split_rows_kernel<R, H, DEPTH, PIECES>;
    if (const int e = acv_ensure_smem(cfg, kernel, smem)) return e;
    int slots = 1;
    while (slots < groups) slots *= 2;
    const int rows = GR_WARPS / slots * 8 * R;
    const dim3 grid(min((p.N + rows - 1) / rows, 2 * sms), 1, batches);
    if (batches > 65535) return ACV_ERR_SIZE;
    acv_launch(PDL_GEMM, kernel, grid, dim3(GR_WARPS * 32), smem, stream, p, groups, slots);
    return acv_launch_status();
}

int gr_run(const GfArgs& p, bool pieces, int batches, int sms, cudaStream_t stream) {
    const int gl = gf_group_length(p.K), groups = (p.K + gl - 1) / gl;
    // eight weight rows to a warp where sixteen would leave half of the SMs without a block (1024 x 3072 8.0 -> 7.0 us; 2048 x 2048,
    // 128 blocks of sixteen, 6.2 and 8.0)
    int slots = 1;
    while (slots < groups) slots *= 2;
    const int rows = GR_WARPS / slots * 16;
    const bool few = (long long)((p.N + rows - 1) / rows) * batches * 2 <= sms;
#define GR_CASE(RR, HH, DD) \
    return pieces ? gr_launch<RR, HH, DD, true>(p, groups, batches, sms, stream) : gr_launch<RR, HH, DD, false>(p, groups, batches, sms, stream)
    if (p.M > 8) {
        if (few) GR_CASE(1, 2, 4);
        GR_CASE(2, 2, 3);
    }
    if (few) GR_CASE(1, 1, 6);
    GR_CASE(2, 1, 4);
#undef GR_CASE
}
