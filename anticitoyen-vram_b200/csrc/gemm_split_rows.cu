// The 32-bit product of gemm_split_tc.cu for up to 16 tokens, and for few outputs: the same parts, the same products in the same order,
// on mma.sync, whose sums of 16 products are the tcgen05 unit's to the bit, so a row's result does not depend on how many rows
// there are.  No document says that the two units sum alike: it is measured, and the tests compare them over terms of all sizes, terms
// that cancel, sums that grow throughout, and operands at both ends of a float's range.
//
// What bounds it is the weights' stream.  Every lane brings its own operands by asynchronous copies into a ring of its
// own (four neighbouring k of a weight row; which k of a step of 16 a lane holds is the same for tokens and weights), so the
// ring's depth is under way at any time, no registers hold what is on its way and no barrier stands in the loop.  A warp takes
// one group of K (gf_group_length) for 8 R weight rows, which fill the tensor core's M; the groups of a row meet in shared
// memory.  A block goes on to its next rows with their first copies already under way.  Microseconds, multiply-adds on the
// CUDA cores (gemm_simt.cu) and now: 1, 4, 8 and 16 tokens 4096 x 1024 5.6, 6.2, 7.5, 8.9 -> 5.8, 5.7, 6.0, 7.3; 1024 x 3072 6.0,
// 7.7, 10.1, 12.3 -> 6.3, 6.3, 6.4, 9.4; 12288 x 2048 21.5, 28.6, 36.2, 40.9 -> 19.9, 21.9, 23.4, 31.8; 151936 x 1024 107, 125, 165, 235
// -> 96 (6.4 TB/s of weights), 98, 104, 152.  One token on few or long rows is what it makes more slowly: 1024 x 2048 4.6 -> 5.0,
// 2048 x 2048 5.5 -> 6.0, 2048 x 6144 12.1 -> 13.3, 512 x 4096 6.9 -> 8.1, 1024 x 12288 19 -> 22; and K just above 1024, whose groups are
// six (3000 x 1100, 2 tokens 6.1 -> 7.8).  Rows without 16-byte pieces, 50000 x 1026: 127, 128, 317, 317 ->
// 68, 71, 71, 86.
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

// R: octets of weight rows of a warp (1 or 2); H: octets of tokens; DEPTH: chunks of 32 k in a warp's ring; Q: chunks that are made side
// by side (a chunk is a chain of twelve products, each behind the one before it).  PARTS: the tokens' parts are made once and stay in
// shared memory (192 bytes a token and chunk), else the tokens' floats come through the ring and are taken apart for every tile.
template <int R, int H, int DEPTH, int Q, bool PARTS, bool PIECES>
__global__ void __launch_bounds__(GR_WARPS * 32, Q > 2 ? 1 : 2)
gemm_split_rows_kernel(const GfArgs p, int groups) {
    constexpr int ROWS = R + (PARTS ? 0 : H), CHUNK = 2 * ROWS * 512, COLS = 8 * R;     // CHUNK: two steps' rows, a lane's 16 bytes side by side
    extern __shared__ __align__(16) unsigned char ring[];
    __shared__ float part[2][GR_WARPS][8 * H][COLS + 1];
    const int group = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;      // (a warp to a group)
    const int m0 = blockIdx.y * 8 * H, M = min(p.M - m0, 8 * H);        // the block's tokens
    const float* A = p.A + (size_t)blockIdx.z * p.a_batch + (size_t)m0 * p.lda;
    const float* W = p.W + (size_t)blockIdx.z * p.w_batch;
    float* C = p.C + (size_t)blockIdx.z * p.c_batch + (size_t)m0 * p.ldc;
    const float* gate = p.gate ? p.gate + (size_t)blockIdx.z * p.g_batch + (size_t)m0 * p.ldg : nullptr;
    bool again = false;
    const int gl = gf_group_length(p.K), k_begin = group * gl, mine = group < groups ? min(gl, p.K - k_begin) : 0;
    const int chunks = (mine + 31) / 32, tiles = (p.N + COLS - 1) / COLS;
    const uint32_t own = smem_u32(ring) + group * (DEPTH * CHUNK) + lane * 16;
    const float* wr[R];
    const float* ar[H];
    int next_tile = blockIdx.x, next = 0, into = 0;         // the chunk that is asked for next, and its place in the ring
    auto rows = [&]() {         // weight rows that do not exist: the last one that does (their outputs go nowhere); tokens: zeros
#pragma unroll
        for (int r = 0; r < R; ++r) wr[r] = W + (size_t)min(next_tile * COLS + r * 8 + g, p.N - 1) * p.ldw + k_begin + tq * 4;
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
                for (int r = 0; r < R; ++r) copy(dst + (e * ROWS + r) * 512, wr[r] + e * 16, left);
                if constexpr (!PARTS) {
#pragma unroll
                    for (int h = 0; h < H; ++h) copy(dst + (e * ROWS + R + h) * 512, ar[h] + e * 16, h * 8 + g < M ? left : 0);
                }
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
    // the tokens' parts: of each chunk and token, of each four lanes' k, the parts of the first and of the second step (a lane's 48 bytes)
    const uint32_t parts_at = smem_u32(ring) + GR_WARPS * DEPTH * CHUNK + group * (gl / 32) * M * 192;
    pdl_wait();
    if (chunks) {
        rows();
#pragma unroll
        for (int i = 0; i < DEPTH - Q; ++i) ask();
        if constexpr (PARTS) {
#pragma unroll 4
            for (int i = lane; i < chunks * M * 8; i += 32) {
                const int q = i & 3, e = i >> 2 & 1, m = (i >> 3) % M, c = (i >> 3) / M, k = c * 32 + e * 16 + q * 4;
                const float* src = A + (size_t)m * p.lda + k_begin + k;
                float4 v;
                if (PIECES && k + 4 <= mine) {
                    v = *reinterpret_cast<const float4*>(src);
                } else {
                    v.x = k < mine ? src[0] : 0.f;
                    v.y = k + 1 < mine ? src[1] : 0.f;
                    v.z = k + 2 < mine ? src[2] : 0.f;
                    v.w = k + 3 < mine ? src[3] : 0.f;
                }
                uint32_t h[3][2];
                gr_parts(v.x, v.y, h[0][0], h[1][0], h[2][0]);
                gr_parts(v.z, v.w, h[0][1], h[1][1], h[2][1]);
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(parts_at + ((c * M + m) * 4 + q) * 48 + e * 24 + j * 8), "r"(h[j][0]), "r"(h[j][1]) : "memory");
            }
            __syncwarp();
        }
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
            for (int n = 0; n < chunks; n += Q) {
                cp_async_wait<DEPTH - 2 * Q>();         // (a lane reads what it brought itself)
                uint32_t w[Q][2][3][4], t[Q][2][3][H][2];       // weights: (g, low k) (g + 8, low) (g, high) (g + 8, high)
#pragma unroll
                for (int z = 0; z < Q; ++z) {           // (chunks behind the last are made of what there is and not added)
                    const uint32_t src = own + from * CHUNK;
                    if (n + z < chunks) from = from + 1 == DEPTH ? 0 : from + 1;
                    auto read = [&](int at) {
                        float4 v;
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(src + at * 512) : "memory");
                        return v;
                    };
                    if constexpr (PARTS) {
#pragma unroll
                        for (int h = 0; h < H; ++h) {
                            uint32_t u[12];
#pragma unroll
                            for (int j = 0; j < 12; ++j) u[j] = 0;
                            if (h * 8 + g < M && n + z < chunks) {
                                const uint32_t at = parts_at + (((n + z) * M + h * 8 + g) * 4 + tq) * 48;
#pragma unroll
                                for (int j = 0; j < 3; ++j)
                                    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                                                 : "=r"(u[4 * j]), "=r"(u[4 * j + 1]), "=r"(u[4 * j + 2]), "=r"(u[4 * j + 3]) : "r"(at + j * 16));
                            }
#pragma unroll
                            for (int e = 0; e < 2; ++e)
#pragma unroll
                                for (int q = 0; q < 3; ++q)
#pragma unroll
                                    for (int i = 0; i < 2; ++i) t[z][e][q][h][i] = u[e * 6 + q * 2 + i];
                        }
                    }
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const float4 v = read(e * ROWS + r);
                            gr_parts(v.x, v.y, w[z][e][0][r], w[z][e][1][r], w[z][e][2][r]);
                            gr_parts(v.z, v.w, w[z][e][0][2 + r], w[z][e][1][2 + r], w[z][e][2][2 + r]);
                        }
                        if constexpr (R == 1) {
#pragma unroll
                            for (int q = 0; q < 3; ++q) w[z][e][q][1] = w[z][e][q][3] = 0;
                        }
                        if constexpr (!PARTS) {
#pragma unroll
                            for (int h = 0; h < H; ++h) {
                                const float4 v = read(e * ROWS + R + h);
                                gr_parts(v.x, v.y, t[z][e][0][h][0], t[z][e][1][h][0], t[z][e][2][h][0]);
                                gr_parts(v.z, v.w, t[z][e][0][h][1], t[z][e][1][h][1], t[z][e][2][h][1]);
                            }
                        }
                    }
                }
#pragma unroll
                for (int z = 0; z < Q; ++z)
                    if (n + z < chunks) ask();          // (into the places that were read in the turn before this one)
                float c[Q][H][4];
#pragma unroll
                for (int z = 0; z < Q; ++z)
#pragma unroll
                    for (int h = 0; h < H; ++h)
#pragma unroll
                        for (int i = 0; i < 4; ++i) c[z][h][i] = 0.f;
                auto product = [&](int e, int pt, int pw) {
#pragma unroll
                    for (int z = 0; z < Q; ++z)
#pragma unroll
                        for (int h = 0; h < H; ++h) gr_mma(c[z][h], w[z][e][pw], t[z][e][pt][h][0], t[z][e][pt][h][1]);
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
                for (int z = 0; z < Q; ++z)
                    if (n + z < chunks) {
#pragma unroll
                        for (int h = 0; h < H; ++h)
#pragma unroll
                            for (int i = 0; i < 4; ++i) sum[h][i] += c[z][h][i];
                    }
            }
            // c: (row g, tokens 2 tq and the next), (row g + 8, the same)
#pragma unroll
            for (int h = 0; h < H; ++h)
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int e = 0; e < 2; ++e) part[turn][group][h * 8 + 2 * tq + e][r * 8 + g] = sum[h][2 * r + e];
        }
        __syncthreads();
        if (tile + (int)gridDim.x >= tiles) pdl_launch_dependents();
        // outputs: token by token, weight rows side by side
        for (int i = threadIdx.x; i < M * COLS; i += GR_WARPS * 32) {
            const int m = i / COLS, c = i - m * COLS, gn = tile * COLS + c;
            if (gn >= p.N) continue;
            float v[GF_GROUPS];
#pragma unroll
            for (int j = 0; j < GF_GROUPS; ++j) v[j] = j < groups ? part[turn][j][m][c] : 0.f;
            float x = v[0];
#pragma unroll
            for (int j = 1; j < GF_GROUPS; ++j)
                if (j < groups) x = x + v[j];
            const bool number = fabsf(x) <= 3.402823466e38f;
            again |= !number;
            x *= GF_SCALE_BACK;
            if (gate && number) x /= 1.f + expf(-gate[(size_t)m * p.ldg + gn]);
            C[(size_t)m * p.ldc + gn] = x;
        }
    }
    cp_async_wait<0>();
    if (!again) return;
    // this thread's outputs once more, those that are no finite number (a gate that is none leaves none again)
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x)
        for (int i = threadIdx.x; i < M * COLS; i += GR_WARPS * 32) {
            const int m = i / COLS, gn = tile * COLS + i - m * COLS;
            if (gn >= p.N) continue;
            float x = C[(size_t)m * p.ldc + gn];
            if (fabsf(x) <= 3.402823466e38f) continue;
            x = gf_plain(A + (size_t)m * p.lda, W + (size_t)gn * p.ldw, p.K);
            if (gate) x /= 1.f + expf(-gate[(size_t)m * p.ldg + gn]);
            C[(size_t)m * p.ldc + gn] = x;
        }
}

// Shared memory of a block, and how many blocks of it an SM holds (of 228 KB, 1 KB of it the system's for each block; 200 KB where
// copies of four bytes go through what is left as its first-level cache).
template <int R, int H, int DEPTH, bool PARTS>
static int gr_smem(const GfArgs& p, int groups) {
    return GR_WARPS * DEPTH * 2 * (R + (PARTS ? 0 : H)) * 512 + (PARTS ? groups * (gf_group_length(p.K) / 32) * min(p.M, 8 * H) * 192 : 0);
}
template <int R, int H, int DEPTH, bool PARTS, bool PIECES>
static int gr_resident(const GfArgs& p, int groups) {
    return (PIECES ? 228 : 200) * 1024 / (gr_smem<R, H, DEPTH, PARTS>(p, groups) + 2 * GR_WARPS * 8 * H * (8 * R + 1) * 4 + 1024);
}

template <int R, int H, int DEPTH, int Q, bool PARTS, bool PIECES>
static int gr_launch(const GfArgs& p, int groups, int batches, int sms, cudaStream_t stream) {
    static_assert(DEPTH >= 2 * Q, "chunks are asked for while as many are made");
    const int smem = gr_smem<R, H, DEPTH, PARTS>(p, groups), resident = gr_resident<R, H, DEPTH, PARTS, PIECES>(p, groups);
    static AcvSmemConfig cfg;
    auto kernel = gemm_split_rows_kernel<R, H, DEPTH, Q, PARTS, PIECES>;
    if (const int e = acv_ensure_smem(cfg, kernel, smem)) return e;
    if (batches > 65535) return ACV_ERR_SIZE;
    const dim3 grid(min((p.N + 8 * R - 1) / (8 * R), max(1, min(resident, Q > 2 ? 1 : 2)) * sms), (p.M + 8 * H - 1) / (8 * H), batches);
    acv_launch(PDL_GEMM, kernel, grid, dim3(GR_WARPS * 32), smem, stream, p, groups);
    return acv_launch_status();
}

// Which way, all measured in microseconds.
// Few outputs: a block to eight weight rows and eight tokens, whatever the number of tokens, as long as each has an SM to itself (or
// shares one with one other, up to K = 4096; longer chains take longer than the tiles' kernel there), since what counts is how many
// chains run side by side.  64 tokens, tiles, and this: 64 x 1024 6.5, 2.9; 64 x 5120 16.2, 9.0; 256 x 1024 (256 blocks) 6.9, 4.4,
// 256 x 5120 16.7, 17.7; 16 tokens 1024 x 2048 (256 blocks) sixteen tokens to a block 6.9, eight 7.8.  A block that has its SM to
// itself makes chunks side by side, as it waits for its chains: by threes (1 token 1024 x 3072 one by one 6.7, by twos 6.5, by threes
// 6.3), by twos where a group is four chunks (8 tokens 256 x 1024 3.4, 2.9).
// Sixteen weight rows to a warp otherwise (2048 x 2048, 128 blocks, 6.0, with eight rows 7.6).
// The tokens' parts made once pay where a block meets enough tiles with them, the more tokens the more of them, and two blocks still
// fit an SM (1, 4, 8 tokens, through the ring and made once: 4096 x 1024 5.6, 5.9, 6.0 and 5.7, 6.0, 6.8; 12288 x 2048 22.9, 23.0 and 19.9,
// 21.7 (8 do not fit); 151936 x 1024 119, 119, 123 and 96, 98, 104; 16 tokens, one block to an SM, 174 and 152, 6144 x 1024 9.7 and 11.4),
// and wherever they fit for rows that come float by float (4096 x 1025, 1, 4, 8, 16 tokens 12.9, 14.0, 15.7, 19.0 and 8.9, 9.8, 10.2,
// 13.0).  One token on few long rows: made once and by twos (2048 x 6144 14.0 -> 13.3).
static long long gr_octets(const GfArgs& p, int batches) { return (long long)((p.N + 7) / 8) * ((p.M + 7) / 8) * batches; }
bool gr_takes(const GfArgs& p, int batches, int sms) { return p.M <= 16 || gr_octets(p, batches) <= (p.K <= 4096 ? 2 : 1) * sms; }

template <bool PIECES>
static int gr_run_as(const GfArgs& p, int batches, int sms, cudaStream_t stream) {
    const int gl = gf_group_length(p.K), groups = (p.K + gl - 1) / gl;
    const long long tiles = (long long)((p.N + 15) / 16) * batches, octets = gr_octets(p, batches);
    if (octets <= sms && gl > 128) return gr_launch<1, 1, 9, 3, false, PIECES>(p, groups, batches, sms, stream);
    if (octets <= sms || p.M > 16) return gr_launch<1, 1, 6, 2, false, PIECES>(p, groups, batches, sms, stream);
    if (p.M > 8) {
        if (tiles * 2 <= sms) return gr_launch<1, 2, 4, 1, false, PIECES>(p, groups, batches, sms, stream);
        if ((!PIECES || tiles >= 12LL * sms) && gr_resident<2, 2, 4, true, PIECES>(p, groups) >= 1)
            return gr_launch<2, 2, 4, 1, true, PIECES>(p, groups, batches, sms, stream);
        return gr_launch<2, 2, 3, 1, false, PIECES>(p, groups, batches, sms, stream);
    }
    if (!PIECES || 2 * tiles >= (2LL + p.M) * sms) {
        if (PIECES && gr_resident<2, 1, 4, true, PIECES>(p, groups) >= 2) return gr_launch<2, 1, 4, 1, true, PIECES>(p, groups, batches, sms, stream);
        if (gr_resident<2, 1, 3, true, PIECES>(p, groups) >= 2) return gr_launch<2, 1, 3, 1, true, PIECES>(p, groups, batches, sms, stream);
        if (!PIECES && gr_resident<2, 1, 4, true, PIECES>(p, groups) >= 1) return gr_launch<2, 1, 4, 1, true, PIECES>(p, groups, batches, sms, stream);
    }
    if (PIECES && p.M == 1 && p.K >= 4096 && tiles <= sms && gr_resident<2, 1, 6, true, PIECES>(p, groups) >= 1)
        return gr_launch<2, 1, 6, 2, true, PIECES>(p, groups, batches, sms, stream);
    return gr_launch<2, 1, 4, 1, false, PIECES>(p, groups, batches, sms, stream);
}

int gr_run(const GfArgs& p, bool pieces, int batches, int sms, cudaStream_t stream) {
    return pieces ? gr_run_as<true>(p, batches, sms, stream) : gr_run_as<false>(p, batches, sms, stream);
}
