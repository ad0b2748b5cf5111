// The experts' products where an expert has a few rows: C[r] = W_e x_r for the rows r that the grouping gave to expert e, in tiles
// of eight or sixteen rows of one expert each.
//
// What bounds them is the stream of the chosen experts' weights, and the tiled form (moe.cu: 64 columns to a block, K walked
// through three stages behind a barrier each, a new block for every tile) draws 5.1 to 5.5 TB/s.  Here blocks stay and walk over
// (tile, columns) as gemm_rows.cu walks over columns (the inner loop is shared, rows_ring.cuh): eight warps take an eighth of K each, a lane brings its own operands
// by 16-byte copies into a ring of its own, and the next columns' first copies are under way before the sums of these meet.
// A layer of 64 experts of 1024 at width 4096, six choices, microseconds, the tiled form and now: 1 token 102 -> 57, 16 tokens 273 -> 229,
// 64 tokens 360 -> 302; 32 experts of 768 at width 2048, four choices: 1 token 61 -> 29, 16 tokens 86 -> 70.
#include "rows_ring.cuh"
#include "moe_act.cuh"

#define MX_TILES 512        // tiles, and rows in them, that a block keeps the list of
#define MX_ROWS 2048

struct MoeRowsParams {
    const bf16 *x, *w;
    void* out;
    long long w_expert;
    int ldx, ldw, ldo, top, N, K, which, pairs;         // which: 0 gated pair, 1 plain (out float), 2 plain activation, as acv_moe_gemm_mma
    float limit, alpha, shift;
    const int *grouped, *tile_expert, *tiles_used;
    const float* row_weight;
};

// H: octets of rows of a tile; DEPTH: chunks of 64 k in a warp's ring.  A block's 32 weight rows are 32 outputs, or the gate and the
// up rows of sixteen.
template <int H, int DEPTH, bool GLU>
__global__ void __launch_bounds__(RR_WARPS * 32, 1)
moe_rows_kernel(const MoeRowsParams p) {
    constexpr int R = 4, COLS = GLU ? 16 : 32, ROWS = 8 * H;
    using Chunk = RrChunk<R, H>;
    constexpr int CHUNK = Chunk::BYTES;
    extern __shared__ __align__(16) unsigned char ring[];
    __shared__ float part[2][RR_WARPS][ROWS][36];
    __shared__ int experts[MX_TILES], rows[MX_ROWS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    pdl_launch_dependents();
    pdl_wait();
    const int used = *p.tiles_used;
    for (int i = threadIdx.x; i < used; i += RR_WARPS * 32) experts[i] = p.tile_expert[i];
    for (int i = threadIdx.x; i < used * ROWS; i += RR_WARPS * 32) rows[i] = p.grouped[i];
    __syncthreads();
    const int all = p.K / 64, across = p.N / COLS, items = used * across;
    const int c0 = all * warp / RR_WARPS, chunks = all * (warp + 1) / RR_WARPS - c0;       // this warp's chunks of K
    const uint32_t own = smem_u32(ring) + warp * (DEPTH * CHUNK) + lane * 16;
    const int step_u = GLU ? (p.pairs ? 1 : p.N) : 16;          // from octets 0, 1 to octets 2, 3: the up rows, or the next sixteen
    const int step_n = GLU && p.pairs ? 2 : 1;                  // from an output's weight row to the next one's
    const bf16 *wr = nullptr, *xr[H];
    int next_item = blockIdx.x, next = 0, into = 0;
    auto begin = [&]() {
        if (next_item >= items) return;
        const int tile = next_item / across, n0 = (next_item - tile * across) * COLS;
        wr = p.w + (size_t)experts[tile] * p.w_expert + (size_t)((n0 + g) * step_n) * p.ldw + c0 * 64 + tq * 8;
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const int s = rows[tile * ROWS + h * 8 + g];
            xr[h] = s < 0 ? nullptr : p.x + (size_t)(p.which == 1 ? tile * ROWS + h * 8 + g : s / p.top) * p.ldx + c0 * 64 + tq * 8;
        }
    };
    auto ask = [&]() {
        if (next_item < items) {
            const uint32_t dst = own + into * CHUNK;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const bf16* from = wr + (size_t)((r >> 1) * step_u + (r & 1) * 8 * step_n) * p.ldw;
#pragma unroll
                for (int b = 0; b < 2; ++b) cp_async16(Chunk::weights_at(dst, b, r), from + b * 32, true);
            }
#pragma unroll
            for (int h = 0; h < H; ++h)
#pragma unroll
                for (int b = 0; b < 2; ++b)         // (rows that hold no token are zeros)
                    cp_async16(Chunk::tokens_at(dst, b, h), xr[h] ? xr[h] + next * 64 + b * 32 : p.x, xr[h] != nullptr);
            into = into + 1 == DEPTH ? 0 : into + 1;
            if (++next == chunks) {
                next = 0;
                next_item += gridDim.x;
                begin();
            } else {
                wr += 64;
            }
        }
        cp_async_commit();
    };
    if (chunks) {
        begin();
#pragma unroll
        for (int i = 0; i < DEPTH - 1; ++i) ask();
    }
    int from = 0;
    for (int item = blockIdx.x, turn = 0; item < items; item += gridDim.x, turn ^= 1) {
        RrSums<R, H> sums;
        sums.clear();
#pragma unroll 1
        for (int n = 0; n < chunks; ++n) {
            cp_async_wait<DEPTH - 2>();         // (a lane reads what it brought itself)
            const uint32_t src = own + from * CHUNK;
            from = from + 1 == DEPTH ? 0 : from + 1;
            Chunk chunk;
            chunk.read(src);
            ask();                              // (into the place that the turn before this one read)
            sums.add(chunk);
        }
        sums.leave(part, turn, warp, g, tq);
        __syncthreads();
        const int tile = item / across, n0 = (item - tile * across) * COLS;
        for (int i = threadIdx.x; i < ROWS * COLS; i += RR_WARPS * 32) {
            const int m = i / COLS, q = i - m * COLS, s = rows[tile * ROWS + m];
            if (s < 0) continue;
            const float w = p.row_weight ? p.row_weight[s] : 1.f;
            const size_t at = (size_t)(tile * ROWS + m) * p.ldo + n0 + q;
            const float v = rr_sum(part[turn], m, q);
            if constexpr (GLU) {
                const float u = rr_sum(part[turn], m, 16 + q);
                ((bf16*)p.out)[at] = __float2bfloat16_rn(glu_act<bf16>(v * w, u * w, p.limit, p.alpha, p.shift));
            } else if (p.which == 2) {
                ((bf16*)p.out)[at] = __float2bfloat16_rn(plain_act(v * w, p.pairs));
            } else {
                ((float*)p.out)[at] = v * w;
            }
        }
    }
    cp_async_wait<0>();
}

template <int H, int DEPTH, bool GLU>
static int mx_launch(const MoeRowsParams& p, int blocks, cudaStream_t stream) {
    constexpr int smem = RR_WARPS * DEPTH * RrChunk<4, H>::BYTES;
    static AcvSmemConfig cfg;
    auto kernel = moe_rows_kernel<H, DEPTH, GLU>;
    if (const int e = acv_ensure_smem(cfg, kernel, smem)) return e;
    acv_launch(PDL_GEMM, kernel, dim3(blocks), dim3(RR_WARPS * 32), smem, stream, p);
    return acv_launch_status();
}

// The arguments of acv_moe_gemm_mma, beside them: tile_rows 8 or 16, as acv_moe_group made the tiles, and the count it left.
ACV_API int acv_moe_rows(const void* A, int lda, const void* W, long long w_expert_stride, int ldw, void* C, int ldc, const int* grouped,
                         const int* tile_expert, const int* tiles_used, int tile_rows, const float* row_weight, int top, int max_tiles, int N,
                         int K, int which, float limit, float alpha, float shift, int pairs, int sms, cudaStream_t stream) {
    if (max_tiles <= 0 || N <= 0) return 0;
    if (K <= 0 || K % 64 || top <= 0 || which < 0 || which > 2 || N % (which == 0 ? 16 : 32) || (tile_rows != 8 && tile_rows != 16) ||
        max_tiles > MX_TILES || max_tiles * tile_rows > MX_ROWS || !tiles_used)
        return ACV_ERR_SIZE;
    if ((lda % 8) || (ldw % 8) || (w_expert_stride % 8) || ((uintptr_t)A & 15) || ((uintptr_t)W & 15)) return ACV_ERR_ALIGN;
    const MoeRowsParams p = {(const bf16*)A, (const bf16*)W, C, w_expert_stride, lda, ldw, ldc, top, N, K, which, pairs, limit, alpha, shift,
                             grouped, tile_expert, tiles_used, row_weight};
    const long long most = (long long)max_tiles * (N / (which == 0 ? 16 : 32));
    const int blocks = most < sms ? (int)most : sms;
    if (tile_rows == 8) return which == 0 ? mx_launch<1, 4, true>(p, blocks, stream) : mx_launch<1, 4, false>(p, blocks, stream);
    return which == 0 ? mx_launch<2, 3, true>(p, blocks, stream) : mx_launch<2, 3, false>(p, blocks, stream);
}
