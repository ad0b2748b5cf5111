// C[M,N] = X[M,K] . W[N,K]^T in bfloat16 for up to 32 tokens, float accumulators: the products of a decode step.
//
// What bounds such a product beside its weights' stream is what comes before the first and after the last of it: of the 5 us that
// a product of a few MB took on tcgen05 (128 weight rows to a tile, K split over a cluster, the splits' tiles sent to one CTA, the
// accumulator fetched from tensor memory, the tile turned through shared memory) most was hand-over.  Here a block takes 8 R
// weight rows and its eight warps an eighth of K each, on mma.sync (weight rows are its M, tokens its N): a lane brings its
// own operands by 16-byte asynchronous copies into a ring of its own (eight neighbouring k of a row; which k of a step of 32 a
// lane holds is the same for tokens and weights), weights before the wait for the kernel in front, so no barrier stands
// in the loop, and after it there is one, for the eight warps' sums.  A block goes on to its next rows with their first copies under way.
//
// Microseconds in a chain of such products, tcgen05 (gemm_tc.cu) and now, 8 tokens: 4096 x 1024 5.4 -> 2.6, 1024 x 3072 5.9 ->
// 2.7, 12288 x 2048 12.6 -> 9.9, 4096 x 4096 10.2 -> 7.2, 4096 x 12288 22.0 -> 20.1 (4.9 TB/s), 151936 x 4096 206 -> 193 (6.4 TB/s); with the q,k,v way out
// 32 heads of 128, K 1024, 6.1 -> 4.2, 48 heads, K 4096, 14.1 -> 13.3.
#include "gemm_epilogue.cuh"
#include "rows_ring.cuh"

struct RowsParams {
    const bf16 *x, *w;
    void* out;
    int ldx, ldw, ldo, M, N, K, out_f32, swiglu, early_w;
    // stacked q,k,v projection: per-head RMS norm of q and k, rotation, append of k and v to their pages (see GemmParams)
    int q_heads, kv_heads, head_dim, table_rows, bt_stride, page_size, num_pages;
    const float *q_w, *k_w, *cos_sin;
    float eps;
    const int *positions, *seq_of_token, *block_table, *bt_rows;
    bf16 *k_pages, *v_pages;
};

// R: octets of weight rows of a block (2 or 4); H: octets of tokens; DEPTH: chunks of 64 k in a warp's ring.
// QKV: a block holds 32 rows of a head, sixteen of each half, so that an angle's two rows meet in it; the head's blocks are a cluster
// (two for heads of 64, four for 128) whose blocks tell each other their sums of squares.
template <int R, int H, int DEPTH, bool QKV>
__global__ void __launch_bounds__(RR_WARPS * 32, 2)
gemm_rows_kernel(const RowsParams p) {
    using Chunk = RrChunk<R, H>;
    constexpr int CHUNK = Chunk::BYTES, COLS = 8 * R;
    extern __shared__ __align__(16) unsigned char ring[];
    __shared__ float part[2][RR_WARPS][8 * H][COLS + 4];
    __shared__ float squares[QKV ? 4 : 1][8 * H];
    ACV_TL(TL_GEMM, 0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tq = lane & 3;
    const int all = p.K / 64, tiles = p.N / COLS;
    const int c0 = all * warp / RR_WARPS, chunks = all * (warp + 1) / RR_WARPS - c0;       // this warp's chunks of K
    const uint32_t own = smem_u32(ring) + warp * (DEPTH * CHUNK) + lane * 16;
    // the first row of octet r of a tile
    auto row_of = [&](int tile, int r) {
        if constexpr (QKV) {
            const int per = p.head_dim / COLS;          // tiles of a head
            return tile / per * p.head_dim + (r >> 1) * (p.head_dim >> 1) + tile % per * 16 + (r & 1) * 8;
        } else {
            return tile * COLS + r * 8;
        }
    };
    const bf16* xr = p.x + (size_t)g * p.ldx + c0 * 64 + tq * 8;
    const bf16* wr = p.w + (size_t)(row_of(blockIdx.x, 0) + g) * p.ldw + c0 * 64 + tq * 8;
    int w_tile = blockIdx.x, w_next = 0, w_into = 0, x_tile = blockIdx.x, x_next = 0, x_into = 0;
    auto ask_w = [&]() {
        if (w_tile >= tiles) return;
        const uint32_t dst = own + w_into * CHUNK;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = QKV ? (r >> 1) * (p.head_dim >> 1) + (r & 1) * 8 : r * 8;
#pragma unroll
            for (int b = 0; b < 2; ++b) cp_async16(Chunk::weights_at(dst, b, r), wr + (size_t)row * p.ldw + b * 32, true);
        }
        w_into = w_into + 1 == DEPTH ? 0 : w_into + 1;
        if (++w_next == chunks) {
            w_next = 0;
            w_tile += gridDim.x;
            wr = p.w + (size_t)(row_of(w_tile, 0) + g) * p.ldw + c0 * 64 + tq * 8;
        } else {
            wr += 64;
        }
    };
    auto ask_x = [&]() {            // (tokens that do not exist are zeros)
        if (x_tile < tiles) {
            const uint32_t dst = own + x_into * CHUNK;
#pragma unroll
            for (int h = 0; h < H; ++h)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const bool in = h * 8 + g < p.M;
                    cp_async16(Chunk::tokens_at(dst, b, h), in ? xr + (size_t)h * 8 * p.ldx + x_next * 64 + b * 32 : p.x, in);
                }
            x_into = x_into + 1 == DEPTH ? 0 : x_into + 1;
            if (++x_next == chunks) { x_next = 0; x_tile += gridDim.x; }
        }
        cp_async_commit();
    };
    if (p.early_w && chunks) {
#pragma unroll
        for (int i = 0; i < DEPTH - 1; ++i) ask_w();
    }
    if constexpr (QKV) cluster_arrive();        // (waited for before the first word to a peer)
    pdl_launch_dependents();
    pdl_wait();
    if (chunks) {
#pragma unroll
        for (int i = 0; i < DEPTH - 1; ++i) {
            if (!p.early_w) ask_w();
            ask_x();
        }
    }
    // q,k,v: sixteen threads a token, each one angle's two rows; where the token stands is asked for now, used when the sums are there
    const int m_of = threadIdx.x >> 4, angle = QKV ? (int)(blockIdx.x % (p.head_dim / COLS)) * 16 + (threadIdx.x & 15) : 0;
    [[maybe_unused]] int pos = 0, page = -1;
    [[maybe_unused]] float co = 1.f, si = 0.f;
    if constexpr (QKV) {
        if (m_of < p.M) {
            pos = p.positions[m_of];
            const int sq = p.seq_of_token[m_of];
            page = p.block_table[(size_t)(p.bt_rows ? p.bt_rows[sq] : sq) * p.bt_stride + pos / p.page_size];
            if (page >= p.num_pages) page = -1;
            if (p.cos_sin && pos >= 0 && pos < p.table_rows) {
                co = p.cos_sin[(size_t)pos * p.head_dim + angle];
                si = p.cos_sin[(size_t)pos * p.head_dim + (p.head_dim >> 1) + angle];
            }
        }
    }
    int from = 0;
    for (int tile = blockIdx.x, turn = 0; tile < tiles; tile += gridDim.x, turn ^= 1) {
        RrSums<R, H> sums;
        sums.clear();
#pragma unroll 1
        for (int n = 0; n < chunks; ++n) {
            cp_async_wait<DEPTH - 2>();         // (a lane reads what it brought itself)
            const uint32_t src = own + from * CHUNK;
            from = from + 1 == DEPTH ? 0 : from + 1;
            Chunk chunk;
            chunk.read(src);
            ask_w();                            // (into the place that the turn before this one read)
            ask_x();
            sums.add(chunk);
        }
        sums.leave(part, turn, warp, g, tq);
        __syncthreads();
        auto sum = [&](int m, int q) { return rr_sum(part[turn], m, q); };
        if constexpr (QKV) {
            // (the grid is the tiles: one turn)
            const int head = tile / (p.head_dim / COLS), half = p.head_dim >> 1;
            const bool is_q = head < p.q_heads, is_k = !is_q && head < p.q_heads + p.kv_heads;
            const float* w = is_q ? p.q_w : is_k ? p.k_w : nullptr;
            const bool live = m_of < p.M;
            const int q = threadIdx.x & 15;
            float a = 0.f, b = 0.f;         // rounded as the projection's output is
            if (live) {
                a = __bfloat162float(__float2bfloat16_rn(sum(m_of, q)));
                b = __bfloat162float(__float2bfloat16_rn(sum(m_of, 16 + q)));
            }
            cluster_wait();                 // every block of the head has started
            if (w) {                        // (for a head's blocks alike)
                float ss = a * a + b * b;
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o, 16);
                const int blocks = p.head_dim / COLS;
                if (live && q < blocks)
                    cluster_store_f32(cluster_map(smem_u32(&squares[cluster_ctarank()][m_of]), q), ss);
                cluster_sync_all();
                if (live) {
                    ss = 0.f;
                    for (int r = 0; r < blocks; ++r) ss += squares[r][m_of];
                    const float inv = rsqrtf(ss / (float)p.head_dim + p.eps);
                    a = a * inv * w[angle];
                    b = b * inv * w[half + angle];
                }
            }
            if (live) {
                if ((is_q || is_k) && p.cos_sin && pos >= 0 && pos < p.table_rows) {
                    const float x0 = a, x1 = b;
                    a = x0 * co - x1 * si;
                    b = x1 * co + x0 * si;
                }
                bf16* dst = nullptr;
                if (is_q) {
                    dst = (bf16*)p.out + (size_t)m_of * p.ldo + (size_t)head * p.head_dim;
                } else if (page >= 0) {
                    const int kvh = is_k ? head - p.q_heads : head - p.q_heads - p.kv_heads;
                    dst = (is_k ? p.k_pages : p.v_pages) + (((size_t)page * p.kv_heads + kvh) * p.page_size + pos % p.page_size) * p.head_dim;
                }
                if (dst) {
                    dst[angle] = __float2bfloat16_rn(a);
                    dst[half + angle] = __float2bfloat16_rn(b);
                }
            }
        } else if (p.swiglu) {
            for (int i = threadIdx.x; i < p.M * (COLS / 2); i += RR_WARPS * 32) {
                const int m = i / (COLS / 2), q = i - m * (COLS / 2);
                ((bf16*)p.out)[(size_t)m * p.ldo + tile * (COLS / 2) + q] = swiglu_pair(sum(m, 2 * q), sum(m, 2 * q + 1));
            }
        } else {
            for (int i = threadIdx.x; i < p.M * COLS; i += RR_WARPS * 32) {
                const int m = i / COLS, q = i - m * COLS;
                const size_t at = (size_t)m * p.ldo + tile * COLS + q;
                if (p.out_f32) ((float*)p.out)[at] = sum(m, q);
                else ((bf16*)p.out)[at] = __float2bfloat16_rn(sum(m, q));
            }
        }
    }
    cp_async_wait<0>();
}

template <int R, int H, int DEPTH, bool QKV>
static int rw_launch(const RowsParams& p, int sms, cudaStream_t stream) {
    constexpr int smem = RR_WARPS * DEPTH * RrChunk<R, H>::BYTES, fixed = 2 * RR_WARPS * 8 * H * (8 * R + 4) * 4 + 2048;
    constexpr int resident = 228 * 1024 / (smem + fixed) > 2 ? 2 : 228 * 1024 / (smem + fixed);
    static_assert(resident >= 1, "a block fits an SM's shared memory");
    static AcvSmemConfig cfg;
    auto kernel = gemm_rows_kernel<R, H, DEPTH, QKV>;
    if (const int e = acv_ensure_smem(cfg, kernel, smem)) return e;
    if (QKV)
        acv_launch_cluster(PDL_GEMM, dim3(p.head_dim / (8 * R), 1, 1), kernel, dim3(p.N / (8 * R)), dim3(RR_WARPS * 32), smem, stream, p);
    else
        acv_launch(PDL_GEMM, kernel, dim3(min(p.N / (8 * R), resident * sms)), dim3(RR_WARPS * 32), smem, stream, p);
    return acv_launch_status();
}

// Sixteen or 32 weight rows to a block, and how deep a ring: the blocks that come one after the other on an SM times their rows
// decide, 32 rows where that is nearly even, for the tokens are read once for each block (8 tokens, microseconds with sixteen and 32:
// 6144 x 4096 11.0 and 11.9, 2048 x 6144 6.3 and 6.9, 4096 x 4096 7.6 and 7.2, 12288 x 2048 11.6 and 9.9, 19456 x 2560 21.5 and 19.8).
// K = 1024 leaves a warp two chunks: 6144 x 1024 3.5 and 3.3, and no use for a deeper ring.  Many rounds want the shallow one
// (151936 x 4096 193 and 207).
static bool rw_wide(int N, int K, int sms) {
    if (N % 32) return false;
    const long long narrow = (N / 16 + sms - 1) / sms * 2, wide = (N / 32 + sms - 1) / sms * 4;
    return narrow * 10 >= wide * (K <= 1024 ? 7 : 8);
}

static int rw_checks(const RowsParams& p) {
    if (p.M > 32 || p.K <= 0 || p.K % 64 || p.N % 16) return ACV_ERR_SIZE;
    if (((uintptr_t)p.x | (uintptr_t)p.w) % 16 || p.ldx % 8 || p.ldw % 8) return ACV_ERR_ALIGN;
    return 0;
}

// x [M,K], w [N,K] bfloat16; out [M,N] bfloat16 or float, or with `swiglu` (rows of w in (gate, up) pairs) bfloat16 [M,N/2].
// flags: 1 the weights were written long before, they may be read while the kernel in front still runs.
ACV_API int acv_gemm_rows(const void* x, int ldx, const void* w, int ldw, void* out, int ldo, int M, int N, int K, int out_f32, int swiglu,
                          int flags, int sms, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    RowsParams p = {};
    p.x = (const bf16*)x; p.w = (const bf16*)w; p.out = out;
    p.ldx = ldx; p.ldw = ldw; p.ldo = ldo; p.M = M; p.N = N; p.K = K;
    p.out_f32 = out_f32; p.swiglu = swiglu; p.early_w = flags & 1;
    if (const int e = rw_checks(p)) return e;
    if (swiglu && out_f32) return ACV_ERR_DTYPE;
    if (M > 16) return rw_launch<2, 4, 3, false>(p, sms, stream);
    const bool wide = rw_wide(N, K, sms);
    if (M > 8) return wide ? rw_launch<4, 2, 3, false>(p, sms, stream) : rw_launch<2, 2, 6, false>(p, sms, stream);
    if (!wide) return K <= 1024 ? rw_launch<2, 1, 3, false>(p, sms, stream) : rw_launch<2, 1, 6, false>(p, sms, stream);
    return K <= 1024 || N / 32 > 6 * sms ? rw_launch<4, 1, 3, false>(p, sms, stream) : rw_launch<4, 1, 5, false>(p, sms, stream);
}

// The stacked q,k,v projection with heads of 64 or 128 (see acv_gemm_tc_qkv for the arguments).
ACV_API int acv_gemm_rows_qkv(const void* x, int ldx, const void* w, int ldw, void* out, int ldo, int M, int N, int K, int flags, int sms,
                              int NH, int NKV, int D, const float* q_w, const float* k_w, float eps, const float* cos_sin, int table_rows,
                              const int* positions, const int* seq_of_token, const int* block_table, int bt_stride, const int* bt_rows,
                              void* k_pages, void* v_pages, int page_size, int num_pages, cudaStream_t stream) {
    // (what acv_gemm_tc_qkv refuses, whose calls of few tokens come here: an empty product is none of it)
    if ((D != 64 && D != 128) || NH <= 0 || NKV <= 0 || N != (NH + 2 * NKV) * D || !k_pages || !v_pages || !positions || !seq_of_token ||
        !block_table || page_size <= 0 || ((uintptr_t)k_pages & 15) || ((uintptr_t)v_pages & 15) || (cos_sin && ((uintptr_t)cos_sin & 15)))
        return ACV_ERR_SIZE;
    if (M <= 0) return 0;
    if (((uintptr_t)out & 15) || (ldo & 7)) return ACV_ERR_SIZE;
    RowsParams p = {};
    p.x = (const bf16*)x; p.w = (const bf16*)w; p.out = out;
    p.ldx = ldx; p.ldw = ldw; p.ldo = ldo; p.M = M; p.N = N; p.K = K; p.early_w = flags & 1;
    p.q_heads = NH; p.kv_heads = NKV; p.head_dim = D; p.q_w = q_w; p.k_w = k_w; p.eps = eps; p.cos_sin = cos_sin; p.table_rows = table_rows;
    p.positions = positions; p.seq_of_token = seq_of_token; p.block_table = block_table; p.bt_stride = bt_stride; p.bt_rows = bt_rows;
    p.k_pages = (bf16*)k_pages; p.v_pages = (bf16*)v_pages; p.page_size = page_size; p.num_pages = num_pages;
    if (const int e = rw_checks(p)) return e;
    if (M > 16) return ACV_ERR_SIZE;
    if (M > 8) return rw_launch<4, 2, 3, true>(p, sms, stream);
    // more heads than come at once with an SM to a block: a shallow ring, two blocks to an SM
    if (N / D > (D == 128 ? 33 : 74) * sms / 148) return rw_launch<4, 1, 2, true>(p, sms, stream);
    return K <= 1024 ? rw_launch<4, 1, 3, true>(p, sms, stream) : rw_launch<4, 1, 5, true>(p, sms, stream);
}

ACV_TL_EXPORT(gemm_rows)
