// C[M,N] = A[M,K] . W[N,K]^T in 32-bit precision on the fifth-generation tensor cores.
//
// A float, times 2^24 so that the smallest ones are among them (gemm_split_tc.h), is the exact sum of three bfloat16 values,
// x = x1 + x2 + x3 (each the rounding of what the ones before it leave: 8 + 8 + 8 bits), and products of bfloat16 values are exact
// in the tensor core's float accumulators.  Of the nine products of parts the six above 2^-24 of the result are made: over a chunk of GF_CHUNK k the accumulator takes w1 a2, w2 a1, w1 a3,
// w2 a2, w3 a1 (2^-8 of the result and less) and at last w1 a1.  The tensor core's additions cut off instead of rounding, so
// no more than the two of w1 a1 follow one another at full size; the chunks are added in registers, to nearest.
//
// The order of a sum is a property of K alone, as in gemm_simt.cu: K is cut into up to eight groups of gf_group_length(K), a
// group is its chunks in ascending order, groups are added in ascending order.  So a row's result does not depend
// on the other rows, on M, N or the tile.  An output that is no finite number this way (an infinity among the operands has no
// three parts; operands from 2^104 and sums from 2^80 on leave a float's range by the scale) is made again by a plain chain of
// multiply-adds, with the order of gemm_simt.cu.
//
// Weight rows fill the tensor core's M = 128, tokens are its N (BT of them): weights are read once for up to 128 tokens.
// Converter warps read float rows straight into registers (a stage ahead), cut them into parts and leave those in shared
// memory as swizzled K-major tiles; one thread issues the products; other warps add up the chunks.
//
// What bounds it: shared memory (a stage of 128 tokens takes it some 2300 clocks, 96 KB of parts written and what the products read
// of them, the tensor cores 1536) and the stages' hand-overs; the tensor cores are busy 50 % of the time.  Microseconds, eight chains
// of multiply-adds on the CUDA cores (gemm_simt.cu) and now: 696 tokens
// 4096 x 1024 212 -> 73, 1024 x 2048 101 -> 51, 1024 x 3072 142 -> 65, 2048 tokens 4096 x 4096 1750 -> 489 (141 TFLOP/s),
// 64 tokens 4096 x 1024 22 -> 15, 17 tokens 151936 x 1024 354 -> 214.  Error against 64 bits (2-norm): K 1024 2.1e-7 ->
// 0.94e-7, 4096 4.1e-7 -> 1.1e-7, 12288 6.8e-7 -> 1.5e-7.
#include "tc_ptx.cuh"
#include "gemm_split_tc.h"

#define GF_CHUNK 32         // k that are summed in tensor memory
#define GF_BUFS 3           // chunks in tensor memory: one made, one read, one on its way
#define GF_CONV 8           // converter warps
#define GF_ROWS 128         // weight rows of a tile

template <int BT_, int STAGES_, int EPI_>
struct GfTile {
    static constexpr int BT = BT_, STAGES = STAGES_, EPI = EPI_;
    static constexpr int W_PART = GF_ROWS * GF_BK * 2, T_PART = BT * GF_BK * 2, STAGE = 3 * (W_PART + T_PART);
    // (registers are given out to warps by fours, so the one warp that issues the products comes with three that do nothing)
    static constexpr int THREADS = (GF_CONV + EPI + 4) * 32;
    static constexpr int COLS = BT / (EPI / 4);                 // tokens of an epilogue thread
    // the next stage's rows asked for once this one is handed over, not row by row as their registers come free: 2048 tokens
    // 4096 x 4096 518 -> 479 us (before operands were scaled) in tiles of 128 tokens, whose converters are short of registers, no change in the others
    static constexpr bool LATE = EPI == 8;
    static constexpr int PIECE = EPI == 8 ? 16 : 32;            // columns read at a time (96 registers a thread, or 128)
    static constexpr int TMEM = 4 * BT < 32 ? 32 : 4 * BT;      // three chunks | the groups' sum
    static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
    static_assert(2 * BT * GF_ROWS * 4 <= STAGES * STAGE, "two groups of a tile in float fit where the stages were");
    static_assert(SMEM + 1024 <= 228 * 1024, "a CTA fits an SM's shared memory");
};

// eight consecutive floats of a row (by plain loads: the rows may be the kernel's in front, which runs while this one begins, and the
// read-only path is not ordered behind the wait for it)
template <bool PIECES>
__device__ __forceinline__ void gf_load8(const float* from, float (&x)[8]) {
    if constexpr (PIECES) {
        const float4 a = reinterpret_cast<const float4*>(from)[0], b = reinterpret_cast<const float4*>(from)[1];
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = from[i];
    }
}

// the three parts of eight floats into shared memory, `part` bytes apart
__device__ __forceinline__ void gf_store_parts(uint32_t dst, uint32_t part, float (&x)[8]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) gf_scale(x[2 * i], x[2 * i + 1]);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        uint32_t h[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            h[i] = pack_bf16x2(x[2 * i], x[2 * i + 1]);
            if (p < 2) gf_less(x[2 * i], x[2 * i + 1], h[i]);
        }
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + p * part), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]) : "memory");
    }
}

template <typename T, bool PIECES>
__global__ void __launch_bounds__(T::THREADS, 1)
gemm_split_tc_kernel(const GfArgs p, int parts, int per) {
    constexpr int BT = T::BT, ST = T::STAGES;
    extern __shared__ unsigned char gf_raw[];
    unsigned char* tiles = gf_raw + ((1024u - (gt_smem(gf_raw) & 1023u)) & 1023u);
    const uint32_t tiles_addr = gt_smem(tiles);
    // barriers: full[ST], empty[ST], chunk full[GF_BUFS], chunk empty[GF_BUFS]
    const uint32_t full0 = tiles_addr + ST * T::STAGE, empty0 = full0 + 8 * ST, cfull0 = empty0 + 8 * ST, cempty0 = cfull0 + 8 * GF_BUFS;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* A = p.A + (size_t)blockIdx.z * p.a_batch;
    const float* W = p.W + (size_t)blockIdx.z * p.w_batch;
    // the groups of a tile: all of them by one CTA (parts 1), or `per` (1 or 2) by each CTA of a cluster
    const int part = blockIdx.x % parts, n0 = (blockIdx.x / parts) * GF_ROWS, m0 = blockIdx.y * BT;
    const int gl = gf_group_length(p.K), groups = (p.K + gl - 1) / gl;
    const int k_begin = part * per * gl, k_end = min(p.K, k_begin + per * gl);
    const int iters = (k_end - k_begin + GF_BK - 1) / GF_BK, per_group = gl / GF_BK;
    constexpr int CHUNKS = GF_BK / GF_CHUNK;

    if (tid == 0) {
        abort_s = 0;
        for (int s = 0; s < ST; ++s) { mbar_init(full0 + 8 * s, GF_CONV); mbar_init(empty0 + 8 * s, 1); }
        for (int b = 0; b < GF_BUFS; ++b) { mbar_init(cfull0 + 8 * b, 1); mbar_init(cempty0 + 8 * b, T::EPI); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gt_smem(&tmem_base_s)), "r"(T::TMEM));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    auto give_up = [&](int code) { abort_s = 1; if (p.status) atomicExch(p.status, code); };

    // the products of one stage (one thread)
    auto issue = [&](int it) {
        const int s = it % ST;
        if (!mbar_wait(full0 + 8 * s, (it / ST) & 1, &abort_s)) { give_up(31); return; }
        tc_fence_after();
        const uint32_t w1 = umma_desc_lo(tiles_addr + s * T::STAGE), t1 = umma_desc_lo(tiles_addr + s * T::STAGE + 3 * T::W_PART);
        constexpr uint32_t WP = T::W_PART >> 4, TP = T::T_PART >> 4;
        const uint32_t idesc = umma_idesc(BT);
#pragma unroll
        for (int ch = 0; ch < CHUNKS; ++ch) {
            const int n = it * CHUNKS + ch, buf = n % GF_BUFS;
            if (!mbar_wait(cempty0 + 8 * buf, (n / GF_BUFS & 1) ^ 1, &abort_s)) { give_up(32); return; }
            tc_fence_after();
            const uint32_t c = tmem + buf * BT;
#pragma unroll
            for (int k = 0; k < GF_CHUNK / 16; ++k) {
                const uint32_t at = 2 * (ch * (GF_CHUNK / 16) + k);
                tc_mma_bf16_h(c, w1 + at, t1 + TP + at, idesc, k > 0);
                tc_mma_bf16_h(c, w1 + WP + at, t1 + at, idesc, 1);
                tc_mma_bf16_h(c, w1 + at, t1 + 2 * TP + at, idesc, 1);
                tc_mma_bf16_h(c, w1 + WP + at, t1 + TP + at, idesc, 1);
                tc_mma_bf16_h(c, w1 + 2 * WP + at, t1 + at, idesc, 1);
            }
#pragma unroll
            for (int k = 0; k < GF_CHUNK / 16; ++k) {
                const uint32_t at = 2 * (ch * (GF_CHUNK / 16) + k);
                tc_mma_bf16_h(c, w1 + at, t1 + at, idesc, 1);
            }
            tc_commit(cfull0 + 8 * buf);
        }
        tc_commit(empty0 + 8 * s);
    };

    float acc[T::COLS];                 // (epilogue threads)
    const int et = warp < GF_CONV + T::EPI ? warp - GF_CONV : -1;      // among the epilogue's warps
    const int col0 = (et >> 2) * T::COLS;
    const int f = (warp & 3) * 32 + lane, gn = n0 + f;
    float* C = p.C + (size_t)blockIdx.z * p.c_batch + gn;
    const float* gate = p.gate ? p.gate + (size_t)blockIdx.z * p.g_batch + gn : nullptr;
    bool again = gate != nullptr;       // this thread's outputs are looked at again: a gate, or one that is no finite number
    auto put = [&](int gm, float x) {
        again |= !(fabsf(x) <= 3.402823466e38f);
        C[(size_t)gm * p.ldc] = x * GF_SCALE_BACK;
    };
    auto look_again = [&](int first, int behind, int step) {
#pragma unroll 1
        for (int gm = first; gm < min(p.M, behind); gm += step) {
            float x = C[(size_t)gm * p.ldc];
            if (!(fabsf(x) <= 3.402823466e38f)) x = gf_plain(A + (size_t)gm * p.lda, W + (size_t)gn * p.ldw, p.K);
            if (gate) x /= 1.f + expf(-gate[(size_t)gm * p.ldg]);
            C[(size_t)gm * p.ldc] = x;
        }
    };

    if (warp < GF_CONV) {
        // ------------------------------------------------------------------ float rows into parts
        constexpr int TASKS = (GF_ROWS + BT) * 8, ROUNDS = (TASKS + GF_CONV * 32 - 1) / (GF_CONV * 32), W_ROUNDS = GF_ROWS / (GF_CONV * 4);
        const int c = tid & 7, r0 = tid >> 3;       // eight threads a row, eight floats each
        float x[ROUNDS][8];
        pdl_wait();
        // rows that do not exist: the last one that does (their outputs go nowhere)
        auto row_of = [&](int i) {
            return i < W_ROUNDS ? W + (size_t)min(n0 + r0 + i * (GF_CONV * 4), p.N - 1) * p.ldw
                                : A + (size_t)min(m0 + r0 + (i - W_ROUNDS) * (GF_CONV * 4), p.M - 1) * p.lda;
        };
        auto mine = [&](int i) { return TASKS % (GF_CONV * 32) == 0 || i * (GF_CONV * 4) + r0 < GF_ROWS + BT; };
        auto ragged = [&](int k) {                  // where K ends within the eight
#pragma unroll 1
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int i = 0; i < ROUNDS; ++i) {
                    const float v = k + j < k_end && mine(i) ? row_of(i)[k + j] : 0.f;
#pragma unroll
                    for (int q = 0; q < 8; ++q) x[i][q] = q == j ? v : x[i][q];
                }
        };
        {
            const int k = k_begin + c * 8;
            if (k + 8 <= k_end) {
#pragma unroll
                for (int i = 0; i < ROUNDS; ++i)
                    if (mine(i)) gf_load8<PIECES>(row_of(i) + k, x[i]);
            } else {
                ragged(k);
            }
        }
        for (int it = 0; it < iters; ++it) {
            const int s = it % ST, next = k_begin + (it + 1) * GF_BK + c * 8;
            if (!__all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, ((it / ST) & 1) ^ 1, &abort_s))) { give_up(34); break; }
            const uint32_t at = tiles_addr + s * T::STAGE + r0 * 128 + ((c ^ (r0 & 7)) << 4);
            const bool whole = next + 8 <= k_end;
#pragma unroll
            for (int i = 0; i < ROUNDS; ++i) {
                if (!mine(i)) break;
                gf_store_parts(at + (i < W_ROUNDS ? i : i - W_ROUNDS) * (GF_CONV * 4 * 128) + (i < W_ROUNDS ? 0 : 3 * T::W_PART),
                               i < W_ROUNDS ? T::W_PART : T::T_PART, x[i]);
                if (!T::LATE && whole) gf_load8<PIECES>(row_of(i) + next, x[i]);
            }
            if (!T::LATE && !whole && it + 1 < iters) ragged(next);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(full0 + 8 * s);
            if constexpr (T::LATE) {
                if (whole) {
#pragma unroll
                    for (int i = 0; i < ROUNDS; ++i) gf_load8<PIECES>(row_of(i) + next, x[i]);
                } else if (it + 1 < iters) {
                    ragged(next);
                }
            }
        }
    } else if (warp < GF_CONV + T::EPI) {
        // ------------------------------------------------------------------ chunks and groups added up
#pragma unroll
        for (int j = 0; j < T::COLS; ++j) acc[j] = 0.f;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        pdl_wait();
        bool ok = true;
        for (int it = 0; it < iters && ok; ++it) {
#pragma unroll
            for (int ch = 0; ch < CHUNKS; ++ch) {
                const int n = it * CHUNKS + ch, buf = n % GF_BUFS;
                if (!__all_sync(0xffffffffu, mbar_wait(cfull0 + 8 * buf, n / GF_BUFS & 1, &abort_s))) { give_up(35); ok = false; break; }
                tc_fence_after();
                const uint32_t from = tmem + lanes + buf * BT + col0;
#pragma unroll
                for (int j = 0; j < T::COLS; j += T::PIECE) {
                    uint32_t v[T::PIECE];
                    if constexpr (T::PIECE == 32) tc_ld32(from + j, v);
                    else tc_ld16(from + j, v);
#pragma unroll
                    for (int i = 0; i < T::PIECE; ++i) acc[j + i] += __uint_as_float(v[i]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(cempty0 + 8 * buf);
            }
            if (!ok || !(it % per_group == per_group - 1 || it == iters - 1)) continue;
            const int group = it / per_group;
            // what there is of the groups before waits in tensor memory, in columns that no product writes: their sum, or
            // the first of a CTA's two
            const uint32_t kept = tmem + lanes + GF_BUFS * BT + col0;
            const bool last = it == iters - 1;
            float* left = reinterpret_cast<float*>(tiles) + (size_t)col0 * GF_ROWS + f;        // [group of this CTA][token][feature]
#pragma unroll
            for (int j = 0; j < T::COLS; j += 16) {
                uint32_t b[16];
                if (group > 0) {
                    tc_ld16(kept + j, b);
                    if (parts == 1) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) acc[j + i] = __uint_as_float(b[i]) + acc[j + i];
                    } else {            // (the CTA's last chunk has been made: its stages are free)
#pragma unroll
                        for (int i = 0; i < 16; ++i) left[(j + i) * GF_ROWS] = __uint_as_float(b[i]);
                    }
                }
                if (!last) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        b[i] = __float_as_uint(acc[j + i]);
                        acc[j + i] = 0.f;
                    }
                    tc_st16_nowait(kept + j, b);
                } else if (parts > 1) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) left[((group * BT) + j + i) * GF_ROWS] = acc[j + i];
                }
            }
            if (!last) tc_wait_st();
        }
        if (parts == 1 && gn < p.N) {
#pragma unroll
            for (int j = 0; j < T::COLS; ++j)
                if (m0 + col0 + j < p.M) put(m0 + col0 + j, acc[j]);
            if (again) look_again(m0 + col0, m0 + col0 + T::COLS, 1);
        }
    } else {
        if (warp == GF_CONV + T::EPI && lane == 0)
            for (int it = 0; it < iters && !abort_s; ++it) issue(it);
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();                    // all products of this CTA are complete and read
    pdl_launch_dependents();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::TMEM));
    if (parts == 1) return;
    // the groups of a tile meet: they lie in their CTAs' shared memory, each CTA adds up its share of the tokens
    cluster_sync_all();
    if (et >= 0 && gn < p.N) {
        constexpr int WARPS = T::EPI / 4, BATCH = 4;
        const int step = parts * WARPS, first = part * WARPS + (et >> 2);
#pragma unroll 1
        for (int t0 = first; t0 < BT && m0 + t0 < p.M; t0 += BATCH * step) {
            float v[BATCH][GF_GROUPS];          // (all asked for before the first is used)
#pragma unroll
            for (int j = 0; j < BATCH; ++j)
#pragma unroll
                for (int q = 0; q < GF_GROUPS; ++q) {
                    const int r = per == 1 ? q : q >> 1, slot = q - r * per;
                    if (q < groups && t0 + j * step < BT)
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[j][q])
                                     : "r"(cluster_map(tiles_addr + ((slot * BT + t0 + j * step) * GF_ROWS + f) * 4, r)) : "memory");
                }
#pragma unroll
            for (int j = 0; j < BATCH; ++j) {
                const int t = t0 + j * step;
                float x = v[j][0];
#pragma unroll
                for (int q = 1; q < GF_GROUPS; ++q)
                    if (q < groups) x = x + v[j][q];
                if (t < BT && m0 + t < p.M) put(m0 + t, x);
            }
        }
        if (again) look_again(m0 + first, m0 + BT, step);
    }
    cluster_sync_all();                 // nobody leaves while its tile is read
}

template <typename T, bool PIECES>
static int gf_launch(const GfArgs& p, int parts, int per, int batches, cudaStream_t stream) {
    auto kernel = gemm_split_tc_kernel<T, PIECES>;
    static AcvSmemConfig cfg;
    if (const int e = acv_ensure_smem(cfg, kernel, T::SMEM)) return e;
    const dim3 grid((p.N + GF_ROWS - 1) / GF_ROWS * parts, (p.M + T::BT - 1) / T::BT, batches);
    if (grid.y > 65535 || grid.z > 65535) return ACV_ERR_SIZE;
    acv_launch_cluster(PDL_GEMM, dim3(parts, 1, 1), kernel, grid, dim3(T::THREADS), T::SMEM, stream, p, parts, per);
    return acv_launch_status();
}

typedef GfTile<32, 3, 4> GfTokens32;
typedef GfTile<64, 3, 4> GfTokens64;
typedef GfTile<128, 2, 8> GfTokens128;

// way: an index of GF_WAYS; per: the groups of a CTA, 1 or 2 (in a cluster), or all
int gf_run_as(const GfArgs& p, bool pieces, int batches, int way, int per, cudaStream_t stream) {
    const int gl = gf_group_length(p.K), groups = (p.K + gl - 1) / gl, parts = (groups + per - 1) / per;
#define GF_CASE(TT) return pieces ? gf_launch<TT, true>(p, parts, per, batches, stream) : gf_launch<TT, false>(p, parts, per, batches, stream)
    switch (way) {
        case 0: GF_CASE(GfTokens32);
        case 1: GF_CASE(GfTokens64);
        default: GF_CASE(GfTokens128);
    }
#undef GF_CASE
}

// Which tile and how the groups are shared out: the way whose rounds of the device take least.  A round is as many CTAs as
// have an SM each, with clusters as many as fit the device's parts; its time in nanoseconds is a stage's times the stages of a CTA
// and what comes before and after them, measured (4096 x 1024, microseconds: 64 tokens as 64 x all / 64 x 2 / 64 x 1 groups
// 30 / 14 / 28; 696 tokens as 128 x all / 128 x 2 / 64 x all 71 / 104 / 82).
struct GfWay { int bt, stage, rest; };
static const GfWay GF_WAYS[3] = {{32, 1200, 5200}, {64, 1350, 6800}, {128, 1700, 10000}};

int gf_run(const GfArgs& p, bool pieces, int batches, int sms, cudaStream_t stream) {
    if (gr_takes(p, batches, sms)) return gr_run(p, pieces, batches, sms, stream);
    const int gl = gf_group_length(p.K), stages = (p.K + GF_BK - 1) / GF_BK, group = gl / GF_BK, groups = (p.K + gl - 1) / gl;
    int way = 0, per = groups;
    double best = -1.;
    for (int w = 0; w < 3; ++w)
        for (int q = 0; q < 3; ++q) {
            const GfWay& g = GF_WAYS[w];
            const int each = q == 2 ? groups : q + 1, parts = (groups + each - 1) / each;
            const long long tiles = (long long)((p.M + g.bt - 1) / g.bt) * ((p.N + GF_ROWS - 1) / GF_ROWS) * batches;
            const long long at_once = max(1, ACV_CLUSTERS_AT_ONCE[parts] * sms / 148);
            const double t = (double)((tiles + at_once - 1) / at_once) * (min(stages, each * group) * (double)g.stage + g.rest);
            if (best < 0. || t < best) { best = t; way = w; per = each; }
        }
    return gf_run_as(p, pieces, batches, way, per, stream);
}
