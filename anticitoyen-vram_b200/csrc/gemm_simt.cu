// C[M,N] = A[M,K] . W[N,K]^T on the CUDA cores, accumulated in true 32-bit
// (FFMA; no tensor-core mode, hence no TF32 anywhere).  It is the matrix product
// of the 32-bit path of the model for K under GF_MIN_K (longer float sums are made of exact parts on the
// tensor cores, gemm_split_tc.cu; the entry points here choose), and it computes logits in float from bfloat16
// operands (the reference upcasts the head's input and accumulates and returns
// float32, acvram/engine/model.py:369-410; products of bfloat16 values are exact
// in float, so float accumulation of bfloat16 operands is that computation).
//
// The order of a sum is a property of K alone (and so is which of the two makes it), so a row's result does not depend on
// the other rows, on M, N or the tile that computes it: K is cut into eight groups of
// gs_group_length(K) consecutive elements; a group is one chain of fused multiply-adds in
// ascending order; the groups are added as a balanced tree,
// ((g0+g1)+(g2+g3))+((g4+g5)+(g6+g7)).  The CTAs that share a tile (a cluster of 1, 2, 4
// or 8) each take a whole subtree.
//
// What bounds it: for many rows the FFMA pipes (of 73 TFLOP/s; three different registers to an instruction leave 60), for few
// rows the weights' stream.  Measured when it made the sums of every K, microseconds before (tiles of 64 x 64, scalar reads, no
// split of K) and after (gemm_split_tc.cu has what these sizes take there): 696 rows
// 4096 x 1024 240 -> 209, 1024 x 2048 174 -> 100, 1024 x 3072 258 -> 143, 2048 rows 4096 x 4096 -> 1750 (39 TFLOP/s); 3 rows
// 4096 x 1024 71 -> 6.5, 1024 x 3072 211 -> 7.7, 151936 x 1024 713 -> 114 (5460 GB/s of weights).  Both
// operands lie in shared memory as they lie in global memory (K innermost, rows padded to
// 36 floats so that eight rows' 16-byte reads meet no bank twice); a thread reads two or
// four k of a row at a time and holds MI x NJ outputs.  Rows come by cp.async, 32 elements a
// stage; operands that are bfloat16 or not made of 16-byte pieces go through registers
// instead (ASYNC = false).
#include "common.cuh"
#include "gemm_split_tc.h"

#define GS_BK 32
#define GS_LD (GS_BK + 4)
#define GS_GROUPS 8

__host__ __device__ __forceinline__ int gs_group_length(int K) {
    return ((K + GS_GROUPS - 1) / GS_GROUPS + GS_BK - 1) / GS_BK * GS_BK;
}

__device__ __forceinline__ void gs_copy16(uint32_t dst, const void* src, int bytes) {   // the rest of the 16 bytes: zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ float gs_peer_float(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
template <int N> __device__ __forceinline__ void gs_read(float* v, const float* from) {
    if constexpr (N == 4) {
        const float4 t = *reinterpret_cast<const float4*>(from);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
        const float2 t = *reinterpret_cast<const float2*>(from);
        v[0] = t.x; v[1] = t.y;
    }
}

// NW warps, WM of them along M; a warp is TY (M) x 32/TY (N) threads, a thread MI x NJ outputs: rows ty + TY i and columns
// tx + TX j of its warp's.  TY = 1 for few rows: a lane a column, so a 16-byte read of 32 weight rows moves 512 different
// bytes and the activations' reads are one address a warp.
template <int NW_, int WM, int TY_, int MI, int NJ, int STAGES_, int RESIDENT_, int KS_>
struct GsTile {
    static constexpr int NW = NW_, WN = NW / WM, TY = TY_, TX = 32 / TY, BM = WM * TY * MI, BN = WN * TX * NJ, STAGES = STAGES_;
    static constexpr int STAGE = (BM + BN) * GS_LD;      // floats
    static constexpr int SMEM = (STAGES * STAGE > BM * BN ? STAGES * STAGE : BM * BN) * 4;
    static constexpr int RESIDENT = RESIDENT_;           // CTAs that share an SM
    static constexpr int M_WARPS = WM, ROWS = MI, COLS = NJ, THREADS = NW * 32, KS = KS_;
    static_assert(RESIDENT * (SMEM + 1024) <= 228 * 1024, "RESIDENT CTAs of this tile do not fit an SM's shared memory");
};

struct GsArgs {
    const void *A, *W, *gate;
    void* C;
    int lda, ldw, ldc, ldg, M, N, K;
    long long a_batch, w_batch, c_batch, g_batch;
};

template <typename TI, typename TO, bool ASYNC, typename T>
__global__ void __launch_bounds__(T::THREADS, T::RESIDENT)
gemm_simt_kernel(const GsArgs p, int parts) {
    constexpr int BM = T::BM, BN = T::BN, MI = T::ROWS, NJ = T::COLS, TY = T::TY, TX = T::TX, ST = T::STAGES, NT = T::THREADS;
    extern __shared__ __align__(16) float gs_sm[];
    // blockIdx.z: one product of a batch (A, W and C each move by their batch stride, in elements)
    const TI* A = (const TI*)p.A + (size_t)blockIdx.z * p.a_batch;
    const TI* W = (const TI*)p.W + (size_t)blockIdx.z * p.w_batch;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = lane % TX, ty = lane / TX;
    const int row0 = (warp % T::M_WARPS) * TY * MI + ty, col0 = (warp / T::M_WARPS) * TX * NJ + tx;     // in the tile
    const int part = blockIdx.x % parts;
    const int m0 = blockIdx.y * BM, n0 = (blockIdx.x / parts) * BN;
    const int gl = gs_group_length(p.K), share_of_k = GS_GROUPS / parts * gl;
    const int k_begin = part * share_of_k;
    const int k_end = min(p.K, k_begin + share_of_k);
    // (as many groups as K reaches, rounded up to a whole subtree: the others would add nothing)
    int groups = 1;
    while (groups * parts < GS_GROUPS && k_begin + groups * gl < k_end) groups *= 2;
    const int iters = k_end > k_begin ? (k_end - k_begin + GS_BK - 1) / GS_BK : 0;

    float acc[MI][NJ];
    float st[4][MI * NJ];       // finished subtrees of 1, 2, 4 (and, at the end, all 8) groups
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) acc[i][j] = 0.f;

    auto fold = [&](int g) {    // group g of this CTA is complete
        int b = 0;
        while ((g >> b) & 1) ++b;
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                float v = acc[i][j];
                acc[i][j] = 0.f;
                for (int l = 0; l < b; ++l) v = st[l][i * NJ + j] + v;
                st[b][i * NJ + j] = v;
            }
    };
    auto multiply = [&](const float* as, const float* ws) {
        as += row0 * GS_LD;
        ws += col0 * GS_LD;
#pragma unroll
        for (int kk = 0; kk < GS_BK; kk += T::KS) {
            float a[MI][T::KS];
#pragma unroll
            for (int i = 0; i < MI; ++i) gs_read<T::KS>(a[i], as + i * TY * GS_LD + kk);
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                float b[T::KS];
                gs_read<T::KS>(b, ws + j * TX * GS_LD + kk);
#pragma unroll
                for (int k = 0; k < T::KS; ++k)
#pragma unroll
                    for (int i = 0; i < MI; ++i) acc[i][j] = fmaf(a[i][k], b[k], acc[i][j]);
            }
        }
    };
    const int per_group = gl / GS_BK;
    int done = 0, left = per_group;     // groups folded; iterations left of the current one

    pdl_wait();
    if constexpr (ASYNC) {
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(gs_sm);
        auto load = [&](int it) {
            const int k = k_begin + it * GS_BK + (tid & 7) * 4;       // eight threads a row: 16 bytes each
            const uint32_t dst = base + ((it % ST) * T::STAGE + (tid & 7) * 4) * 4;
#pragma unroll
            for (int r = 0; r < (BM + BN + NT / 8 - 1) / (NT / 8); ++r) {
                const int row = r * (NT / 8) + (tid >> 3);
                if ((BM + BN) % (NT / 8) && row >= BM + BN) break;
                const bool is_a = row < BM;
                const int g = is_a ? m0 + row : n0 + row - BM;
                const bool in = g < (is_a ? p.M : p.N) && k < k_end;
                const TI* src = is_a ? A + (size_t)g * p.lda + k : W + (size_t)g * p.ldw + k;
                gs_copy16(dst + row * GS_LD * 4, in ? (const void*)src : (const void*)W, in ? min(16, (k_end - k) * 4) : 0);
            }
        };
#pragma unroll
        for (int s = 0; s < ST - 1; ++s) {
            if (s < iters) load(s);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        for (int it = 0; it < iters; ++it) {
            asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
            __syncthreads();
            if (it + ST - 1 < iters) load(it + ST - 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
            const float* s = gs_sm + (it % ST) * T::STAGE;
            multiply(s, s + BM * GS_LD);
            if (--left == 0) { fold(done++); left = per_group; }
        }
    } else {
        constexpr int R = (BM + BN + T::NW - 1) / T::NW;         // a warp a row, a lane an element
        float reg[R];
        auto fetch = [&](int it) {
            const int k = k_begin + it * GS_BK + lane;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int row = r * T::NW + warp;
                const bool is_a = row < BM;
                const int g = is_a ? m0 + row : n0 + row - BM;
                const bool in = row < BM + BN && g < (is_a ? p.M : p.N) && k < k_end;
                reg[r] = in ? to_f32(is_a ? A[(size_t)g * p.lda + k] : W[(size_t)g * p.ldw + k]) : 0.f;
            }
        };
        if (iters) fetch(0);
        for (int it = 0; it < iters; ++it) {
            float* s = gs_sm + (it & 1) * T::STAGE;
#pragma unroll
            for (int r = 0; r < R; ++r)
                if ((BM + BN) % T::NW == 0 || r * T::NW + warp < BM + BN) s[(r * T::NW + warp) * GS_LD + lane] = reg[r];
            __syncthreads();
            if (it + 1 < iters) fetch(it + 1);
            multiply(s, s + BM * GS_LD);
            if (--left == 0) { fold(done++); left = per_group; }
        }
    }
    // (not earlier: a successor whose CTAs wait beside this one's would leave its own CTAs unevenly over the SMs)
    pdl_launch_dependents();
    while (done < groups) fold(done++);       // a group that K ends in, and those behind K
    const float* total = st[31 - __clz(groups)];

    TO* C = (TO*)p.C + (size_t)blockIdx.z * p.c_batch;
    const TI* gate = p.gate ? (const TI*)p.gate + (size_t)blockIdx.z * p.g_batch : nullptr;
    auto put = [&](int gm, int gn, float x) {
        if (gate) x /= 1.f + expf(-to_f32(gate[(size_t)gm * p.ldg + gn]));
        C[(size_t)gm * p.ldc + gn] = from_f32<TO>(x);
    };
    if (parts == 1) {
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const int gm = m0 + row0 + TY * i, gn = n0 + col0 + TX * j;
                if (gm < p.M && gn < p.N) put(gm, gn, total[i * NJ + j]);
            }
        return;
    }
    // the cluster's subtrees meet: each CTA leaves its tile in its own shared memory and adds up its share of the outputs
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) gs_sm[(row0 + TY * i) * BN + col0 + TX * j] = total[i * NJ + j];
    cluster_sync_all();
    const int share = BM * BN / parts;
    for (int e = part * share + tid; e < (part + 1) * share; e += NT) {
        const int gm = m0 + e / BN, gn = n0 + e % BN;
        if (gm >= p.M || gn >= p.N) continue;
        const uint32_t local = (uint32_t)__cvta_generic_to_shared(gs_sm + e);
        float v[GS_GROUPS];
#pragma unroll
        for (int r = 0; r < GS_GROUPS; ++r) v[r] = r < parts ? gs_peer_float(cluster_map(local, r)) : 0.f;
        const float x = parts == 2 ? v[0] + v[1] : parts == 4 ? (v[0] + v[1]) + (v[2] + v[3])
                                                 : ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        put(gm, gn, x);
    }
    cluster_sync_all();         // nobody leaves while its tile is read
}

template <typename TI, typename TO, bool ASYNC, typename T>
static int gs_launch(const GsArgs& p, int parts, int batches, cudaStream_t stream) {
    auto kernel = gemm_simt_kernel<TI, TO, ASYNC, T>;
    static AcvSmemConfig cfg;
    if (const int e = acv_ensure_smem(cfg, kernel, T::SMEM)) return e;
    const dim3 grid((p.N + T::BN - 1) / T::BN * parts, (p.M + T::BM - 1) / T::BM, batches);
    if (grid.y > 65535 || grid.z > 65535) return ACV_ERR_SIZE;
    acv_launch_cluster(PDL_GEMM, dim3(parts, 1, 1), kernel, grid, dim3(T::THREADS), T::SMEM, stream, p, parts);
    return acv_launch_status();
}

typedef GsTile<2, 1, 1, 1, 1, 6, 4, 4> GsRow1Narrow;       // 1 x 64
typedef GsTile<4, 1, 1, 1, 1, 5, 2, 4> GsRow1;             // 1 x 128
typedef GsTile<2, 1, 1, 4, 1, 6, 3, 4> GsRow4Narrow;       // 4 x 64
typedef GsTile<4, 1, 1, 4, 1, 5, 2, 4> GsRow4;             // 4 x 128
typedef GsTile<4, 1, 1, 8, 1, 4, 2, 4> GsRow8;             // 8 x 128
typedef GsTile<4, 1, 2, 8, 2, 4, 2, 4> GsRow16;            // 16 x 128
typedef GsTile<4, 2, 4, 4, 4, 4, 3, 4> GsRow32;            // 32 x 64
typedef GsTile<8, 4, 2, 8, 2, 3, 3, 2> GsSquare64;         // 64 x 64
typedef GsTile<8, 4, 2, 8, 4, 3, 2, 2> GsWide64;           // 64 x 128
// 64 x 64 with rows by way of registers, which three CTAs to an SM have not enough of
typedef GsTile<8, 4, 2, 8, 2, 2, 2, 2> GsSquare64Loads;

// Which tile and how many CTAs to a tile: the way whose busiest SM is done first.  `one` and `full`: cycles for 32 k of a
// CTA that has its SM to itself and of as many as fit beside each other, measured (a tile's cycles for few rows are its
// weights' bytes at the memory's speed).  Rows of a tile that hold nothing cost what full ones do, so the narrowest tile
// that holds all rows is the only one asked for up to 16 of them.
struct GsWay { int bm, bn, resident, one, full; };
static const GsWay GS_WAYS[10] = {{1, 64, 4, 400, 1420}, {1, 128, 2, 760, 1420}, {4, 64, 3, 420, 1275}, {4, 128, 2, 800, 1480},
                                 {8, 128, 2, 1100, 1900}, {16, 128, 2, 1700, 2750}, {32, 64, 3, 1800, 3400}, {64, 64, 3, 2400, 5850},
                                 {64, 128, 2, 4100, 6500}, {64, 64, 2, 2400, 4125}};

// What is counted of K: the stages of the CTA that has most of them (groups behind K have none, and a cluster that K does not
// reach is no help: 64 rows of 64 x 64 took 11 us as two CTAs of which one was empty, 5 as one).
static double gs_cost(const GsWay& g, int c, int M, int N, int K, int batches, int sms) {
    const int gl = gs_group_length(K), stages = min((K + GS_BK - 1) / GS_BK, GS_GROUPS / c * (gl / GS_BK));
    const long long tiles = (long long)((M + g.bm - 1) / g.bm) * ((N + g.bn - 1) / g.bn) * batches;
    const long long each = (tiles * c + sms - 1) / sms, rounds = each / g.resident, rest = each % g.resident;
    const double iter = rounds * (double)g.full + (rest ? g.one + (rest - 1) * (double)(g.full - g.one) / (g.resident - 1) : 0.);
    return iter * stages + (rounds + (rest > 0)) * 2500.;         // a CTA's first stages and its way out
}

static void gs_plan(int M, int N, int K, int batches, int sms, int first, int last, int* way, int* parts) {
    double best = -1.;
    for (int w = first; w <= last; ++w)
        for (int c = 1; c <= GS_GROUPS; c *= 2) {
            const double t = gs_cost(GS_WAYS[w], c, M, N, K, batches, sms);
            if (best < 0. || t < best) { best = t; *way = w; *parts = c; }
        }
}

static int gs_multiprocessors(int* sms) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, device);
    return (int)e;
}

static int gs_run_async(const GsArgs& p, int batches, cudaStream_t stream) {
    int sms = 0;
    if (const int e = gs_multiprocessors(&sms)) return e;
    int way = 0, parts = 1;
    const int M = p.M, first = M <= 1 ? 0 : M <= 4 ? 2 : M <= 8 ? 4 : M <= 16 ? 5 : 6, last = M <= 1 ? 1 : M <= 4 ? 3 : M <= 8 ? 4 : M <= 16 ? 5 : 8;
    gs_plan(M, p.N, p.K, batches, sms, first, last, &way, &parts);
    switch (way) {
        case 0: return gs_launch<float, float, true, GsRow1Narrow>(p, parts, batches, stream);
        case 1: return gs_launch<float, float, true, GsRow1>(p, parts, batches, stream);
        case 2: return gs_launch<float, float, true, GsRow4Narrow>(p, parts, batches, stream);
        case 3: return gs_launch<float, float, true, GsRow4>(p, parts, batches, stream);
        case 4: return gs_launch<float, float, true, GsRow8>(p, parts, batches, stream);
        case 5: return gs_launch<float, float, true, GsRow16>(p, parts, batches, stream);
        case 6: return gs_launch<float, float, true, GsRow32>(p, parts, batches, stream);
        case 7: return gs_launch<float, float, true, GsSquare64>(p, parts, batches, stream);
        default: return gs_launch<float, float, true, GsWide64>(p, parts, batches, stream);
    }
}

// operands without 16-byte pieces, or bfloat16 (a fallback of odd sizes): two tiles
template <typename TI, typename TO>
static int gs_run_any(const GsArgs& p, int batches, cudaStream_t stream) {
    int sms = 0;
    if (const int e = gs_multiprocessors(&sms)) return e;
    int way = 0, parts = 1;
    gs_plan(p.M, p.N, p.K, batches, sms, p.M <= 4 ? 3 : 9, p.M <= 4 ? 3 : 9, &way, &parts);
    return p.M <= 4 ? gs_launch<TI, TO, false, GsRow4>(p, parts, batches, stream) : gs_launch<TI, TO, false, GsSquare64Loads>(p, parts, batches, stream);
}

// in_dtype: type of A and W; out_dtype: type of C.  `batches` products side by side (a head's own matrix for each
// head, say): product b reads A + b a_batch, W + b w_batch and writes C + b c_batch (strides in elements).  gate (of
// in_dtype, C's shape, or null): C is multiplied by its sigmoid, in float.
ACV_API int acv_gemm_simt_batched(const void* A, int lda, long long a_batch, const void* W, int ldw, long long w_batch,
                                  void* C, int ldc, long long c_batch, int M, int N, int K, int batches, int in_dtype,
                                  int out_dtype, const void* gate, int ldg, long long g_batch, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batches <= 0) return 0;
    if (K <= 0 || batches > 65535) return ACV_ERR_SIZE;
    const GsArgs p = {A, W, gate, C, lda, ldw, ldc, ldg, M, N, K, a_batch, w_batch, c_batch, g_batch};
    if (in_dtype == ACV_F32 && out_dtype == ACV_F32) {
        // 16-byte copies: both operands' starts, rows and batches on 16-byte boundaries (a row's end need not be one)
        const bool pieces = ((uintptr_t)A | (uintptr_t)W) % 16 == 0 && (lda | ldw) % 4 == 0 && (a_batch | w_batch) % 4 == 0;
        if (K >= GF_MIN_K) {
            int sms = 0;
            if (const int e = gs_multiprocessors(&sms)) return e;
            const GfArgs q = {(const float*)A, (const float*)W, (const float*)gate, (float*)C, status, lda, ldw, ldc, ldg, M, N, K,
                              a_batch, w_batch, c_batch, g_batch};
            return gf_run(q, pieces, batches, sms, stream);
        }
        return pieces ? gs_run_async(p, batches, stream) : gs_run_any<float, float>(p, batches, stream);
    }
    if (in_dtype == ACV_BF16 && out_dtype == ACV_F32) return gs_run_any<bf16, float>(p, batches, stream);
    if (in_dtype == ACV_BF16 && out_dtype == ACV_BF16) return gs_run_any<bf16, bf16>(p, batches, stream);
    return ACV_ERR_DTYPE;
}

ACV_API int acv_gemm_simt(const void* A, int lda, const void* W, int ldw, void* C, int ldc, int M, int N, int K,
                          int in_dtype, int out_dtype, int* status, cudaStream_t stream) {
    return acv_gemm_simt_batched(A, lda, 0, W, ldw, 0, C, ldc, 0, M, N, K, 1, in_dtype, out_dtype, nullptr, 0, 0, status, stream);
}
