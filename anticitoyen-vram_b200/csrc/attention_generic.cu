// Paged causal attention, generic form: any number of query tokens per request,
// any head size up to 1024 (value rows may have another size than key rows, DV != D, up to 512; with v_pages == k_pages
// and v_row = D the values are the first DV elements of the key rows themselves: one kept row per token serves as key
// and as value, as a latent that every head reads does), float or bfloat16 pages.  It is the 32-bit path of the engine
// and the fallback of the bfloat16 path for head sizes and options the tensor-core kernels do not take.
//
// Query-head h reads kv-head h / (NH/NKV) (acvram/engine/layers.py:1012-1017).
// The keys of the step's own tokens are already in the pages, so the query at
// absolute position p sees the keys j <= p, and with a window w > 0 only
// j > p - w (mask aligned to absolute positions, acvram/engine/layers.py:1020-1041); with keep_first = f > 0 the
// first f keys of the request stay visible to every later query, whatever the window (they keep their own
// positions: nothing is shifted).
// s = scale * q.k - slope_h * (p - j) (slopes: one per query head, or none); with sinks (one number per query head) the
// softmax's denominator also holds exp(sink_h), which has no key and no value.  Softmax over the visible keys with a running maximum and sum in
// 32-bit (acvram/kernels/acvram_kernels.cu:993-1146 has the same recurrence).  With a gate (rows like the result's) the
// result is multiplied by sigmoid(gate) before it is rounded.
//
// Three kernels.  attn_rows_kernel: 64 (token, head) rows of a request against tiles of 32 keys, for portions of prompts.
// attn_token_kernel: the query heads of one token and kv-head against its keys, which 8 warps and up to 8 CTAs share, for
// requests that bring one token and for steps of a few tokens.  attn_generic_kernel: one warp per (token, head), for head
// sizes over 256 or of no 4-element pieces.  In a step of many tokens the first two run one after the other and each
// leaves the other's tokens alone.  Measured in float32 with 16 heads on 8 kv-heads of 128 (microseconds, one warp per
// (token, head) before -> now): 696 tokens of three portions 825 -> 130, 3 tokens at contexts of 300-500 429 -> 22.
#include "common.cuh"
#include <type_traits>

#define AG_WARPS 4

template <typename T, int NR>
__global__ void attn_generic_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out, int out_stride,
                                    const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                                    const int* __restrict__ positions, const int* __restrict__ seq_of_token,
                                    const int* __restrict__ block_table, int bt_stride, const int* __restrict__ bt_rows, int NH, int NKV, int D, int DV,
                                    int page_size, int num_pages, float scale, int window, int keep_first, int v_row,
                                    const float* __restrict__ sinks, const float* __restrict__ slopes,
                                    const T* __restrict__ gate, int gate_stride) {
    extern __shared__ float sm_all[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.y * AG_WARPS + warp;
    const int t = blockIdx.x;
    if (h >= NH) return;
    float* qs = sm_all + warp * D;
    const int kvh = h / (NH / NKV);
    const int p = positions[t];
    const int seq = seq_of_token[t];
    const int* bt = block_table + (size_t)(bt_rows ? bt_rows[seq] : seq) * bt_stride;
    const T* qrow = q + (size_t)t * q_stride + (size_t)h * D;
    for (int e = lane; e < D; e += 32) qs[e] = to_f32(qrow[e]) * scale;
    __syncwarp();

    float acc[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) acc[r] = 0.f;
    float m = -INFINITY, l = 0.f;
    const float slope = slopes ? slopes[h] : 0.f;
    const int lo = window > 0 ? max(0, p - window + 1) : 0;
    // two runs of keys: the kept first ones that the window has passed, [0, min(keep_first, lo)), then [lo, p]
    const int kept = window > 0 ? min(max(keep_first, 0), lo) : 0;

    for (int run = kept > 0 ? 0 : 1; run < 2; ++run) {
    const int j_begin = run == 0 ? 0 : lo, j_last = run == 0 ? kept - 1 : p;
    for (int j0 = j_begin; j0 <= j_last; j0 += 32) {
        const int j = j0 + lane;
        bool valid = j <= j_last;
        long long row = 0;
        if (valid) {
            const int pg = bt[j / page_size];
            valid = pg >= 0 && pg < num_pages;
            row = ((long long)pg * NKV + kvh) * page_size + (j % page_size);
        }
        float s = -INFINITY;
        if (valid) {
            const T* kr = k_pages + row * D;
            float dot = 0.f;
            if ((D & 7) == 0 && sizeof(T) == 2) {       // rows of 16-byte pieces: eight elements a load
                const uint4* kv = reinterpret_cast<const uint4*>(kr);
                for (int e = 0; e < D; e += 8) {
                    const uint4 u = kv[e >> 3];
                    const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        dot = fmaf(qs[e + 2 * i], __uint_as_float(w4[i] << 16), dot);
                        dot = fmaf(qs[e + 2 * i + 1], __uint_as_float(w4[i] & 0xffff0000u), dot);
                    }
                }
            } else {
                for (int e = 0; e < D; ++e) dot = fmaf(qs[e], to_f32(kr[e]), dot);
            }
            s = dot - slope * (float)(p - j);
        }
        const float tmax = warp_max(s);
        if (tmax == -INFINITY) continue;  // uniform: no readable key in this tile
        const float m_new = fmaxf(m, tmax);
        const float alpha = expf(m - m_new);
        const float pl = valid ? expf(s - m_new) : 0.f;
        l = l * alpha + warp_sum(pl);
        m = m_new;
#pragma unroll
        for (int r = 0; r < NR; ++r) acc[r] *= alpha;
        const int n_in_tile = min(32, j_last - j0 + 1);
        for (int kk = 0; kk < n_in_tile; ++kk) {
            const float pk = __shfl_sync(0xffffffffu, pl, kk);
            const long long ro = __shfl_sync(0xffffffffu, row, kk);
            if (pk == 0.f) continue;
            const T* vr = v_pages + ro * v_row;
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const int e = lane + 32 * r;
                if (e < DV) acc[r] = fmaf(pk, to_f32(vr[e]), acc[r]);
            }
        }
    }
    }
    if (sinks) {        // a score without key or value: it takes its share of the weights and adds nothing
        const float sink = sinks[h];
        const float m_new = fmaxf(m, sink);
        const float alpha = expf(m - m_new);
        l = l * alpha + expf(sink - m_new);
#pragma unroll
        for (int r = 0; r < NR; ++r) acc[r] *= alpha;
    }
    T* orow = out + (size_t)t * out_stride + (size_t)h * DV;
    const float inv_l = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const int e = lane + 32 * r;
        if (e >= DV) continue;
        float o = acc[r] * inv_l;
        if (gate) o *= 1.f / (1.f + expf(-to_f32(gate[(size_t)t * gate_stride + (size_t)h * DV + e])));
        orow[e] = from_f32<T>(o);
    }
}

// ----------------------------------------------------------------------------- shared by the two tiled kernels
struct AgArgs {
    const void *q, *k_pages, *v_pages, *gate;
    void* out;
    const int *positions, *seq_of_token, *block_table, *bt_rows;
    const float *sinks, *slopes;
    int q_stride, out_stride, gate_stride, bt_stride, T, NH, NKV, D, DV, page_size, num_pages, window, keep_first, v_row;
    float scale;
};

__device__ __forceinline__ float4 ag_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ag_load4(const bf16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
// a token whose neighbours in the batch belong to other requests
__device__ __forceinline__ bool ag_alone(const int* seq, int t, int T) {
    return (t == 0 || seq[t - 1] != seq[t]) && (t + 1 >= T || seq[t + 1] != seq[t]);
}
// the row of key j of a request in the pages of a kv-head, or -1 where there is no page
__device__ __forceinline__ long long ag_row(const AgArgs& a, const int* bt, int kvh, int j) {
    const int pg = bt[j / a.page_size];
    return pg >= 0 && pg < a.num_pages ? ((long long)pg * a.NKV + kvh) * a.page_size + j % a.page_size : -1;
}
__device__ __forceinline__ bool ag_sees(const AgArgs& a, int p, int j) {
    return j <= p && (a.window <= 0 || j > p - a.window || j < a.keep_first);
}
template <typename T>
__device__ __forceinline__ void ag_put(const AgArgs& a, int t, int h, int e, float o) {
    if (a.gate) o *= 1.f / (1.f + expf(-to_f32(((const T*)a.gate)[(size_t)t * a.gate_stride + (size_t)h * a.DV + e])));
    ((T*)a.out)[(size_t)t * a.out_stride + (size_t)h * a.DV + e] = from_f32<T>(o);
}
// a key's weight against the maximum so far: 0 for a score of -inf, whatever the maximum; a score that is no number (the
// maximum passes it over) gives a weight that is none, and so does +inf: the sums and the result are none then
__device__ __forceinline__ float ag_weight(float x, float m) { return x == -INFINITY ? 0.f : expf(x - m); }
__device__ __forceinline__ float ag_peer(const float* local, int rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_map((uint32_t)__cvta_generic_to_shared(local), rank)) : "memory");
    return v;
}

// ----------------------------------------------------------------------------- rows of a portion
// A CTA: 64 / (NH/NKV) tokens of the flat batch times the heads of one kv-head, eight rows to a warp; the requests among
// the tokens one after the other (a tile of a portion has one).  Scores: a lane a key, so a 16-byte read of 32 key rows
// moves 512 different bytes and a row's queries are one address; values: a lane four columns.  Bound by the chains of
// shared-memory reads (9 to 32 multiply-adds of a warp for the scores), hence eight rows a warp and not fewer: 32 rows and
// four warps to a CTA were slower (156 against 125 us, 696 tokens of three portions), and so was bringing the next tile
// under this one's arithmetic (144 us: its registers are what the reads are hidden with).
#define AR_ROWS 64
#define AR_KEYS 32
#define AR_WARP_ROWS 8
#define AR_THREADS 256

template <typename T, int VC>       // VC: runs of 128 value columns
__global__ void __launch_bounds__(AR_THREADS, VC == 1 ? 2 : 1)
attn_rows_kernel(const AgArgs a, int skip_alone) {
    extern __shared__ __align__(16) float ar_sm[];
    const int G = a.NH / a.NKV, D = a.D, DV = a.DV, ldk = D + 4;
    const int tokens = AR_ROWS / G > 0 ? AR_ROWS / G : 1, heads = G < AR_ROWS ? G : AR_ROWS;
    float* qs = ar_sm;                              // [64][D + 4], scaled
    float* ks = qs + AR_ROWS * ldk;                 // [32][D + 4]
    float* vs = ks + AR_KEYS * ldk;                 // [32][DV]
    float* ps = vs + AR_KEYS * DV;                  // [8 warps][32 keys][8 rows]
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kvh = blockIdx.y, h0 = kvh * G + blockIdx.z * heads, n_heads = min(heads, G - (int)blockIdx.z * heads);
    const int t_begin = blockIdx.x * tokens, t_end = min(a.T, t_begin + tokens);
    float* pw = ps + warp * AR_KEYS * AR_WARP_ROWS;

    for (int t0 = t_begin; t0 < t_end;) {
        const int seq = a.seq_of_token[t0];
        int t1 = t0 + 1;
        while (t1 < t_end && a.seq_of_token[t1] == seq) ++t1;
        if (skip_alone && t1 == t0 + 1 && ag_alone(a.seq_of_token, t0, a.T)) { t0 = t1; continue; }
        const int n = t1 - t0, rows = n * n_heads;      // row r: token t0 + r / n_heads, head h0 + r % n_heads
        const int* bt = a.block_table + (size_t)(a.bt_rows ? a.bt_rows[seq] : seq) * a.bt_stride;
        __syncthreads();
        for (int i = tid; i < AR_ROWS * (D / 4); i += AR_THREADS) {
            const int r = i / (D / 4), c = (i % (D / 4)) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < rows) {
                v = ag_load4((const T*)a.q + (size_t)(t0 + r / n_heads) * a.q_stride + (size_t)(h0 + r % n_heads) * D + c);
                v.x *= a.scale; v.y *= a.scale; v.z *= a.scale; v.w *= a.scale;
            }
            *reinterpret_cast<float4*>(qs + r * ldk + c) = v;
        }
        int lo = 0x7fffffff, last = -1, hi_lo = 0;      // keys any row sees: [lo, last], and the kept first ones before lo
        for (int t = t0; t < t1; ++t) {
            const int p = a.positions[t], l = a.window > 0 ? max(0, p - a.window + 1) : 0;
            lo = min(lo, l); last = max(last, p); hi_lo = max(hi_lo, l);
        }
        const int kept = a.window > 0 ? min(min(max(a.keep_first, 0), hi_lo), lo) : 0;
        const int r0 = warp * AR_WARP_ROWS;
        int pos[AR_WARP_ROWS];
        float slope[AR_WARP_ROWS], m[AR_WARP_ROWS], l[AR_WARP_ROWS];
        float acc[AR_WARP_ROWS][4 * VC];
#pragma unroll
        for (int i = 0; i < AR_WARP_ROWS; ++i) {
            const bool in = r0 + i < rows;
            pos[i] = in ? a.positions[t0 + (r0 + i) / n_heads] : -1;
            slope[i] = in && a.slopes ? a.slopes[h0 + (r0 + i) % n_heads] : 0.f;
            m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
            for (int c = 0; c < 4 * VC; ++c) acc[i][c] = 0.f;
        }
        for (int run = kept > 0 ? 0 : 1; run < 2; ++run) {
            const int j_end = run == 0 ? kept : last + 1;
            for (int j0 = run == 0 ? 0 : lo; j0 < j_end; j0 += AR_KEYS) {
                const int nk = min(AR_KEYS, j_end - j0);
                // a lane looks up one key's row; a warp brings every eighth key, all of its loads on their way together
                const long long my_row = lane < nk ? ag_row(a, bt, kvh, j0 + lane) : -1;
                float4 kx[AR_KEYS / 8][VC], vx[AR_KEYS / 8][VC];
                bool odd = false;       // a value that is no finite number: a weight of 0 must not meet it
#pragma unroll
                for (int i = 0; i < AR_KEYS / 8; ++i) {
                    const long long row = __shfl_sync(0xffffffffu, my_row, i * 8 + warp);
#pragma unroll
                    for (int c = 0; c < VC; ++c) {
                        const int e = c * 128 + lane * 4;
                        kx[i][c] = row >= 0 && e < D ? ag_load4((const T*)a.k_pages + row * D + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                        vx[i][c] = row >= 0 && e < DV ? ag_load4((const T*)a.v_pages + row * a.v_row + e) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                }
                __syncthreads();        // the tile before is done with
#pragma unroll
                for (int i = 0; i < AR_KEYS / 8; ++i)
#pragma unroll
                    for (int c = 0; c < VC; ++c) {
                        const int e = c * 128 + lane * 4;
                        const float4 v = vx[i][c];
                        odd |= !(fabsf(v.x) + fabsf(v.y) + fabsf(v.z) + fabsf(v.w) < INFINITY);
                        if (e < D) *reinterpret_cast<float4*>(ks + (i * 8 + warp) * ldk + e) = kx[i][c];
                        if (e < DV) *reinterpret_cast<float4*>(vs + (i * 8 + warp) * DV + e) = v;
                    }
                odd = __syncthreads_or(odd);
                float s[AR_WARP_ROWS];
#pragma unroll
                for (int i = 0; i < AR_WARP_ROWS; ++i) s[i] = 0.f;
#pragma unroll 4
                for (int d = 0; d < D; d += 4) {
                    const float4 k = *reinterpret_cast<const float4*>(ks + lane * ldk + d);
#pragma unroll
                    for (int i = 0; i < AR_WARP_ROWS; ++i) {
                        const float4 q = *reinterpret_cast<const float4*>(qs + (r0 + i) * ldk + d);
                        s[i] = fmaf(q.x, k.x, s[i]); s[i] = fmaf(q.y, k.y, s[i]);
                        s[i] = fmaf(q.z, k.z, s[i]); s[i] = fmaf(q.w, k.w, s[i]);
                    }
                }
                const int j = j0 + lane;
#pragma unroll
                for (int i = 0; i < AR_WARP_ROWS; ++i) {
                    const bool seen = my_row >= 0 && ag_sees(a, pos[i], j);
                    const float x = seen ? s[i] - slope[i] * (float)(pos[i] - j) : -INFINITY;
                    const float m_new = fmaxf(m[i], warp_max(x));
                    const float alpha = m_new == -INFINITY ? 1.f : expf(m[i] - m_new);
                    const float w = ag_weight(x, m_new);
                    l[i] = l[i] * alpha + w;            // a lane's share of the sum
                    m[i] = m_new;
#pragma unroll
                    for (int c = 0; c < 4 * VC; ++c) acc[i][c] *= alpha;
                    s[i] = w;
                }
                *reinterpret_cast<float4*>(pw + lane * 8) = make_float4(s[0], s[1], s[2], s[3]);
                *reinterpret_cast<float4*>(pw + lane * 8 + 4) = make_float4(s[4], s[5], s[6], s[7]);
                __syncwarp();
                auto weigh = [&](auto guard) {
#pragma unroll
                    for (int c = 0; c < VC; ++c) {
                        const int col = c * 128 + lane * 4;
                        if (col >= DV) continue;
#pragma unroll 4
                        for (int k = 0; k < nk; ++k) {
                            const float4 v = *reinterpret_cast<const float4*>(vs + k * DV + col);
                            const float4 w0 = *reinterpret_cast<const float4*>(pw + k * 8), w1 = *reinterpret_cast<const float4*>(pw + k * 8 + 4);
                            const float w[AR_WARP_ROWS] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                            for (int i = 0; i < AR_WARP_ROWS; ++i) {
                                if (decltype(guard)::value && w[i] == 0.f) continue;
                                acc[i][c * 4 + 0] = fmaf(w[i], v.x, acc[i][c * 4 + 0]);
                                acc[i][c * 4 + 1] = fmaf(w[i], v.y, acc[i][c * 4 + 1]);
                                acc[i][c * 4 + 2] = fmaf(w[i], v.z, acc[i][c * 4 + 2]);
                                acc[i][c * 4 + 3] = fmaf(w[i], v.w, acc[i][c * 4 + 3]);
                            }
                        }
                    }
                };
                if (odd) weigh(std::true_type()); else weigh(std::false_type());
                __syncwarp();
            }
        }
#pragma unroll
        for (int i = 0; i < AR_WARP_ROWS; ++i) {
            const int r = r0 + i;
            float sum = warp_sum(l[i]), f = 1.f;
            if (r >= rows) continue;
            const int t = t0 + r / n_heads, h = h0 + r % n_heads;
            if (a.sinks) {      // a score without key or value: it takes its share of the weights and adds nothing
                const float sink = a.sinks[h], m_new = fmaxf(m[i], sink);
                f = expf(m[i] - m_new);
                sum = sum * f + expf(sink - m_new);
            }
            const float inv = sum == 0.f ? 0.f : f / sum;
#pragma unroll
            for (int c = 0; c < 4 * VC; ++c) {
                const int e = (c / 4) * 128 + lane * 4 + c % 4;
                if (e < DV) ag_put<T>(a, t, h, e, acc[i][c] * inv);
            }
        }
        t0 = t1;
    }
    pdl_launch_dependents();
}

// ----------------------------------------------------------------------------- one token
// A cluster of CTAs shares the keys of one token and kv-head, its 8 warps take batches of 32 keys in turn: eight lanes to a
// key for the scores (four keys a load), a lane four columns for the values; RG query heads ride on each key and value
// that is read.  Bound by the pages' stream and its latency.  The warps' partial results meet in shared memory, the CTAs'
// in rank order through the cluster's.
#define AT1_WARPS 8
#define AG_STRIDE 8      // tokens that a CTA looks at in a step of many tokens

template <typename T, int RG, int VC>
__global__ void __launch_bounds__(AT1_WARPS * 32)
attn_token_kernel(const AgArgs a, int parts, int only_alone) {
    __shared__ float sm_m[AT1_WARPS][RG], sm_l[AT1_WARPS][RG], tot_m[RG], tot_l[RG];
    __shared__ __align__(16) float sm_w[AT1_WARPS][32][RG];
    extern __shared__ __align__(16) float at_o[];      // [8 warps][RG][DV], then [RG][DV] of the CTA in front
    pdl_launch_dependents();
    pdl_wait();
    const int D = a.D, DV = a.DV, G = a.NH / a.NKV;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sub = lane & 7, grp = lane >> 3;
    const int part = blockIdx.x % parts;
    const int chunks = (G + RG - 1) / RG, kvh = blockIdx.y / chunks, h0 = kvh * G + (blockIdx.y % chunks) * RG;
    const int n_heads = min(RG, (kvh + 1) * G - h0);
    // one token a cluster; in a step of many tokens, without clusters, those of the tokens x, x + gridDim.x .. that are alone
    // (bit i: token x + i gridDim.x; all asked for at once, since a look is a round trip to memory)
    uint32_t mine = 1;
    if (only_alone) {
        const int cand = blockIdx.x + lane * gridDim.x;
        mine = __ballot_sync(0xffffffffu, lane < AG_STRIDE && cand < a.T && ag_alone(a.seq_of_token, cand, a.T));
    }
    for (; mine; mine &= mine - 1) {
        const int t = only_alone ? blockIdx.x + (__ffs(mine) - 1) * gridDim.x : blockIdx.x / parts;
        if (only_alone) __syncthreads();        // the token before is done with the shared memory
        const int p = a.positions[t], seq = a.seq_of_token[t];
        const int* bt = a.block_table + (size_t)(a.bt_rows ? a.bt_rows[seq] : seq) * a.bt_stride;
        const int lo = a.window > 0 ? max(0, p - a.window + 1) : 0;
        const int kept = a.window > 0 ? min(max(a.keep_first, 0), lo) : 0;
        const int total = kept + p + 1 - lo;        // visible keys: the kept first ones, then [lo, p]

        // queries: lane `sub` of a key's eight holds elements sub*4 + 32 c
        constexpr int QC = VC * 4;
        float4 q[RG][QC];
#pragma unroll
        for (int r = 0; r < RG; ++r)
#pragma unroll
            for (int c = 0; c < QC; ++c) {
                const int e = sub * 4 + 32 * c;
                q[r][c] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < n_heads && e < D) {
                    q[r][c] = ag_load4((const T*)a.q + (size_t)t * a.q_stride + (size_t)(h0 + r) * D + e);
                    q[r][c].x *= a.scale; q[r][c].y *= a.scale; q[r][c].z *= a.scale; q[r][c].w *= a.scale;
                }
            }
        float m[RG], l[RG], acc[RG][4 * VC];
#pragma unroll
        for (int r = 0; r < RG; ++r) {
            m[r] = -INFINITY; l[r] = 0.f;
#pragma unroll
            for (int c = 0; c < 4 * VC; ++c) acc[r][c] = 0.f;
        }
        for (int b = (part * AT1_WARPS + warp) * 32; b < total; b += parts * AT1_WARPS * 32) {
            const int i = b + lane, j = i < kept ? i : lo + i - kept;
            const long long row = i < total ? ag_row(a, bt, kvh, j) : -1;
#pragma unroll
            for (int g = 0; g < 8; ++g) {           // keys g*4 .. g*4 + 3 of the batch, eight lanes each
                const long long kr_row = __shfl_sync(0xffffffffu, row, g * 4 + grp);
                const T* kr = (const T*)a.k_pages + kr_row * D;
                float s[RG];
#pragma unroll
                for (int r = 0; r < RG; ++r) s[r] = 0.f;
#pragma unroll
                for (int c = 0; c < QC; ++c) {
                    const int e = sub * 4 + 32 * c;
                    const float4 k = kr_row >= 0 && e < D ? ag_load4(kr + e) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int r = 0; r < RG; ++r) {
                        s[r] = fmaf(q[r][c].x, k.x, s[r]); s[r] = fmaf(q[r][c].y, k.y, s[r]);
                        s[r] = fmaf(q[r][c].z, k.z, s[r]); s[r] = fmaf(q[r][c].w, k.w, s[r]);
                    }
                }
#pragma unroll
                for (int r = 0; r < RG; ++r) {
                    s[r] += __shfl_xor_sync(0xffffffffu, s[r], 1);
                    s[r] += __shfl_xor_sync(0xffffffffu, s[r], 2);
                    s[r] += __shfl_xor_sync(0xffffffffu, s[r], 4);
                    if (sub == 0) sm_w[warp][g * 4 + grp][r] = s[r];
                }
            }
            __syncwarp();
#pragma unroll
            for (int r = 0; r < RG; ++r) {
                const float slope = a.slopes && r < n_heads ? a.slopes[h0 + r] : 0.f;
                const float x = row >= 0 ? sm_w[warp][lane][r] - slope * (float)(p - j) : -INFINITY;
                const float m_new = fmaxf(m[r], warp_max(x));
                const float alpha = m_new == -INFINITY ? 1.f : expf(m[r] - m_new);
                const float w = ag_weight(x, m_new);
                l[r] = l[r] * alpha + w;
                m[r] = m_new;
#pragma unroll
                for (int c = 0; c < 4 * VC; ++c) acc[r][c] *= alpha;
                sm_w[warp][lane][r] = w;
            }
            __syncwarp();
            const int nk = min(32, total - b);
#pragma unroll
            for (int c = 0; c < VC; ++c) {
                const int col = c * 128 + lane * 4;
#pragma unroll 8
                for (int k = 0; k < nk; ++k) {
                    const long long vr_row = __shfl_sync(0xffffffffu, row, k);
                    const float4 v = vr_row >= 0 && col < DV ? ag_load4((const T*)a.v_pages + vr_row * a.v_row + col) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int r = 0; r < RG; ++r) {
                        const float w = sm_w[warp][k][r];
                        if (w == 0.f) continue;     // (a weight of 0 must not meet a value that is no finite number)
                        acc[r][c * 4 + 0] = fmaf(w, v.x, acc[r][c * 4 + 0]);
                        acc[r][c * 4 + 1] = fmaf(w, v.y, acc[r][c * 4 + 1]);
                        acc[r][c * 4 + 2] = fmaf(w, v.z, acc[r][c * 4 + 2]);
                        acc[r][c * 4 + 3] = fmaf(w, v.w, acc[r][c * 4 + 3]);
                    }
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int r = 0; r < RG; ++r) {
            const float sum = warp_sum(l[r]);
            if (lane == 0) { sm_m[warp][r] = m[r]; sm_l[warp][r] = sum; }
#pragma unroll
            for (int c = 0; c < VC; ++c)
                if (c * 128 + lane * 4 < DV)
                    *reinterpret_cast<float4*>(at_o + (warp * RG + r) * DV + c * 128 + lane * 4) =
                        make_float4(acc[r][c * 4], acc[r][c * 4 + 1], acc[r][c * 4 + 2], acc[r][c * 4 + 3]);
        }
        __syncthreads();
        if (tid < RG) {
            float mx = -INFINITY, sum = 0.f;
            for (int w = 0; w < AT1_WARPS; ++w) mx = fmaxf(mx, sm_m[w][tid]);
            for (int w = 0; w < AT1_WARPS; ++w) {
                const float f = sm_m[w][tid] == -INFINITY ? 0.f : expf(sm_m[w][tid] - mx);
                sum += sm_l[w][tid] * f;
                sm_m[w][tid] = f;       // from here on the warp's factor
            }
            tot_m[tid] = mx; tot_l[tid] = sum;
        }
        __syncthreads();
        for (int e = tid; e < RG * DV; e += AT1_WARPS * 32) {
            float o = 0.f;
            for (int w = 0; w < AT1_WARPS; ++w) {
                const float f = sm_m[w][e / DV];
                if (f != 0.f) o = fmaf(f, at_o[w * RG * DV + e], o);
            }
            at_o[e] = o;                // (the thread alone reads and writes column e of the warps' rows)
        }
        if (parts > 1) cluster_sync_all(); else __syncthreads();
        const int share = (RG * DV + parts - 1) / parts;
        for (int e = part * share + tid; e < min(RG * DV, (part + 1) * share); e += AT1_WARPS * 32) {
            const int r = e / DV;
            if (r >= n_heads) continue;
            float mx = tot_m[r], sum = tot_l[r], o = at_o[e];
            if (parts > 1) {
                mx = -INFINITY; sum = 0.f; o = 0.f;
                for (int c = 0; c < parts; ++c) mx = fmaxf(mx, ag_peer(tot_m + r, c));
                for (int c = 0; c < parts; ++c) {
                    const float pm = ag_peer(tot_m + r, c), pl = ag_peer(tot_l + r, c), po = ag_peer(at_o + e, c);
                    const float f = pm == -INFINITY ? 0.f : expf(pm - mx);
                    sum = fmaf(pl, f, sum);
                    if (f != 0.f) o = fmaf(po, f, o);
                }
            }
            if (a.sinks) {
                const float sink = a.sinks[h0 + r], m_new = fmaxf(mx, sink);
                const float f = expf(mx - m_new);
                sum = sum * f + expf(sink - m_new);
                o *= f;
            }
            ag_put<T>(a, t, h0 + r, e % DV, sum == 0.f ? 0.f : o / sum);
        }
        if (parts > 1) cluster_sync_all();      // nobody leaves while its results are read
    }
}

template <typename T, int RG, int VC>
static int launch_token(const AgArgs& a, int parts, int only_alone, cudaStream_t stream) {
    auto kernel = attn_token_kernel<T, RG, VC>;
    const int smem = AT1_WARPS * RG * a.DV * 4;
    static AcvSmemConfig cfg;
    if (const int e = acv_ensure_smem(cfg, kernel, smem)) return e;
    const int G = a.NH / a.NKV, x = only_alone ? (a.T + AG_STRIDE - 1) / AG_STRIDE : a.T * parts;
    acv_launch_cluster(PDL_ATTN, dim3(parts, 1, 1), kernel, dim3(x, a.NKV * ((G + RG - 1) / RG)), dim3(AT1_WARPS * 32), smem, stream, a, parts, only_alone);
    return acv_launch_status();
}

template <typename T, int VC>
static int launch_rows(const AgArgs& a, int skip_alone, cudaStream_t stream) {
    auto kernel = attn_rows_kernel<T, VC>;
    const int smem = ((AR_ROWS + AR_KEYS) * (a.D + 4) + AR_KEYS * a.DV + AR_ROWS * AR_KEYS) * 4;
    static AcvSmemConfig cfg;
    if (const int e = acv_ensure_smem(cfg, kernel, smem)) return e;
    const int G = a.NH / a.NKV, tokens = AR_ROWS / G > 0 ? AR_ROWS / G : 1, heads = G < AR_ROWS ? G : AR_ROWS;
    acv_launch(PDL_ATTN, kernel, dim3((a.T + tokens - 1) / tokens, a.NKV, (G + heads - 1) / heads), dim3(AR_THREADS), smem, stream, a, skip_alone);
    return acv_launch_status();
}

// Steps of up to AG_FEW tokens: every token by itself, with as many CTAs to a token and kv-head as put the SMs to work
// (a short context's CTAs without keys leave at the merge).  More tokens: rows of portions, then the tokens that are alone
// (a portion's 64 rows read each key once for all of them, one token's warps once for its own heads).
#define AG_FEW 64
template <typename T>
static int launch_tiled(const AgArgs& a, cudaStream_t stream) {
    const int G = a.NH / a.NKV, wide = (a.D > 128 || a.DV > 128) ? 2 : 1;
    const bool few = a.T <= AG_FEW;
    if (!few) {
        const int e = wide == 1 ? launch_rows<T, 1>(a, 1, stream) : launch_rows<T, 2>(a, 1, stream);
        if (e) return e;
    }
    const int rg = G == 1 ? 1 : G == 2 || wide == 2 ? 2 : 4;
    const long long ctas = (long long)a.T * a.NKV * ((G + rg - 1) / rg);
    int parts = 1;
    while (few && parts < 8 && ctas * parts < 296) parts *= 2;
    const int alone = few ? 0 : 1;
    if (wide == 2) return rg == 1 ? launch_token<T, 1, 2>(a, parts, alone, stream) : launch_token<T, 2, 2>(a, parts, alone, stream);
    return rg == 1 ? launch_token<T, 1, 1>(a, parts, alone, stream) : rg == 2 ? launch_token<T, 2, 1>(a, parts, alone, stream)
                                                                         : launch_token<T, 4, 1>(a, parts, alone, stream);
}

template <typename T>
static int launch_generic(const void* q, int q_stride, void* out, int out_stride, const void* k_pages,
                          const void* v_pages, const int* positions, const int* seq_of_token, const int* block_table,
                          int bt_stride, const int* bt_rows, int T_tokens, int NH, int NKV, int D, int DV, int page_size, int num_pages,
                          float scale, int window, int keep_first, int v_row, const float* sinks, const float* slopes, const void* gate, int gate_stride,
                          cudaStream_t stream) {
    dim3 grid(T_tokens, (NH + AG_WARPS - 1) / AG_WARPS);
    const size_t smem = (size_t)AG_WARPS * D * sizeof(float);
    const int nr = (DV + 31) / 32;
#define AG_CASE(N)                                                                                                   \
    case N:                                                                                                          \
        attn_generic_kernel<T, N><<<grid, AG_WARPS * 32, smem, stream>>>(                                            \
            (const T*)q, q_stride, (T*)out, out_stride, (const T*)k_pages, (const T*)v_pages, positions,             \
            seq_of_token, block_table, bt_stride, bt_rows, NH, NKV, D, DV, page_size, num_pages, scale, window, keep_first, v_row, sinks, slopes, \
            (const T*)gate, gate_stride);                                                                            \
        break;
    switch (nr) {
        AG_CASE(1) AG_CASE(2) AG_CASE(3) AG_CASE(4) AG_CASE(5) AG_CASE(6) AG_CASE(7) AG_CASE(8)
        AG_CASE(9) AG_CASE(10) AG_CASE(11) AG_CASE(12) AG_CASE(13) AG_CASE(14) AG_CASE(15) AG_CASE(16)
        default: return ACV_ERR_SIZE;
    }
#undef AG_CASE
    return acv_launch_status();
}

ACV_API int acv_attention_generic(const void* q, int q_stride, void* out, int out_stride, const void* k_pages,
                                  const void* v_pages, const int* positions, const int* seq_of_token,
                                  const int* block_table, int bt_stride, const int* bt_rows, int T_tokens, int NH, int NKV, int D,
                                  int page_size, int num_pages, float scale, int window, int dtype,
                                  int value_dim, int keep_first, const float* sinks, const float* slopes, const void* gate,
                                  int gate_stride, cudaStream_t stream) {
    if (T_tokens <= 0) return 0;
    const int DV = value_dim > 0 ? value_dim : D;
    if (D <= 0 || D > 1024 || DV > 512 || NKV <= 0 || NH % NKV) return ACV_ERR_SIZE;
    // values inside the key rows: the same pages, rows of D elements
    const int v_row = v_pages == k_pages ? D : DV;
    if (v_row < DV) return ACV_ERR_SIZE;
    // rows of 4-element pieces at 4-element boundaries: the tiled kernels
    const int piece = dtype == ACV_F32 ? 16 : 8;
    if (D <= 256 && DV <= 256 && (D | DV | q_stride) % 4 == 0 && ((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages) % piece == 0 &&
        (dtype == ACV_F32 || dtype == ACV_BF16)) {
        const AgArgs a = {q, k_pages, v_pages, gate, out, positions, seq_of_token, block_table, bt_rows, sinks, slopes,
                          q_stride, out_stride, gate_stride, bt_stride, T_tokens, NH, NKV, D, DV, page_size, num_pages, window, keep_first, v_row, scale};
        return dtype == ACV_F32 ? launch_tiled<float>(a, stream) : launch_tiled<bf16>(a, stream);
    }
    if (dtype == ACV_F32)
        return launch_generic<float>(q, q_stride, out, out_stride, k_pages, v_pages, positions, seq_of_token,
                                     block_table, bt_stride, bt_rows, T_tokens, NH, NKV, D, DV, page_size, num_pages, scale, window,
                                     keep_first, v_row, sinks, slopes, gate, gate_stride, stream);
    if (dtype == ACV_BF16)
        return launch_generic<bf16>(q, q_stride, out, out_stride, k_pages, v_pages, positions, seq_of_token,
                                    block_table, bt_stride, bt_rows, T_tokens, NH, NKV, D, DV, page_size, num_pages, scale, window,
                                    keep_first, v_row, sinks, slopes, gate, gate_stride, stream);
    return ACV_ERR_DTYPE;
}
