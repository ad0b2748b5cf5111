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
// leaves the other's tokens alone.  Both have one order of sums (below), so a token's result does not depend on the rest of
// the step.  Measured in float32 with 16 heads on 8 kv-heads of 128 (microseconds, one warp per
// (token, head) before -> now): 696 tokens of three portions 831 -> 119, 3 tokens at contexts of 300-500 256 -> 20.
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
// One order of sums.  What a (token, head) comes to depends on its position, its options and its keys alone: not on the
// other tokens of the step, on how a prompt was cut into portions, or on which of the two kernels, how many warps or how many
// CTAs computed it.  The keys lie in tiles of 32 at absolute positions (key % 32 is the lane), of which a token visits
// those with a key that it may see (AgTiles), in ascending order; what it does not see in them weighs 0 and leaves every
// number as it is.  A score is eight chains of multiply-adds (elements whose number / 4 is the same modulo 8, ascending)
// added one by one, ascending.  Up to AgArgs::chunks chunks of consecutive tiles (as even as whole tiles allow, by the number of
// tiles alone) each have a running maximum, a sum per lane and a value sum of their own, ascending over the keys
// (ag_weight), and are added to the total one by one, ascending, rescaled to the larger maximum (ag_fold).  So the rows of
// a portion add a chunk to their totals when it ends, and a token's warps keep theirs until the last is there: 64 chunks
// where two CTAs' worth of them fits an SM beside each other, else 32 (more than one long context's 64 warps could share
// are no use; three tokens at 8000 keys take 140 us with 64, 272 with 32).
#define AG_CHUNKS(rg, vc) ((rg) * (vc) <= 2 ? 64 : 32)

struct AgArgs {
    const void *q, *k_pages, *v_pages, *gate;
    void* out;
    const int *positions, *seq_of_token, *block_table, *bt_rows;
    const float *sinks, *slopes;
    int q_stride, out_stride, gate_stride, bt_stride, T, NH, NKV, D, DV, page_size, num_pages, window, keep_first, v_row, chunks;
    float scale;
};

__device__ __forceinline__ float4 ag_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ag_load4(const bf16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
__device__ __forceinline__ float4 ag_scale4(float4 v, float f) {
    return make_float4(__fmul_rn(v.x, f), __fmul_rn(v.y, f), __fmul_rn(v.z, f), __fmul_rn(v.w, f));
}
__device__ __forceinline__ float ag_dot4(float4 q, float4 k, float s) { return fmaf(q.w, k.w, fmaf(q.z, k.z, fmaf(q.y, k.y, fmaf(q.x, k.x, s)))); }
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
__device__ __forceinline__ float ag_rescale(float from, float to) { return to == -INFINITY ? 1.f : expf(from - to); }
// total + chunk under the factors of their maxima (a factor of 0 must not meet a sum that is no finite number)
__device__ __forceinline__ float ag_fold(float total, float fa, float chunk, float fb) {
    return fmaf(fa == 0.f ? 0.f : total, fa, fb == 0.f ? 0.f : __fmul_rn(chunk, fb));
}
// what the total is multiplied by: a sink is a score without key or value, it takes its share of the weights and adds nothing
__device__ __forceinline__ float ag_inverse(const AgArgs& a, int h, float m, float sum) {
    float f = 1.f;
    if (a.sinks) {
        const float sink = a.sinks[h], m_new = fmaxf(m, sink);
        f = expf(m - m_new);
        sum = fmaf(sum, f, expf(sink - m_new));
    }
    return sum == 0.f ? 0.f : f / sum;
}
// the tiles of a token at position p: [0, kept) for the first keys that stay visible, then [from, last], n in all
struct AgTiles { int kept, from, last, n; };
__device__ __forceinline__ AgTiles ag_tiles(const AgArgs& a, int p) {
    AgTiles t = {0, 0, -1, 0};
    if (p < 0) return t;
    const int lo = a.window > 0 ? max(0, p - a.window + 1) : 0;
    t.kept = a.window > 0 ? (min(max(a.keep_first, 0), lo) + 31) / 32 : 0;
    t.from = max(lo / 32, t.kept);
    t.last = p / 32;
    t.kept = min(t.kept, t.last + 1);
    t.n = t.kept + max(0, t.last - t.from + 1);
    return t;
}
__device__ __forceinline__ float ag_peer(const float* local, int rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_map((uint32_t)__cvta_generic_to_shared(local), rank)) : "memory");
    return v;
}

// ----------------------------------------------------------------------------- rows of a portion
// A stretch: up to 64 / (NH/NKV) tokens of one request, within a block of that many tokens of the flat batch, times the heads of one
// kv-head, eight rows to a warp.  A CTA takes the stretches that begin among its AR_OWN tokens: a portion leaves most
// CTAs without one (they return at once), and a block of two-token portions has work for as many CTAs as it has (33 requests of two tokens
// and 500 keys, 16 heads on 8: one CTA a block 1620 us, looking at 8, 4, 2 tokens 471, 257, 146; prompts of 696 tokens 119 with 8
// and 4, 122 with 2).  Scores: a lane a key, so a 16-byte read of 32 key rows
// moves 512 different bytes and a row's queries are one address; values: a lane four columns.  What belongs to a row (its
// tiles, maximum and total) lies in the lanes 4 i to 4 i + 3 for row i of the warp, so that eight rows' maxima and sums over
// the lanes take nine exchanges instead of forty.  Bound by the chains of
// shared-memory reads (9 to 32 multiply-adds of a warp for the scores), hence eight rows a warp and not fewer: 32 rows and
// four warps to a CTA were slower (156 against 125 us in the form before this one, 696 tokens of three portions), and so was
// bringing the next tile under this one's arithmetic (144 us: its registers are what the reads are hidden with).  The one
// order of sums (eight chains to a score, totals in shared memory, tiles at absolute positions) costs 4 % behind 3000 keys
// (1453 -> 1505 us for 1000 tokens) and one more tile behind a window; shorter prompts are none the worse (130 -> 119).
#define AR_ROWS 64
#define AR_KEYS 32
#define AR_WARP_ROWS 8
#define AR_THREADS 256
#define AR_OWN 4          // tokens among which a CTA looks for stretches to take; under 32

// eight values a lane -> lane l: value l / 4 over all lanes, pairs of lanes 16 apart first, then 8, 4, 2, 1 (warp_sum's order)
template <bool MAX>
__device__ __forceinline__ float ar_over_lanes(const float (&v)[AR_WARP_ROWS], int lane) {
    auto join = [](float x, float y) { return MAX ? fmaxf(x, y) : x + y; };
    float w[4];
    const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = join(h16 ? v[i + 4] : v[i], __shfl_xor_sync(0xffffffffu, h16 ? v[i] : v[i + 4], 16));
#pragma unroll
    for (int i = 0; i < 2; ++i) w[i] = join(h8 ? w[i + 2] : w[i], __shfl_xor_sync(0xffffffffu, h8 ? w[i] : w[i + 2], 8));
    float x = join(h4 ? w[1] : w[0], __shfl_xor_sync(0xffffffffu, h4 ? w[0] : w[1], 4));
    x = join(x, __shfl_xor_sync(0xffffffffu, x, 2));
    return join(x, __shfl_xor_sync(0xffffffffu, x, 1));
}

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
    float* ts = ps + AR_ROWS * AR_KEYS;             // [64][DV]: the rows' totals
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kvh = blockIdx.y, h0 = kvh * G + blockIdx.z * heads, n_heads = min(heads, G - (int)blockIdx.z * heads);
    float* pw = ps + warp * AR_KEYS * AR_WARP_ROWS;

    // the stretches that begin among this CTA's AR_OWN tokens: where a request begins, or a multiple of `tokens`
    const int t_mine = blockIdx.x * AR_OWN;
    uint32_t begins;
    {
        const int t = t_mine + lane, before = t > 0 && t <= a.T ? a.seq_of_token[t - 1] : -1;
        const int own = __shfl_down_sync(0xffffffffu, before, 1);
        begins = __ballot_sync(0xffffffffu, lane < AR_OWN && t < a.T && (t % tokens == 0 || own != before));
    }
    for (; begins; begins &= begins - 1) {
        const int t0 = t_mine + __ffs(begins) - 1, seq = a.seq_of_token[t0];
        int t1 = min(a.T, (t0 / tokens + 1) * tokens);
        for (int t = t0 + 1; t < t1; t += 32) {         // where the request ends, 32 tokens a look
            const uint32_t other = __ballot_sync(0xffffffffu, t + lane < t1 && a.seq_of_token[t + lane] != seq);
            if (other) t1 = t + __ffs(other) - 1;
        }
        if (skip_alone && t1 == t0 + 1 && ag_alone(a.seq_of_token, t0, a.T)) continue;
        const int n = t1 - t0, rows = n * n_heads;      // row r: token t0 + r / n_heads, head h0 + r % n_heads
        const int* bt = a.block_table + (size_t)(a.bt_rows ? a.bt_rows[seq] : seq) * a.bt_stride;
        __syncthreads();
        for (int i = tid; i < AR_ROWS * (D / 4); i += AR_THREADS) {
            const int r = i / (D / 4), c = (i % (D / 4)) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < rows) v = ag_scale4(ag_load4((const T*)a.q + (size_t)(t0 + r / n_heads) * a.q_stride + (size_t)(h0 + r % n_heads) * D + c), a.scale);
            *reinterpret_cast<float4*>(qs + r * ldk + c) = v;
        }
        // the tiles that any row visits
        int kept_tiles = 0, from = 0x7fffffff, last = -1, last_key = -1;
        for (int t = t0 + lane; t < t1; t += 32) {
            const int p = a.positions[t];
            const AgTiles u = ag_tiles(a, p);
            if (u.n == 0) continue;
            kept_tiles = max(kept_tiles, u.kept);
            from = min(from, u.from);
            last = max(last, u.last);
            last_key = max(last_key, p);
        }
        kept_tiles = __reduce_max_sync(0xffffffffu, kept_tiles);
        last = __reduce_max_sync(0xffffffffu, last);
        last_key = __reduce_max_sync(0xffffffffu, last_key);
        from = max(min(__reduce_min_sync(0xffffffffu, from), last + 1), kept_tiles);
        const int r0 = warp * AR_WARP_ROWS;
        int pos[AR_WARP_ROWS];
        float l[AR_WARP_ROWS], acc[AR_WARP_ROWS][4 * VC];
#pragma unroll
        for (int i = 0; i < AR_WARP_ROWS; ++i) {
            pos[i] = r0 + i < rows ? a.positions[t0 + (r0 + i) / n_heads] : -1;
            l[i] = 0.f;
#pragma unroll
            for (int c = 0; c < 4 * VC; ++c) acc[i][c] = 0.f;
#pragma unroll
            for (int c = 0; c < VC; ++c)
                if (c * 128 + lane * 4 < DV) *reinterpret_cast<float4*>(ts + (r0 + i) * DV + c * 128 + lane * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        // this lane's row
        const int my = r0 + lane / 4;
        const AgTiles mt = ag_tiles(a, my < rows ? a.positions[t0 + my / n_heads] : -1);
        float m = -INFINITY, total_m = -INFINITY, total_l = 0.f;
        int filled = 0;             // a.chunks times the tiles of the chunk so far, modulo n

        // a lane looks up one key's row, a tile ahead of its use
        auto look_up = [&](int tile) {
            const int j = tile * AR_KEYS + lane;
            return tile <= last && j <= last_key ? ag_row(a, bt, kvh, j) : -1ll;
        };
        long long next_row = look_up(kept_tiles > 0 ? 0 : from);
        for (int tile = kept_tiles > 0 ? 0 : from; tile <= last; tile = tile + 1 == kept_tiles ? from : tile + 1) {
            const int j0 = tile * AR_KEYS, nk = min(AR_KEYS, last_key + 1 - j0);
            // a warp brings every eighth key, all of its loads on their way together
            const long long my_row = next_row;
            next_row = look_up(tile + 1 == kept_tiles ? from : tile + 1);
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
            if (r0 >= rows) continue;           // (a warp without rows brings its keys and no more)
            float s[AR_WARP_ROWS];
#pragma unroll
            for (int i = 0; i < AR_WARP_ROWS; ++i) s[i] = 0.f;
            auto score = [&](auto pieces) {     // a row's pieces of 32 elements, or 0: as many as there are, the last not whole
#pragma unroll 1
                for (int chain = 0; chain < 32; chain += 4) {
                    float x[AR_WARP_ROWS];
#pragma unroll
                    for (int i = 0; i < AR_WARP_ROWS; ++i) x[i] = 0.f;
                    auto piece = [&](int d) {
                        const float4 k = *reinterpret_cast<const float4*>(ks + lane * ldk + d);
#pragma unroll
                        for (int i = 0; i < AR_WARP_ROWS; ++i) x[i] = ag_dot4(*reinterpret_cast<const float4*>(qs + (r0 + i) * ldk + d), k, x[i]);
                    };
                    if constexpr (decltype(pieces)::value > 0) {
#pragma unroll
                        for (int c = 0; c < decltype(pieces)::value; ++c) piece(chain + c * 32);
                    } else {
                        for (int d = chain; d < D; d += 32) piece(d);
                    }
#pragma unroll
                    for (int i = 0; i < AR_WARP_ROWS; ++i) s[i] += x[i];
                }
            };
            if (D == 128 * VC) score(std::integral_constant<int, 4 * VC>());
            else if (D == 64) score(std::integral_constant<int, 2>());
            else score(std::integral_constant<int, 0>());
            const int j = j0 + lane;
#pragma unroll
            for (int i = 0; i < AR_WARP_ROWS; ++i) {
                if (a.slopes && r0 + i < rows) s[i] = fmaf(-a.slopes[h0 + (r0 + i) % n_heads], (float)(pos[i] - j), s[i]);
                if (my_row < 0 || !ag_sees(a, pos[i], j)) s[i] = -INFINITY;
            }
            const float m_new = fmaxf(m, ar_over_lanes<true>(s, lane)), alpha = ag_rescale(m, m_new);
            if (__any_sync(0xffffffffu, alpha != 1.f && m != -INFINITY)) {     // (a chunk's first tile finds sums of 0)
#pragma unroll
                for (int i = 0; i < AR_WARP_ROWS; ++i) {
                    const float f = __shfl_sync(0xffffffffu, alpha, i * 4);
                    l[i] = __fmul_rn(l[i], f);
#pragma unroll
                    for (int c = 0; c < 4 * VC; ++c) acc[i][c] *= f;
                }
            }
            m = m_new;
#pragma unroll
            for (int i = 0; i < AR_WARP_ROWS; ++i) {
                s[i] = ag_weight(s[i], __shfl_sync(0xffffffffu, m_new, i * 4));
                l[i] = __fadd_rn(l[i], s[i]);             // a lane's share of the sum
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
            // rows whose chunk this tile ends
            bool ends = false;
            if (tile < mt.kept || (tile >= mt.from && tile <= mt.last)) {
                filled += a.chunks;
                ends = filled >= mt.n;
                if (ends) filled -= mt.n;
            }
            const uint32_t ending = __ballot_sync(0xffffffffu, ends);
            if (ending) {
                const float sum = ar_over_lanes<false>(l, lane), both = fmaxf(total_m, m);
                const float fa = ag_rescale(total_m, both), fb = ag_rescale(m, both);
                if (ends) { total_l = fmaf(total_l, fa, __fmul_rn(sum, fb)); total_m = both; m = -INFINITY; }
#pragma unroll
                for (int i = 0; i < AR_WARP_ROWS; ++i) {
                    const float ga = __shfl_sync(0xffffffffu, fa, i * 4), gb = __shfl_sync(0xffffffffu, fb, i * 4);
                    if (!(ending >> (i * 4) & 1)) continue;
                    l[i] = 0.f;
#pragma unroll
                    for (int c = 0; c < VC; ++c) {
                        float4* at = reinterpret_cast<float4*>(ts + (r0 + i) * DV + c * 128 + lane * 4);
                        const bool in = c * 128 + lane * 4 < DV;
                        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (ga != 0.f && in) o = *at;       // (ag_fold's ways, one at a time; the first chunk's ga is 0)
                        if (gb == 0.f) acc[i][c * 4] = acc[i][c * 4 + 1] = acc[i][c * 4 + 2] = acc[i][c * 4 + 3] = 0.f;
                        o.x = fmaf(o.x, ga, __fmul_rn(acc[i][c * 4], gb)); o.y = fmaf(o.y, ga, __fmul_rn(acc[i][c * 4 + 1], gb));
                        o.z = fmaf(o.z, ga, __fmul_rn(acc[i][c * 4 + 2], gb)); o.w = fmaf(o.w, ga, __fmul_rn(acc[i][c * 4 + 3], gb));
                        if (in) *at = o;
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[i][c * 4 + e] = 0.f;
                    }
                }
            }
        }
        const float my_inv = my < rows ? ag_inverse(a, h0 + my % n_heads, total_m, total_l) : 0.f;
#pragma unroll
        for (int i = 0; i < AR_WARP_ROWS; ++i) {
            const float inv = __shfl_sync(0xffffffffu, my_inv, i * 4);
            const int r = r0 + i;
            if (r >= rows) continue;
#pragma unroll
            for (int c = 0; c < VC; ++c) {
                const int e = c * 128 + lane * 4;
                if (e >= DV) continue;
                const float4 o = *reinterpret_cast<const float4*>(ts + r * DV + e);
                const int t = t0 + r / n_heads, h = h0 + r % n_heads;
                ag_put<T>(a, t, h, e, __fmul_rn(o.x, inv)); ag_put<T>(a, t, h, e + 1, __fmul_rn(o.y, inv));
                ag_put<T>(a, t, h, e + 2, __fmul_rn(o.z, inv)); ag_put<T>(a, t, h, e + 3, __fmul_rn(o.w, inv));
            }
        }
    }
    pdl_launch_dependents();
}

// ----------------------------------------------------------------------------- one token
// A cluster of CTAs shares the chunks of one token and kv-head, each of its warps consecutive ones: eight lanes to a key for
// the scores (four keys a load), a lane four columns for the values; RG query heads ride on each key and value
// that is read.  Bound by the pages' stream and its latency.  The chunks' results wait in the CTAs' shared memory; each CTA
// then adds up its share of the columns over all of them.
#define AT1_WARPS 8

template <typename T, int RG, int VC>
__global__ void __launch_bounds__(AT1_WARPS * 32, RG * VC == 1 ? 3 : 2)
attn_token_kernel(const AgArgs a, int parts, int stride) {
    constexpr int CHUNKS = AG_CHUNKS(RG, VC);
    __shared__ float sm_m[CHUNKS][RG], sm_l[CHUNKS][RG];                        // this CTA's chunks
    __shared__ float fac_a[RG][CHUNKS], fac_b[RG][CHUNKS], head_inv[RG];        // all chunks' factors, once all are there
    __shared__ uint32_t chunk_at[CHUNKS];                                       // and where their value sums lie
    __shared__ __align__(16) float sm_w[AT1_WARPS][32][RG], sm_s[AT1_WARPS][RG][32 * 8];
    extern __shared__ __align__(16) float at_o[];      // [CHUNKS / parts][RG][DV]
    pdl_launch_dependents();
    pdl_wait();
    const int D = a.D, DV = a.DV, G = a.NH / a.NKV;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sub = lane & 7, grp = lane >> 3;
    const int part = blockIdx.x % parts;
    const int chunks = (G + RG - 1) / RG, kvh = blockIdx.y / chunks, h0 = kvh * G + (blockIdx.y % chunks) * RG;
    const int n_heads = min(RG, (kvh + 1) * G - h0);
    // one token a cluster; with a stride those of the `stride` tokens x, x + X .. that are alone, X clusters in a row of the grid
    // (bit i: token x + i X; all asked for at once, since a look is a round trip to memory)
    const int x = blockIdx.x / parts, X = gridDim.x / parts;
    uint32_t mine = 1;
    if (stride) {
        const int cand = x + lane * X;
        mine = __ballot_sync(0xffffffffu, lane < stride && cand < a.T && ag_alone(a.seq_of_token, cand, a.T));
    }
    for (; mine; mine &= mine - 1) {
        const int t = x + (__ffs(mine) - 1) * X;
        if (stride) __syncthreads();        // the token before is done with the shared memory
        const int p = a.positions[t], seq = a.seq_of_token[t];
        const int* bt = a.block_table + (size_t)(a.bt_rows ? a.bt_rows[seq] : seq) * a.bt_stride;
        const AgTiles mt = ag_tiles(a, p);
        // chunk c: the tiles whose number among the visited ones lies in [c n / n_chunks, (c + 1) n / n_chunks)
        const int n_chunks = min(mt.n, CHUNKS);
        const int gw = part * AT1_WARPS + warp, GW = parts * AT1_WARPS;
        const int c_begin = gw * n_chunks / GW, c_end = (gw + 1) * n_chunks / GW, c_base = part * n_chunks / parts;

        // queries: lane `sub` of a key's eight holds elements sub*4 + 32 c
        constexpr int QC = VC * 4;
        float4 q[RG][QC];
#pragma unroll
        for (int r = 0; r < RG; ++r)
#pragma unroll
            for (int c = 0; c < QC; ++c) {
                const int e = sub * 4 + 32 * c;
                q[r][c] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < n_heads && e < D) q[r][c] = ag_scale4(ag_load4((const T*)a.q + (size_t)t * a.q_stride + (size_t)(h0 + r) * D + e), a.scale);
            }
        float m[RG], l[RG], acc[RG][4 * VC];
        auto tile_begin = [&](int o) { return (o < mt.kept ? o : mt.from + o - mt.kept) * 32; };
        for (int chunk = c_begin; chunk < c_end; ++chunk) {
#pragma unroll
            for (int r = 0; r < RG; ++r) {
                m[r] = -INFINITY; l[r] = 0.f;
#pragma unroll
                for (int c = 0; c < 4 * VC; ++c) acc[r][c] = 0.f;
            }
            const int o_end = ((chunk + 1) * mt.n + n_chunks - 1) / n_chunks;
            for (int o = (chunk * mt.n + n_chunks - 1) / n_chunks; o < o_end; ++o) {
                const int j0 = tile_begin(o), j = j0 + lane;
                const long long row = ag_sees(a, p, j) ? ag_row(a, bt, kvh, j) : -1;
#pragma unroll
                for (int g = 0; g < 8; ++g) {           // keys g*4 .. g*4 + 3 of the tile, eight lanes each
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
                        for (int r = 0; r < RG; ++r) s[r] = ag_dot4(q[r][c], k, s[r]);
                    }
#pragma unroll
                    for (int r = 0; r < RG; ++r) sm_s[warp][r][(g * 4 + grp) * 8 + (sub ^ (g & 1) * 4)] = s[r];     // (halves swapped: no bank met twice)
                }
                __syncwarp();
#pragma unroll
                for (int r = 0; r < RG; ++r) {
                    const float slope = a.slopes && r < n_heads ? a.slopes[h0 + r] : 0.f;
                    const float4* mine = reinterpret_cast<const float4*>(sm_s[warp][r] + lane * 8);
                    const float4 x0 = mine[lane >> 2 & 1], x1 = mine[(lane >> 2 & 1) ^ 1];
                    const float dot = ((((((x0.x + x0.y) + x0.z) + x0.w) + x1.x) + x1.y) + x1.z) + x1.w;
                    const float score = row >= 0 ? fmaf(-slope, (float)(p - j), dot) : -INFINITY;
                    const float m_new = fmaxf(m[r], warp_max(score)), alpha = ag_rescale(m[r], m_new);
                    const float w = ag_weight(score, m_new);
                    l[r] = __fadd_rn(__fmul_rn(l[r], alpha), w);
                    m[r] = m_new;
#pragma unroll
                    for (int c = 0; c < 4 * VC; ++c) acc[r][c] *= alpha;
                    sm_w[warp][lane][r] = w;
                }
                __syncwarp();
                const int nk = min(32, p + 1 - j0);
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
            const int slot = chunk - c_base;
#pragma unroll
            for (int r = 0; r < RG; ++r) {
                const float sum = warp_sum(l[r]);
                if (lane == 0) { sm_m[slot][r] = m[r]; sm_l[slot][r] = sum; }
#pragma unroll
                for (int c = 0; c < VC; ++c)
                    if (c * 128 + lane * 4 < DV)
                        *reinterpret_cast<float4*>(at_o + (slot * RG + r) * DV + c * 128 + lane * 4) =
                            make_float4(acc[r][c * 4], acc[r][c * 4 + 1], acc[r][c * 4 + 2], acc[r][c * 4 + 3]);
            }
        }
        if (parts > 1) cluster_sync_all(); else __syncthreads();
        // chunk c lies with the CTA whose range of them, [b n_chunks / parts, (b + 1) n_chunks / parts), holds it
        auto owner = [&](int c) { return ((c + 1) * parts - 1) / n_chunks; };
        if (warp < RG) {            // a warp a head, a lane a chunk: the total's maximum in front of it and with it
            float front_all = -INFINITY, sum = 0.f;
#pragma unroll
            for (int c0 = 0; c0 < CHUNKS; c0 += 32) {
                if (c0 >= n_chunks) break;
                const int c = c0 + lane;
                float cm = -INFINITY, cl = 0.f;
                if (c < n_chunks) {
                    const int b = owner(c), slot = c - b * n_chunks / parts;
                    cm = ag_peer(&sm_m[slot][warp], b);
                    cl = ag_peer(&sm_l[slot][warp], b);
                }
                float with = cm;
#pragma unroll
                for (int h = 1; h < 32; h <<= 1) {
                    const float up = __shfl_up_sync(0xffffffffu, with, h);
                    if (lane >= h) with = fmaxf(with, up);
                }
                with = fmaxf(with, front_all);
                const float front = __shfl_up_sync(0xffffffffu, with, 1);
                const float fa = ag_rescale(lane ? front : front_all, with), fb = ag_rescale(cm, with), add = __fmul_rn(cl, fb);
                fac_a[warp][c] = fa;
                fac_b[warp][c] = fb;
#pragma unroll
                for (int i = 0; i < 32; ++i)        // (behind the last chunk: times 1, plus 0)
                    sum = fmaf(sum, __shfl_sync(0xffffffffu, fa, i), __shfl_sync(0xffffffffu, add, i));
                front_all = __shfl_sync(0xffffffffu, with, 31);
            }
            if (lane == 0) head_inv[warp] = warp < n_heads ? ag_inverse(a, h0 + warp, front_all, sum) : 0.f;
        } else if (warp == RG) {
            for (int c = lane; c < n_chunks; c += 32) {
                const int b = owner(c);
                chunk_at[c] = cluster_map((uint32_t)__cvta_generic_to_shared(at_o + (c - b * n_chunks / parts) * RG * DV), b);
            }
        }
        __syncthreads();
        const int share = (RG * DV + parts - 1) / parts;
        for (int e = part * share + tid; e < min(RG * DV, (part + 1) * share); e += AT1_WARPS * 32) {
            const int r = e / DV;
            if (r >= n_heads) continue;
            float o = 0.f;
            for (int c0 = 0; c0 < n_chunks; c0 += 16) {         // sixteen on their way together
                float v[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    v[i] = 0.f;
                    if (c0 + i < n_chunks) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[i]) : "r"(chunk_at[c0 + i] + e * 4) : "memory");
                }
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (c0 + i < n_chunks) o = ag_fold(o, fac_a[r][c0 + i], v[i], fac_b[r][c0 + i]);
            }
            ag_put<T>(a, t, h0 + r, e % DV, __fmul_rn(o, head_inv[r]));
        }
        if (parts > 1) cluster_sync_all();      // nobody leaves while its results are read
    }
}

template <typename T, int RG, int VC>
static int launch_token(const AgArgs& a, int parts, int stride, cudaStream_t stream) {
    auto kernel = attn_token_kernel<T, RG, VC>;
    const int smem = AG_CHUNKS(RG, VC) / parts * RG * a.DV * 4;
    static AcvSmemConfig cfg;
    if (const int e = acv_ensure_smem(cfg, kernel, smem)) return e;
    const int G = a.NH / a.NKV, x = (stride ? (a.T + stride - 1) / stride : a.T) * parts;
    acv_launch_cluster(PDL_ATTN, dim3(parts, 1, 1), kernel, dim3(x, a.NKV * ((G + RG - 1) / RG)), dim3(AT1_WARPS * 32), smem, stream, a, parts, stride);
    return acv_launch_status();
}

template <typename T, int VC>
static int launch_rows(const AgArgs& a, int skip_alone, cudaStream_t stream) {
    auto kernel = attn_rows_kernel<T, VC>;
    const int smem = ((AR_ROWS + AR_KEYS) * (a.D + 4) + (AR_KEYS + AR_ROWS) * a.DV + AR_ROWS * AR_KEYS) * 4;
    static AcvSmemConfig cfg;
    if (const int e = acv_ensure_smem(cfg, kernel, smem)) return e;
    const int G = a.NH / a.NKV, heads = G < AR_ROWS ? G : AR_ROWS;
    acv_launch(PDL_ATTN, kernel, dim3((a.T + AR_OWN - 1) / AR_OWN, a.NKV, (G + heads - 1) / heads), dim3(AR_THREADS), smem, stream, a, skip_alone);
    return acv_launch_status();
}

// Steps of requests that bring one token each (the caller says so; the results are the same whether it does), and of up to
// AG_FEW tokens and AG_FEW_ROWS (token, head) rows: every token by itself.  Others: rows of portions, then the tokens that are
// alone (a portion's 64 rows read each key once for all of them, one token's warps once for its own heads).  Below the line
// lie tokens that fill half a wave (bfloat16, portions of 20, 17 and 9 tokens, every token by itself against both kernels: 8 heads on 8 of 64 11.4
// and 15.2 us, 14 on 2 15.7 and 25.8, 5 on 1 of 256 24.4 and 41.7), above it those that take several (32 on 8 of 128 27.9 and
// 18.7, 40 on 8 39.9 and 29.9; one portion of 64 tokens: 16 on 8 36.6 and 29.6, 40 on 8 77.2 and 31.5).  As many CTAs to a
// token and kv-head as come in one wave (two to
// an SM; 16 requests of 1500 keys, 16 heads on 8, with 1, 2, 4, 8: 206, 110, 150, 165 us).  A CTA looks at as
// many tokens as leave eight CTAs to an SM, at most AG_STRIDE: all of them may be alone, and one behind the other took 65
// requests of 500 keys 532 us where 64 take 144 (150 with a CTA each); of a portion's thousands none are.
#define AG_FEW 64
#define AG_FEW_ROWS 700
#define AG_STRIDE 8
template <typename T>
static int launch_tiled(AgArgs& a, bool singles, cudaStream_t stream) {
    int device = 0, sms = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (err != cudaSuccess) return (int)err;
    const int G = a.NH / a.NKV, wide = (a.D > 128 || a.DV > 128) ? 2 : 1;
    const int rg = G == 1 ? 1 : G == 2 || wide == 2 ? 2 : 4;
    a.chunks = AG_CHUNKS(rg, wide);
    const bool each = singles || (a.T <= AG_FEW && a.T * a.NH <= AG_FEW_ROWS);
    if (!each) {
        const int e = wide == 1 ? launch_rows<T, 1>(a, 1, stream) : launch_rows<T, 2>(a, 1, stream);
        if (e) return e;
    }
    const long long ctas = (long long)a.T * a.NKV * ((G + rg - 1) / rg);
    int parts = 1;
    while (parts < 8 && ctas * parts <= sms) parts *= 2;
    const int stride = each ? 0 : parts > 1 ? 1 : (int)max(1ll, min((long long)AG_STRIDE, ctas / (8 * sms)));
    if (wide == 2) return rg == 1 ? launch_token<T, 1, 2>(a, parts, stride, stream) : launch_token<T, 2, 2>(a, parts, stride, stream);
    return rg == 1 ? launch_token<T, 1, 1>(a, parts, stride, stream) : rg == 2 ? launch_token<T, 2, 1>(a, parts, stride, stream)
                                                                          : launch_token<T, 4, 1>(a, parts, stride, stream);
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

// singles: no request brings more than one token (a hint for the choice of kernels).
ACV_API int acv_attention_generic(const void* q, int q_stride, void* out, int out_stride, const void* k_pages,
                                  const void* v_pages, const int* positions, const int* seq_of_token,
                                  const int* block_table, int bt_stride, const int* bt_rows, int T_tokens, int NH, int NKV, int D,
                                  int page_size, int num_pages, float scale, int window, int dtype,
                                  int value_dim, int keep_first, const float* sinks, const float* slopes, const void* gate,
                                  int gate_stride, int singles, cudaStream_t stream) {
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
        AgArgs a = {q, k_pages, v_pages, gate, out, positions, seq_of_token, block_table, bt_rows, sinks, slopes,
                          q_stride, out_stride, gate_stride, bt_stride, T_tokens, NH, NKV, D, DV, page_size, num_pages, window, keep_first, v_row, 0, scale};
        return dtype == ACV_F32 ? launch_tiled<float>(a, singles != 0, stream) : launch_tiled<bf16>(a, singles != 0, stream);
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
