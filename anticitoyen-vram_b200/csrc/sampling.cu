// On-device sampling over float32 logits [rows, V]: penalties, greedy argmax,
// temperature, top-k, min-p, top-p and the draw, one block per row.
//
// Order and meaning follow the reference (acvram/engine/sampler.py:195-256):
// penalties on the raw logits; scaled = logit / max(T, 1e-5); top-k keeps the
// values >= the k-th largest; min-p drops p < min_p * p_max; top-p drops a token
// when the mass of the tokens before it in descending order exceeds top_p (the
// token that crosses stays, so the set is never empty); the draw is from the
// softmax of what is left.  A row with temperature <= 0 takes the argmax.
//
// Nothing is sorted: the k-th value and the top-p cut are found by bisection on
// an order-preserving 32-bit key of the float, 32 counting passes each over the
// row (which stays in L2; a wide row's cluster finds them four bits a pass).  The reference draws with torch.multinomial from a
// global generator; here each row has a counter-based generator, Philox-4x32-10
// keyed by the request's seed with the request's step as counter, so a draw does
// not depend on what else is in the batch.  The draw is the inverse CDF over the
// kept tokens in index order.
#include "common.cuh"

#define SMP_THREADS 1024

__device__ __forceinline__ uint32_t order_key(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float philox_uniform(uint64_t seed, uint64_t counter) {
    const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
    uint32_t c0 = (uint32_t)counter, c1 = (uint32_t)(counter >> 32), c2 = 0, c3 = 0;
    uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t hi0 = __umulhi(M0, c0), lo0 = M0 * c0;
        const uint32_t hi1 = __umulhi(M1, c2), lo1 = M1 * c2;
        const uint32_t n0 = hi1 ^ c1 ^ k0, n1 = lo1, n2 = hi0 ^ c3 ^ k1, n3 = lo0;
        c0 = n0; c1 = n1; c2 = n2; c3 = n3;
        k0 += W0; k1 += W1;
    }
    return ((float)c0 + 0.5f) * (1.0f / 4294967296.0f);
}

// block-wide reductions over SMP_THREADS threads; all threads get the result
__device__ __forceinline__ float block_reduce_sum(float v, float* red) { return block_sum(v, red); }

__device__ __forceinline__ float block_reduce_max(float v, float* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float t = lane < nwarp ? red[lane] : -INFINITY;
    return warp_max(t);
}

__device__ __forceinline__ int block_reduce_sum_int(int v, int* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    int t = lane < nwarp ? red[lane] : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

// argmax with the lowest index among equal values (torch.argmax's answer)
__device__ __forceinline__ int block_argmax(const float* row, int V, float inv_temp, float* redf, int* redi) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
        const float v = row[i] * inv_temp;
        if (v > best || (v == best && i < bi)) { best = v; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) { redf[warp] = best; redi[warp] = bi; }
    __syncthreads();
    best = lane < nwarp ? redf[lane] : -INFINITY;
    bi = lane < nwarp ? redi[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    return bi;
}

__global__ void __launch_bounds__(SMP_THREADS)
argmax_kernel(const float* __restrict__ logits, int ld, int V, int* __restrict__ out) {
    __shared__ float redf[32];
    __shared__ int redi[32];
    const int bi = block_argmax(logits + (size_t)blockIdx.x * ld, V, 1.f, redf, redi);
    if (threadIdx.x == 0) out[blockIdx.x] = bi == 0x7fffffff ? 0 : bi;     // a row without a value above -inf (all NaN): token 0
}

// Wide rows: each row is cut into ARG_PARTS slices, one block per slice leaves (value, index) in
// scratch, and the block that arrives last at a row picks among the slices in slice order (lowest
// index among equal values, as above).  No block waits for another.
#define ARG_PARTS 16
#define ARG_MAX_ROWS 4096
static __device__ float arg_part_val[ARG_MAX_ROWS * ARG_PARTS];
static __device__ int arg_part_idx[ARG_MAX_ROWS * ARG_PARTS];
static __device__ int arg_counter[ARG_MAX_ROWS];

__global__ void __launch_bounds__(256)
argmax_split_kernel(const float* __restrict__ logits, int ld, int V, int* __restrict__ out) {
    __shared__ float redf[32];
    __shared__ int redi[32];
    __shared__ int last_s;
    ACV_TL(TL_ARGMAX, 0);
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.x, part = blockIdx.y;
    const int span = ((V + ARG_PARTS - 1) / ARG_PARTS + 3) & ~3;
    const int lo = part * span, hi = min(V, lo + span);
    const float* r = logits + (size_t)row * ld;
    float best = -INFINITY;
    int bi = 0x7fffffff;
    if ((((uintptr_t)r) & 15) == 0 && (lo & 3) == 0) {
        // 16-byte loads, four in flight per thread before the first comparison (the slice is short: what
        // counts is that its loads are all on their way at once)
        const int n4 = (hi - lo) >> 2;
        const float4* r4 = reinterpret_cast<const float4*>(r + lo);
        for (int c0 = threadIdx.x; c0 < n4; c0 += 4 * blockDim.x) {
            float4 v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int c = c0 + k * blockDim.x;
                v[k] = c < n4 ? r4[c] : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = lo + 4 * (c0 + k * blockDim.x);
                if (v[k].x > best) { best = v[k].x; bi = i; }
                if (v[k].y > best) { best = v[k].y; bi = i + 1; }
                if (v[k].z > best) { best = v[k].z; bi = i + 2; }
                if (v[k].w > best) { best = v[k].w; bi = i + 3; }
            }
        }
        for (int i = lo + (n4 << 2) + threadIdx.x; i < hi; i += blockDim.x) {
            const float v = r[i];
            if (v > best) { best = v; bi = i; }
        }
    } else {
        for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
            const float v = r[i];
            if (v > best || (v == best && i < bi)) { best = v; bi = i; }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    if (lane == 0) { redf[warp] = best; redi[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        best = lane < nwarp ? redf[lane] : -INFINITY;
        bi = lane < nwarp ? redi[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if (lane == 0) {
            arg_part_val[row * ARG_PARTS + part] = best;
            arg_part_idx[row * ARG_PARTS + part] = bi;
            __threadfence();
            last_s = atomicAdd(&arg_counter[row], 1) == ARG_PARTS - 1;
        }
    }
    __syncthreads();
    if (last_s && threadIdx.x == 0) {
        __threadfence();
        float b = -INFINITY;
        int idx = 0x7fffffff;
        for (int q = 0; q < ARG_PARTS; ++q) {
            const float v = __ldcg(&arg_part_val[row * ARG_PARTS + q]);
            const int i = __ldcg(&arg_part_idx[row * ARG_PARTS + q]);
            if (v > b || (v == b && i < idx)) { b = v; idx = i; }
        }
        out[row] = idx == 0x7fffffff ? 0 : idx;
        arg_counter[row] = 0;
    }
}

ACV_API int acv_argmax(const float* logits, int ld, int rows, int V, int* out, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (V <= 0) return ACV_ERR_SIZE;
    if (V >= 16384 && rows <= ARG_MAX_ROWS) {
        acv_launch(PDL_MISC, argmax_split_kernel, dim3(rows, ARG_PARTS), 256, 0, stream, logits, ld, V, out);
        return acv_launch_status();
    }
    argmax_kernel<<<rows, SMP_THREADS, 0, stream>>>(logits, ld, V, out);
    return acv_launch_status();
}

// ----------------------------------------------------------------------------- penalties
// One thread per (row, distinct token already seen, its count).
__global__ void penalties_kernel(float* __restrict__ logits, int ld, int V, const int* __restrict__ pen_row,
                                 const int* __restrict__ pen_token, const int* __restrict__ pen_count, int n,
                                 const float* __restrict__ repetition, const float* __restrict__ presence,
                                 const float* __restrict__ frequency) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int r = pen_row[i], tok = pen_token[i];
    if (tok < 0 || tok >= V) return;
    float v = logits[(size_t)r * ld + tok];
    const float rep = repetition[r];
    if (rep != 1.f) v = v > 0.f ? v / rep : v * rep;
    v -= presence[r];
    v -= frequency[r] * (float)pen_count[i];
    logits[(size_t)r * ld + tok] = v;
}

ACV_API int acv_apply_penalties(float* logits, int ld, int V, const int* pen_row, const int* pen_token,
                                const int* pen_count, int n, const float* repetition, const float* presence,
                                const float* frequency, cudaStream_t stream) {
    if (n <= 0) return 0;
    penalties_kernel<<<(n + 255) / 256, 256, 0, stream>>>(logits, ld, V, pen_row, pen_token, pen_count, n, repetition,
                                                          presence, frequency);
    return acv_launch_status();
}

// ----------------------------------------------------------------------------- sample
__global__ void __launch_bounds__(SMP_THREADS)
sample_kernel(const float* __restrict__ logits, int ld, int V, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p, const float* __restrict__ min_p,
              const unsigned long long* __restrict__ seed, const unsigned long long* __restrict__ counter,
              int* __restrict__ out_token, float* __restrict__ out_logprob) {
    __shared__ float redf[32];
    __shared__ int redi[32];
    __shared__ float scan[SMP_THREADS];
    const int r = blockIdx.x;
    const float* row = logits + (size_t)r * ld;
    const float temp = temperature[r];

    if (temp <= 0.f) {  // greedy row
        int bi = block_argmax(row, V, 1.f, redf, redi);
        if (bi == 0x7fffffff) bi = 0;           // a row without a value above -inf (all NaN): token 0, as argmax_split_kernel
        float z = 0.f;
        if (out_logprob) {
            const float mx = row[bi];
            for (int i = threadIdx.x; i < V; i += blockDim.x) z += expf(row[i] - mx);
            z = block_reduce_sum(z, redf);
        }
        if (threadIdx.x == 0) {
            out_token[r] = bi;
            if (out_logprob) out_logprob[r] = -logf(z);
        }
        return;
    }

    const float inv_t = 1.f / fmaxf(temp, 1e-5f);
    float mx = -INFINITY;
    for (int i = threadIdx.x; i < V; i += blockDim.x) mx = fmaxf(mx, row[i] * inv_t);
    mx = block_reduce_max(mx, redf);

    uint32_t cut = 0;  // keys >= cut are kept
    const int k = top_k[r];
    if (k > 0 && k < V) {
        uint32_t prefix = 0;
        for (int b = 31; b >= 0; --b) {
            const uint32_t cand = prefix | (1u << b);
            int cnt = 0;
            for (int i = threadIdx.x; i < V; i += blockDim.x) cnt += order_key(row[i] * inv_t) >= cand;
            cnt = block_reduce_sum_int(cnt, redi);
            if (cnt >= k) prefix = cand;
        }
        cut = prefix;
    }
    const float mp = min_p[r];
    const bool use_minp = mp > 0.f;
    // kept(i): key >= cut and (no min-p or exp(s - max) >= min_p)
    const float tp = top_p[r];
    if (tp > 0.f && tp < 1.f) {
        float z = 0.f;
        for (int i = threadIdx.x; i < V; i += blockDim.x) {
            const float s = row[i] * inv_t;
            const float e = expf(s - mx);
            if (order_key(s) >= cut && !(use_minp && e < mp)) z += e;
        }
        z = block_reduce_sum(z, redf);
        const float limit = tp * z;
        uint32_t prefix = 0;  // the largest key value t with mass(key > t) > limit
        for (int b = 31; b >= 0; --b) {
            const uint32_t cand = prefix | (1u << b);
            float mass = 0.f;
            for (int i = threadIdx.x; i < V; i += blockDim.x) {
                const float s = row[i] * inv_t;
                const uint32_t key = order_key(s);
                const float e = expf(s - mx);
                if (key > cand && key >= cut && !(use_minp && e < mp)) mass += e;
            }
            mass = block_reduce_sum(mass, redf);
            if (mass > limit) prefix = cand;
        }
        const uint32_t cut_p = prefix + 1u;
        cut = cut_p > cut ? cut_p : cut;
    }

    // inverse CDF in index order: each thread owns a contiguous range of indices
    const int chunk = (V + blockDim.x - 1) / blockDim.x;
    const int lo = threadIdx.x * chunk, hi = min(V, lo + chunk);
    float local = 0.f;
    for (int i = lo; i < hi; ++i) {
        const float s = row[i] * inv_t;
        const float e = expf(s - mx);
        if (order_key(s) >= cut && !(use_minp && e < mp)) local += e;
    }
    scan[threadIdx.x] = local;
    __syncthreads();
    __shared__ float total_s;
    __shared__ int owner_s;
    __shared__ float before_s;
    if (threadIdx.x == 0) {
        float run = 0.f;
        for (int t = 0; t < (int)blockDim.x; ++t) run += scan[t];
        const float u = philox_uniform(seed[r], counter[r]);
        const float target = u * run;
        float acc = 0.f;
        int owner = -1;
        int last_nonempty = 0;
        for (int t = 0; t < (int)blockDim.x; ++t) {
            if (scan[t] > 0.f) last_nonempty = t;
            if (owner < 0 && scan[t] > 0.f && acc + scan[t] >= target) { owner = t; before_s = acc; }
            if (owner < 0) acc += scan[t];
        }
        if (owner < 0) { owner = last_nonempty; before_s = acc - scan[last_nonempty]; }
        owner_s = owner;
        total_s = run;
        redf[0] = target;
    }
    __syncthreads();
    if ((int)threadIdx.x == owner_s) {
        const float target = redf[0];
        float acc = before_s;
        int pick = -1, last_kept = -1;
        for (int i = lo; i < hi; ++i) {
            const float s = row[i] * inv_t;
            const float e = expf(s - mx);
            if (order_key(s) >= cut && !(use_minp && e < mp)) {
                last_kept = i;
                acc += e;
                if (acc >= target) { pick = i; break; }
            }
        }
        if (pick < 0) pick = last_kept;
        out_token[r] = pick;
        if (out_logprob) out_logprob[r] = (row[pick] * inv_t - mx) - logf(total_s);
    }
}

// ----------------------------------------------------------------------------- sample, a cluster to a row
// A wide row (a vocabulary of 150 thousand) read 70 times by one block is bound by the latency of its loads: a
// second per thousand steps of eight rows.  Here the CTAs of one thread-block cluster share a row: each keeps its
// slice of the scaled logits in shared memory, so the row is read from memory once and the bisections' passes run
// on shared memory; what a pass counts is added up over the cluster through the CTAs' shared memory (every CTA
// writes its part into every CTA's table, one cluster barrier, every CTA adds the parts in rank order, so all take
// the same decision).  The arithmetic is sample_kernel's; sums are formed slice by slice.
#define SMPC_CTAS 8
#define SMPC_THREADS 1024

struct ClusterSum {
    float* parts;          // [2][SMPC_CTAS] in this CTA's shared memory
    float* warps;          // [32]
    float* table;          // [32][17]
    int turn;
    uint32_t rank;
};

// every thread gets the sum over the cluster of `v` (a float; counts up to 2^24 are exact)
__device__ __forceinline__ float cluster_all_sum(ClusterSum& c, float v) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_sum(v);
    if (lane == 0) c.warps[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float t = lane < (int)(blockDim.x >> 5) ? c.warps[lane] : 0.f;
        t = warp_sum(t);
        if (lane < SMPC_CTAS)
            cluster_store_f32(cluster_map((uint32_t)__cvta_generic_to_shared(c.parts + c.turn * SMPC_CTAS + c.rank), lane), t);
    }
    cluster_sync_all();
    float total = 0.f;
#pragma unroll
    for (int r = 0; r < SMPC_CTAS; ++r) total += c.parts[c.turn * SMPC_CTAS + r];
    c.turn ^= 1;
    return total;
}
// the maximum over the cluster of `v`, and the mean over its threads of those `v` that are finite (0 where there are none)
__device__ __forceinline__ float cluster_max_and_mean(ClusterSum& c, float* sums, float v, float& mean) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool finite = fabsf(v) <= 3.402823466e38f;
    const float top = warp_max(v), sum = warp_sum(finite ? v : 0.f), count = (float)__popc(__ballot_sync(0xffffffffu, finite));
    if (lane == 0) { c.table[warp] = top; c.table[32 + warp] = sum; c.table[64 + warp] = count; }
    __syncthreads();
    if (warp < 3) {
        float t = c.table[warp * 32 + lane];
        t = warp == 0 ? warp_max(t) : warp_sum(t);
        float* to = warp == 0 ? c.parts + c.turn * SMPC_CTAS : sums + (warp - 1) * SMPC_CTAS;
        if (lane < SMPC_CTAS) cluster_store_f32(cluster_map((uint32_t)__cvta_generic_to_shared(to + c.rank), lane), t);
    }
    cluster_sync_all();
    float total = -INFINITY, all = 0.f, n = 0.f;
#pragma unroll
    for (int r = 0; r < SMPC_CTAS; ++r) {
        total = fmaxf(total, c.parts[c.turn * SMPC_CTAS + r]);
        all += sums[r];
        n += sums[SMPC_CTAS + r];
    }
    c.turn ^= 1;
    mean = n > 0.f ? all / n : 0.f;
    return total;
}
__device__ __forceinline__ float cluster_all_max(ClusterSum& c, float v) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_max(v);
    if (lane == 0) c.warps[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float t = lane < (int)(blockDim.x >> 5) ? c.warps[lane] : -INFINITY;
        t = warp_max(t);
        if (lane < SMPC_CTAS)
            cluster_store_f32(cluster_map((uint32_t)__cvta_generic_to_shared(c.parts + c.turn * SMPC_CTAS + c.rank), lane), t);
    }
    cluster_sync_all();
    float total = -INFINITY;
#pragma unroll
    for (int r = 0; r < SMPC_CTAS; ++r) total = fmaxf(total, c.parts[c.turn * SMPC_CTAS + r]);
    c.turn ^= 1;
    return total;
}

// What a pass of sixteen bins finds: v[d] is this thread's sum over its elements of digit d, `seen` how many of its elements took
// part.  The bins are added up over warp, CTA and cluster (in an order that the launch shape fixes), and the sums from the top
// down say which bin the wanted key lies in: the largest d for which over + (bins d and above) reaches `limit` (above: exceeds
// it), 0 if none does (found: whether one did).  `over` takes the bins above d.  Returns d; seen: the cluster's count.
// share > 0: the limit is that share of the sum of all bins.
__device__ __forceinline__ uint32_t cluster_bins(ClusterSum& c, float* bins, float (&v)[16], float& seen, float& limit, bool above,
                                                 float& over, bool& found, float share = 0.f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // over the warp: a lane gives away half of what it carries at each exchange and ends with bin `lane % 16`
#pragma unroll
    for (int h = 8; h > 0; h >>= 1) {
        const bool high = lane & h;
#pragma unroll
        for (int d = 0; d < 8; ++d)
            if (d < h) {
                const float give = high ? v[d] : v[d + h], keep = high ? v[d + h] : v[d];
                v[d] = keep + __shfl_xor_sync(0xffffffffu, give, h);
            }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);
    seen = warp_sum(seen);
    if (lane < 16) c.table[warp * 17 + lane] = v[0];
    if (lane == 16) c.table[warp * 17 + 16] = seen;
    __syncthreads();
    if (warp < 17) {        // warp d adds up bin d over the warps and tells every CTA
        const float t = warp_sum(c.table[lane * 17 + warp]);
        if (lane < SMPC_CTAS)
            cluster_store_f32(cluster_map((uint32_t)__cvta_generic_to_shared(bins + (c.turn * SMPC_CTAS + c.rank) * 17 + warp), lane), t);
    }
    cluster_sync_all();
    float s = 0.f;          // lane d: bin d, then the sum of the bins d and above
    seen = 0.f;
#pragma unroll
    for (int r = 0; r < SMPC_CTAS; ++r) {
        s += bins[(c.turn * SMPC_CTAS + r) * 17 + (lane & 15)];
        seen += bins[(c.turn * SMPC_CTAS + r) * 17 + 16];
    }
    c.turn ^= 1;
#pragma unroll
    for (int h = 1; h < 16; h <<= 1) {
        const float up = __shfl_down_sync(0xffffffffu, s, h, 16);
        if ((lane & 15) + h < 16) s += up;
    }
    if (share > 0.f) limit = share * __shfl_sync(0xffffffffu, s, 0, 16);
    const float at = over + s;
    const uint32_t good = __ballot_sync(0xffffffffu, above ? at > limit : at >= limit) & 0xffffu;
    const int d = good ? 31 - __clz(good) : 0;
    const float beyond = __shfl_sync(0xffffffffu, s, (d + 1) & 15, 16);
    if (d < 15) over += beyond;
    found = good != 0;
    return (uint32_t)d;
}

// The largest c for which the sum of w over the elements with key >= c reaches `limit` (above: exceeds it), 0 if none
// does.  Four bits a pass, from the top: the elements that share the bits found so far fall into 16 bins by their next
// four, a thread's in registers.  A pass costs its meeting of the cluster, 2 us, so eight
// passes of sixteen candidates replace 32 of one
// (8 rows of 151 936, microseconds: top-p 141 -> 64, top-k 120 -> 49, both 199 -> 91).
template <typename Element>
__device__ __forceinline__ uint32_t cluster_descend(ClusterSum& c, float* bins, int n, float limit, bool above, Element element) {
    uint32_t prefix = 0;
    float over = 0.f;           // the sum over the elements whose bits so far are larger than c's
    for (int shift = 28; shift >= 0; shift -= 4) {
        float v[16], seen = 0.f;
#pragma unroll
        for (int d = 0; d < 16; ++d) v[d] = 0.f;
        for (int i = threadIdx.x; i < n; i += SMPC_THREADS) {
            uint32_t key;
            float w;
            element(i, key, w);
            if (shift < 28 && (key ^ prefix) >> (shift + 4)) continue;
            const uint32_t digit = key >> shift & 15u;
#pragma unroll
            for (uint32_t d = 0; d < 16; ++d) v[d] += digit == d ? w : 0.f;
        }
        bool found;
        prefix |= cluster_bins(c, bins, v, seen, limit, above, over, found) << shift;
    }
    return prefix;
}

// The same answer in fewer passes where the row's values are spread as a vocabulary's logits are.  The first passes sort by the
// distance from the maximum in units of 1/scale, then 16ths and 256ths of them (a step function of the logit, so its bins
// follow the keys' order; what lies 16 units and further shares the lowest bin).  The unit is a sixth of what lies between the
// maximum and the mean of the threads' own maxima: two fifths of a standard deviation or so, whatever the temperature, and few
// entries at the lowest value of the type do not move it.  As soon as few enough elements took part in a pass, those of
// the bin it chose, a few hundred of the row at most, go to every CTA of the cluster, and each finds c among them by itself:
// the largest key whose sum (over + the candidates of its key and above) reaches the limit.  share > 0: the limit is that share
// of the sum of all w, which the first pass finds.  False: there are too many candidates, none reaches the limit, or an
// element's distance is no number; the caller then searches bit by bit.
// Two or three passes and the lists instead of eight passes (8 rows of 151 936, microseconds: top-p 66 -> 41, top-k 51 -> 34).
#define SMPC_NEAR 64            // candidates that a CTA may bring
struct NearList {
    float2 got[SMPC_CTAS * SMPC_NEAR], list[SMPC_CTAS * SMPC_NEAR];     // key (as bits) and w
    int counts[SMPC_CTAS], scan[32];
    uint32_t best[32];
    float2 kept[SMPC_CTAS * SMPC_NEAR];     // of the cluster's first CTA: what is left of the row (index as bits, logit).  Its own
    int kept_counts[SMPC_CTAS];             // place: no meeting parts it from the reading of the lists above
};

template <typename Element>
__device__ __forceinline__ bool cluster_near(ClusterSum& c, float* bins, NearList& nl, const float* sl, float mx, float scale, int n, float limit,
                                             float share, bool above, Element element, uint32_t& answer) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (!(scale > 0.f && scale <= 1e30f)) return false;
    auto place = [&](int i) { return 4095 - min((int)((mx - sl[i]) * scale), 4095); };
    uint32_t prefix = 0;
    float over = 0.f;
    int all = 0;
    for (int shift = 8;; shift -= 4) {
        if (shift < 0) return false;
        float v[16], seen = 0.f;
#pragma unroll
        for (int d = 0; d < 16; ++d) v[d] = 0.f;
        for (int i = threadIdx.x; i < n; i += SMPC_THREADS) {
            const uint32_t at = (uint32_t)place(i);
            if (shift == 8) {
                if (!(mx - sl[i] >= 0.f)) seen += 1e9f;         // (no number: a count that no list is made for)
            } else if ((at ^ prefix) >> (shift + 4)) {
                continue;
            }
            seen += 1.f;
            uint32_t key;
            float w;
            element(i, key, w);
            const uint32_t digit = at >> shift & 15u;
#pragma unroll
            for (uint32_t d = 0; d < 16; ++d) v[d] += digit == d ? w : 0.f;
        }
        bool found;
        prefix |= cluster_bins(c, bins, v, seen, limit, above, over, found, shift == 8 ? share : 0.f) << shift;
        if (!found || seen >= 1e9f || !(prefix >> 8)) return false;     // (or it lies in the bin of all that is far)
        if (seen > 8.f * SMPC_CTAS * SMPC_NEAR) continue;       // (spread evenly over the bins: half of the lists)
        // this CTA's candidates, thread by thread, then index by index
        int mine = 0;
        for (int i = threadIdx.x; i < n; i += SMPC_THREADS) mine += (uint32_t)place(i) >> shift == prefix >> shift;
        int upto = mine;
#pragma unroll
        for (int h = 1; h < 32; h <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, upto, h);
            if (lane >= h) upto += up;
        }
        if (lane == 31) nl.scan[warp] = upto;
        __syncthreads();
        int total = 0, before = upto - mine;
#pragma unroll
        for (int q = 0; q < 32; ++q) {
            if (q == warp) before += total;
            total += nl.scan[q];
        }
        if (mine && total <= SMPC_NEAR)
            for (int i = threadIdx.x; i < n; i += SMPC_THREADS) {
                if ((uint32_t)place(i) >> shift != prefix >> shift) continue;
                uint32_t key;
                float w;
                element(i, key, w);
                const uint32_t to = (uint32_t)__cvta_generic_to_shared(&nl.got[c.rank * SMPC_NEAR + before++]);
#pragma unroll
                for (int r = 0; r < SMPC_CTAS; ++r) {
                    const uint32_t at = cluster_map(to, r);
                    cluster_store_f32(at, __uint_as_float(key));
                    cluster_store_f32(at + 4, w);
                }
            }
        if (threadIdx.x < SMPC_CTAS)
            cluster_store_f32(cluster_map((uint32_t)__cvta_generic_to_shared(&nl.counts[c.rank]), threadIdx.x), __int_as_float(total));
        cluster_sync_all();
        int my_off = 0;
        bool fits = true;
        const int of = threadIdx.x / SMPC_NEAR;
        all = 0;
#pragma unroll
        for (int r = 0; r < SMPC_CTAS; ++r) {
            const int k = nl.counts[r];
            if (r == of) my_off = all;
            all += k;
            fits = fits && k <= SMPC_NEAR;
        }
        if (!fits) continue;        // (the next pass meets before anybody writes a list or a count again)
        if (of < SMPC_CTAS && (int)(threadIdx.x % SMPC_NEAR) < nl.counts[of]) nl.list[my_off + threadIdx.x % SMPC_NEAR] = nl.got[threadIdx.x];
        __syncthreads();
        break;
    }
    uint32_t best = 0;
    for (int q = warp; q < all; q += SMPC_THREADS / 32) {
        const uint32_t key = __float_as_uint(nl.list[q].x);
        float sum = 0.f;
        for (int j = lane; j < all; j += 32) {
            const float2 e = nl.list[j];
            sum += __float_as_uint(e.x) >= key ? e.y : 0.f;
        }
        const float at = over + warp_sum(sum);
        if (above ? at > limit : at >= limit) best = max(best, key);
    }
    if (lane == 0) nl.best[warp] = best;
    __syncthreads();
    best = nl.best[lane];
#pragma unroll
    for (int h = 16; h > 0; h >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, h));
    answer = best;
    return best != 0;
}

// What is left of a row after a top-k of a few dozen: each CTA's kept entries go to the cluster's first, in index order, which
// makes the top-p cut and the draw alone: one meeting and no pass over the row instead of five and four (8 rows of 151 936 with
// both rules: 53 -> 34 us, 92 with all cuts bit by bit).  The rules are the whole row's.  False: a CTA has more than a list's
// share; the row goes on whole.
#define SMPC_FEW 256            // top-k up to which it is tried: half of what the lists hold, as a row's best may lie unevenly
__device__ __forceinline__ bool sample_few(ClusterSum& c, NearList& nl, float* table, const float* sl, const float* se, float mx, int lo, int n,
                                           uint32_t cut, float mp, float tp, uint64_t seed, uint64_t counter, int* out_token, float* out_logprob) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // a thread's share is a run of neighbours, so the lists are in index order
    const int chunk = (n + SMPC_THREADS - 1) / SMPC_THREADS, c_lo = min(n, (int)threadIdx.x * chunk), c_hi = min(n, c_lo + chunk);
    auto kept = [&](int i) { return order_key(sl[i]) >= cut && !(mp > 0.f && se[i] < mp); };
    int mine = 0;
    for (int i = c_lo; i < c_hi; ++i) mine += kept(i);
    int upto = mine;
#pragma unroll
    for (int h = 1; h < 32; h <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, upto, h);
        if (lane >= h) upto += up;
    }
    __syncthreads();
    if (lane == 31) nl.scan[warp] = upto;
    __syncthreads();
    int total = 0, at = upto - mine;
#pragma unroll
    for (int q = 0; q < 32; ++q) {
        if (q == warp) at += total;
        total += nl.scan[q];
    }
    if (mine && total <= SMPC_NEAR)
        for (int i = c_lo; i < c_hi; ++i) {
            if (!kept(i)) continue;
            const uint32_t to = cluster_map((uint32_t)__cvta_generic_to_shared(&nl.kept[c.rank * SMPC_NEAR + at++]), 0);
            cluster_store_f32(to, __int_as_float(lo + i));
            cluster_store_f32(to + 4, sl[i]);
        }
    if (threadIdx.x < SMPC_CTAS)
        cluster_store_f32(cluster_map((uint32_t)__cvta_generic_to_shared(&nl.kept_counts[c.rank]), threadIdx.x), __int_as_float(total));
    cluster_sync_all();
    int all = 0, my_off = 0;
    bool fits = true;
    const int of = threadIdx.x / SMPC_NEAR;
#pragma unroll
    for (int r = 0; r < SMPC_CTAS; ++r) {
        const int k = nl.kept_counts[r];
        if (r == of) my_off = all;
        all += k;
        fits = fits && k <= SMPC_NEAR;
    }
    if (!fits || all == 0) return false;
    if (c.rank != 0) return true;
    if (of < SMPC_CTAS && (int)(threadIdx.x % SMPC_NEAR) < nl.kept_counts[of])
        nl.list[my_off + threadIdx.x % SMPC_NEAR] = nl.kept[threadIdx.x];
    __syncthreads();
    const bool in = (int)threadIdx.x < all;
    const float s = in ? nl.list[threadIdx.x].y : 0.f;
    float e = in ? expf(s - mx) : 0.f;
    if (tp > 0.f && tp < 1.f) {
        if (threadIdx.x < SMPC_CTAS * SMPC_NEAR) nl.got[threadIdx.x] = make_float2(__uint_as_float(order_key(s)), e);
        const float limit = tp * block_sum(e, table);       // (its barriers also make the list the block's)
        uint32_t best = 0;
        for (int q = warp; q < all; q += SMPC_THREADS / 32) {
            const uint32_t key = __float_as_uint(nl.got[q].x);
            float sum = 0.f;
            for (int j = lane; j < all; j += 32) {
                const float2 o = nl.got[j];
                sum += __float_as_uint(o.x) >= key ? o.y : 0.f;
            }
            if (warp_sum(sum) > limit) best = max(best, key);
        }
        __syncthreads();
        if (lane == 0) nl.best[warp] = best;
        __syncthreads();
        best = nl.best[lane];
#pragma unroll
        for (int h = 16; h > 0; h >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, h));
        if (order_key(s) < best) e = 0.f;
    }
    // the draw: running sums in index order
    const bool live = in && e > 0.f;
    float run = e;
#pragma unroll
    for (int h = 1; h < 32; h <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, run, h);
        if (lane >= h) run += up;
    }
    __syncthreads();
    if (lane == 31) table[warp] = run;
    __syncthreads();
    float front = 0.f, whole = 0.f;
#pragma unroll
    for (int q = 0; q < 32; ++q) {
        if (q == warp) front = whole;
        whole += table[q];
    }
    const float target = philox_uniform(seed, counter) * whole;
    // the first whose running sum reaches the target; the last that is kept, if rounding leaves the target beyond all
    const uint32_t reached = __ballot_sync(0xffffffffu, live && front + run >= target), alive = __ballot_sync(0xffffffffu, live);
    __syncthreads();
    if (lane == 0) {
        nl.scan[warp] = reached ? warp * 32 + __ffs(reached) - 1 : 0x7fffffff;
        nl.best[warp] = alive ? warp * 32 + 31 - __clz(alive) + 1 : 0;
    }
    __syncthreads();
    if (warp == 0) {
        const int first = __reduce_min_sync(0xffffffffu, nl.scan[lane]), last = (int)__reduce_max_sync(0xffffffffu, nl.best[lane]) - 1;
        const int pick = first != 0x7fffffff ? first : max(last, 0);
        if (lane == 0) {
            *out_token = __float_as_int(nl.list[pick].x);
            if (out_logprob) *out_logprob = (nl.list[pick].y - mx) - logf(whole);
        }
    }
    return true;
}

__global__ void __launch_bounds__(SMPC_THREADS)
sample_cluster_kernel(const float* __restrict__ logits, int ld, int V, int slice, const float* __restrict__ temperature,
                      const int* __restrict__ top_k, const float* __restrict__ top_p, const float* __restrict__ min_p,
                      const unsigned long long* __restrict__ seed, const unsigned long long* __restrict__ counter,
                      int* __restrict__ out_token, float* __restrict__ out_logprob) {
    extern __shared__ float sl[];               // this CTA's slice of the scaled logits, and behind it exp(logit - maximum)
    __shared__ float parts[2 * SMPC_CTAS], bins[2 * SMPC_CTAS * 17];
    __shared__ NearList near;
    __shared__ float sums[2 * SMPC_CTAS];
    __shared__ float warps[32], table[32 * 17];
    __shared__ float scan[SMPC_THREADS];
    __shared__ float bestv[2 * SMPC_CTAS];
    __shared__ int owner_s;
    __shared__ float before_s, target_s;
    cluster_arrive();           // (waited for before the first word to a peer)
    ClusterSum cs;
    cs.parts = parts; cs.warps = warps; cs.table = table; cs.turn = 0; cs.rank = cluster_ctarank();
    const int r = blockIdx.x / SMPC_CTAS;
    const float* row = logits + (size_t)r * ld;
    const int lo = (int)cs.rank * slice, hi = min(V, lo + slice), n = max(0, hi - lo);
    const float temp = temperature[r];
    const bool greedy = temp <= 0.f;
    const float inv_t = greedy ? 1.f : 1.f / fmaxf(temp, 1e-5f);
    float mx = -INFINITY;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float v = row[lo + i] * inv_t;
        sl[i] = v;
        mx = fmaxf(mx, v);
    }
    cluster_wait();             // every CTA of the row has started
    const int k = top_k[r];
    const float tp = top_p[r];
    float scale = 0.f;                      // (either meeting's barriers also make the slice visible to the CTA's threads)
    if (!greedy && ((k > 0 && k < V) || (tp > 0.f && tp < 1.f))) {
        float mean;                         // of the threads' maxima
        mx = cluster_max_and_mean(cs, sums, mx, mean);
        scale = 1536.f / (mx - mean);
    } else {
        mx = cluster_all_max(cs, mx);
    }

    if (greedy) {
        // the lowest index that holds the maximum: the smallest of the CTAs' candidates (slices are in index order)
        int bi = 0x7fffffff;
        for (int i = threadIdx.x; i < n; i += blockDim.x)
            if (sl[i] == mx) bi = min(bi, lo + i);
        const float first = -cluster_all_max(cs, bi == 0x7fffffff ? -INFINITY : -(float)bi);     // indices < 2^24: exact
        const int pick = first == INFINITY ? 0 : (int)first;
        float z = 0.f;
        if (out_logprob) {
            float local = 0.f;
            for (int i = threadIdx.x; i < n; i += blockDim.x) local += expf(sl[i] - mx);
            z = cluster_all_sum(cs, local);
        }
        if (cs.rank == 0 && threadIdx.x == 0) {
            out_token[r] = pick;
            if (out_logprob) out_logprob[r] = -logf(z);
        }
        return;
    }

    // the exponentials once, for all the passes that follow (a pass is bound by its instructions, of which the
    // exponential was a third: 160 -> 142 us for 8 rows of 151 936)
    float* se = sl + slice;
    for (int i = threadIdx.x; i < n; i += blockDim.x) se[i] = expf(sl[i] - mx);
    __syncthreads();
    uint32_t cut = 0;  // keys >= cut are kept
    const float mp = min_p[r];
    const bool use_minp = mp > 0.f;
    if (k > 0 && k < V) {   // the largest c with count(key >= c) >= k
        auto element = [&](int i, uint32_t& key, float& w) { key = order_key(sl[i]); w = 1.f; };
        const bool few = cluster_near(cs, bins, near, sl, mx, scale, n, (float)k, 0.f, false, element, cut);
        if (!few) cut = cluster_descend(cs, bins, n, (float)k, false, element);
        if (few && k <= SMPC_FEW &&
            sample_few(cs, near, table, sl, se, mx, lo, n, cut, use_minp ? mp : 0.f, tp, seed[r], counter[r], out_token + r,
                       out_logprob ? out_logprob + r : nullptr))
            return;
    }
    if (tp > 0.f && tp < 1.f) {
        // the largest t with mass(key > t) > limit, that is with mass(key - 1 >= t) > limit
        const uint32_t kept_from = cut;
        auto element = [&](int i, uint32_t& key, float& w) {
            const uint32_t full = order_key(sl[i]);
            const float e = se[i];
            key = full - 1u;
            w = full >= kept_from && full != 0u && !(use_minp && e < mp) ? e : 0.f;
        };
        uint32_t t;
        if (!cluster_near(cs, bins, near, sl, mx, scale, n, 0.f, tp, true, element, t)) {
            float z = 0.f;
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                const float s = sl[i];
                const float e = se[i];
                if (order_key(s) >= cut && !(use_minp && e < mp)) z += e;
            }
            z = cluster_all_sum(cs, z);
            t = cluster_descend(cs, bins, n, tp * z, true, element);
        }
        cut = t + 1u > cut ? t + 1u : cut;
    }

    // inverse CDF in index order: CTA by CTA, inside a CTA each thread owns a contiguous range of its slice
    const int chunk = (n + (int)blockDim.x - 1) / (int)blockDim.x;
    const int c_lo = min(n, (int)threadIdx.x * chunk), c_hi = min(n, c_lo + chunk);
    float local = 0.f;
    for (int i = c_lo; i < c_hi; ++i) {
        const float s = sl[i];
        const float e = se[i];
        if (order_key(s) >= cut && !(use_minp && e < mp)) local += e;
    }
    scan[threadIdx.x] = local;
    // every CTA learns every CTA's total (the same exchange as a sum's, read part by part)
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        float v = warp_sum(local);
        if (lane == 0) warps[warp] = v;
        __syncthreads();
        if (warp == 0) {
            float tot = lane < (int)(blockDim.x >> 5) ? warps[lane] : 0.f;
            tot = warp_sum(tot);
            if (lane < SMPC_CTAS)
                cluster_store_f32(cluster_map((uint32_t)__cvta_generic_to_shared(bestv + cs.rank), lane), tot);
        }
        cluster_sync_all();
    }
    float run = 0.f;
#pragma unroll
    for (int c = 0; c < SMPC_CTAS; ++c) run += bestv[c];
    const float u = philox_uniform(seed[r], counter[r]);
    const float target = u * run;
    // the CTA in which the target falls (the last CTA with anything kept, if rounding leaves the target beyond all)
    int owner_cta = -1, last_cta = 0;
    float acc = 0.f, before_cta = 0.f;
#pragma unroll
    for (int c = 0; c < SMPC_CTAS; ++c) {
        if (bestv[c] > 0.f) last_cta = c;
        if (owner_cta < 0 && bestv[c] > 0.f && acc + bestv[c] >= target) { owner_cta = c; before_cta = acc; }
        if (owner_cta < 0) acc += bestv[c];
    }
    if (owner_cta < 0) { owner_cta = last_cta; before_cta = acc - bestv[last_cta]; }
    if ((int)cs.rank != owner_cta) return;
    // the thread in whose range the target falls, by the first warp: 32 ranges a lane, their sums, then the lane's ranges
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        float mine = 0.f;
        int last = -1;          // the lane's last range with anything kept
        for (int t = lane * 32; t < lane * 32 + 32; ++t) {
            mine += scan[t];
            if (scan[t] > 0.f) last = t;
        }
        float upto = mine;      // the sum of this lane's ranges and those in front
#pragma unroll
        for (int h = 1; h < 32; h <<= 1) {
            const float up = __shfl_up_sync(0xffffffffu, upto, h);
            if (lane >= h) upto += up;
        }
        const uint32_t reached = __ballot_sync(0xffffffffu, last >= 0 && before_cta + upto >= target);
        const uint32_t kept = __ballot_sync(0xffffffffu, last >= 0);     // (a sum that is no number hides no range that is one)
        const int at = reached ? __ffs(reached) - 1 : kept ? 31 - __clz(kept) : 0;      // (rounding may leave the target beyond all)
        const float front = __shfl_up_sync(0xffffffffu, upto, 1);
        if (lane == at) {
            float a2 = before_cta + (lane ? front : 0.f), start = a2;
            int owner = -1;
            for (int t = lane * 32; t < lane * 32 + 32 && owner < 0; ++t) {
                if (!(scan[t] > 0.f)) continue;
                start = a2;
                a2 += scan[t];
                if (a2 >= target || t == last) owner = t;
            }
            owner_s = owner < 0 ? 0 : owner;
            before_s = start;
            target_s = target;
        }
    }
    __syncthreads();
    if ((int)threadIdx.x == owner_s) {
        float a3 = before_s;
        int pick = -1, last_kept = -1;
        for (int i = c_lo; i < c_hi; ++i) {
            const float s = sl[i];
            const float e = se[i];
            if (order_key(s) >= cut && !(use_minp && e < mp)) {
                last_kept = i;
                a3 += e;
                if (a3 >= target_s) { pick = i; break; }
            }
        }
        if (pick < 0) pick = last_kept;
        out_token[r] = lo + pick;
        if (out_logprob) out_logprob[r] = (sl[pick] - mx) - logf(run);
    }
}

ACV_API int acv_sample(const float* logits, int ld, int rows, int V, const float* temperature, const int* top_k,
                       const float* top_p, const float* min_p, const unsigned long long* seed,
                       const unsigned long long* counter, int* out_token, float* out_logprob, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (V <= 0) return ACV_ERR_SIZE;
    // wide rows: a cluster of CTAs to a row, the row's slices in their shared memory
    const int slice = ((V + SMPC_CTAS - 1) / SMPC_CTAS + 3) & ~3;
    const int smem = 2 * slice * (int)sizeof(float);
    if (V >= 16384 && V < (1 << 24) && smem <= 200 * 1024) {
        static AcvSmemConfig smem_config;
        if (int rc = acv_ensure_smem(smem_config, sample_cluster_kernel, smem)) return rc;
        acv_launch_cluster(0, dim3(SMPC_CTAS, 1, 1), sample_cluster_kernel, dim3((unsigned)rows * SMPC_CTAS), dim3(SMPC_THREADS),
                           (size_t)smem, stream, logits, ld, V, slice, temperature, top_k, top_p, min_p, seed, counter,
                           out_token, out_logprob);
        return acv_launch_status();
    }
    sample_kernel<<<rows, SMP_THREADS, 0, stream>>>(logits, ld, V, temperature, top_k, top_p, min_p, seed, counter,
                                                    out_token, out_logprob);
    return acv_launch_status();
}

// ----------------------------------------------------------------------------- the k most probable tokens
// For each row the k largest logits in falling order (equal values: the lower index first) with their log
// probabilities logit - logsumexp(row), the normalisation of the chosen token's log probability
// (acvram/engine/sampler.py:103-117).  One block per row: a pass for the maximum and the sum of exponentials,
// then k passes, each finding the largest entry that comes after the one found before it.
#define TOPLP_MAX_K 64
__global__ void __launch_bounds__(SMP_THREADS)
top_logprobs_kernel(const float* __restrict__ logits, int ld, int V, int k, int* __restrict__ out_ids,
                    float* __restrict__ out_lp) {
    __shared__ float redf[32];
    __shared__ int redi[32];
    const float* row = logits + (size_t)blockIdx.x * ld;
    float mx = -INFINITY;
    for (int i = threadIdx.x; i < V; i += blockDim.x) mx = fmaxf(mx, row[i]);
    mx = block_reduce_max(mx, redf);
    float sum = 0.f;
    for (int i = threadIdx.x; i < V; i += blockDim.x) sum += __expf(row[i] - mx);
    sum = block_reduce_sum(sum, redf);
    const float lse = mx + logf(sum);
    float prev_v = INFINITY;
    int prev_i = -1;
    for (int n = 0; n < k; ++n) {
        float best = -INFINITY;
        int bi = 0x7fffffff;
        for (int i = threadIdx.x; i < V; i += blockDim.x) {
            const float v = row[i];
            const bool after = v < prev_v || (v == prev_v && i > prev_i);      // not yet given out
            if (after && v > -INFINITY && (v > best || (v == best && i < bi))) { best = v; bi = i; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
        __syncthreads();
        if (lane == 0) { redf[warp] = best; redi[warp] = bi; }
        __syncthreads();
        best = lane < nwarp ? redf[lane] : -INFINITY;
        bi = lane < nwarp ? redi[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if (bi == 0x7fffffff) {              // fewer than k finite entries are left (k > V, or a row of -inf)
            if (threadIdx.x == 0) { out_ids[(size_t)blockIdx.x * k + n] = -1; out_lp[(size_t)blockIdx.x * k + n] = -INFINITY; }
            continue;
        }
        if (threadIdx.x == 0) {
            out_ids[(size_t)blockIdx.x * k + n] = bi;
            out_lp[(size_t)blockIdx.x * k + n] = best - lse;
        }
        prev_v = best;
        prev_i = bi;
    }
}

// logits float [rows, V] (row stride ld); out_ids int [rows, k], out_lp float [rows, k]; 1 <= k <= 64.
ACV_API int acv_top_logprobs(const float* logits, int ld, int rows, int V, int k, int* out_ids, float* out_lp,
                             cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (V <= 0 || k < 1 || k > TOPLP_MAX_K) return ACV_ERR_SIZE;
    top_logprobs_kernel<<<rows, SMP_THREADS, 0, stream>>>(logits, ld, V, k, out_ids, out_lp);
    return acv_launch_status();
}

ACV_TL_EXPORT(sampling)
