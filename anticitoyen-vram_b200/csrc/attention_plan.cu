// What a step's attention kernels are given, made on the host (no kernel here): the requests with one token, the tiles of the
// others' queries, and how many thread blocks share a tile's keys.  Native because it is made for every step whose lengths are new:
// microseconds in Python, array by array or one by one, and here, 64 one-token requests 14, 21 and 10, 512 57, 124 and 37, a
// prompt of 32768 20, 61 and 9, eight of 8192 beside 128 decoding 73, 161 and 23; the shares of a tile 15 and 2.
#include <algorithm>
#include <new>

#include "common.cuh"

// The B requests' new tokens, tokens in all and first rows (B + 1) of a step.  dec_seqs, dec_tokens [B]: the requests with one new
// token and their rows; tile_seq, tile_q0 [capacity]: the tiles of `tile` queries of those with more, the tiles whose last query sees
// most keys first, equal ones in the batch's order.  counts: requests with one token, tiles, the most tokens that one of either holds,
// and where there are tiles the tiles of `tile` keys that all of them see, the one that sees most, the one that sees least.
ACV_API int acv_attention_work(const int* q_lens, const int* kv_lens, const int* cu_q, int B, int tile, int* dec_seqs, int* dec_tokens,
                               int* tile_seq, int* tile_q0, int capacity, int* counts) {
    if (B < 0 || tile <= 0) return ACV_ERR_SIZE;
    int n_dec = 0, max_dec = 0, max_tile = 0;
    long long n = 0;
    for (int i = 0; i < B; ++i) {
        if (q_lens[i] == 1) {
            dec_seqs[n_dec] = i;
            dec_tokens[n_dec++] = cu_q[i];
            max_dec = std::max(max_dec, kv_lens[i]);
        } else if (q_lens[i] > 1) {
            n += (q_lens[i] + tile - 1) / tile;
            max_tile = std::max(max_tile, kv_lens[i]);
        }
    }
    if (n > capacity) return ACV_ERR_SCRATCH;
    struct Tile { int keys, seq, q0; };
    Tile* tiles = new (std::nothrow) Tile[n + 1];
    if (!tiles) return ACV_ERR_SCRATCH;
    int t = 0, total = 0, longest = 0, shortest = 0;
    for (int i = 0; i < B; ++i)
        for (int q0 = 0; q_lens[i] > 1 && q0 < q_lens[i]; q0 += tile) {
            tiles[t] = {kv_lens[i] - q_lens[i] + std::min(q0 + tile, q_lens[i]), i, q0};
            const int blocks = (tiles[t].keys + tile - 1) / tile;
            total += blocks;
            longest = t ? std::max(longest, blocks) : blocks;
            shortest = t ? std::min(shortest, blocks) : blocks;
            ++t;
        }
    // the hardware hands out CTAs in this order, and the kernel that gives a CTA two tiles pairs the list's front with its back
    std::sort(tiles, tiles + t, [](const Tile& a, const Tile& b) {
        return a.keys != b.keys ? a.keys > b.keys : a.seq != b.seq ? a.seq < b.seq : a.q0 < b.q0;
    });
    for (int i = 0; i < t; ++i) {
        tile_seq[i] = tiles[i].seq;
        tile_q0[i] = tiles[i].q0;
    }
    delete[] tiles;
    const int out[7] = {n_dec, t, max_dec, max_tile, total, longest, shortest};
    for (int i = 0; i < 7; ++i) counts[i] = out[i];
    return 0;
}

// Microseconds in acv_attention_tc: a round of blocks, a round that merges its clusters' parts, a tile of 128 keys of two heads; and
// what a head without a partner takes of that.
static const double TC_FIXED = 4., TC_MERGE = 12., TC_BLOCK = 2.1, TC_ODD = 0.6;

// The least microseconds for `units` of blocks with `work` key tiles in all, and with how many blocks to a unit.
static double tc_parts(long long units, double work, double longest, double shortest, int sms, int most, int* parts) {
    double best = 0.;
    *parts = 0;
    for (int n = 1; n <= std::max(1, std::min(8, most)); ++n) {
        const long long at_once = std::max(1, ACV_CLUSTERS_AT_ONCE[n] * sms / 148);
        double span = n == 1 ? longest : longest / most * ((most + n - 1) / n);
        if (units > at_once) span = std::max(span, work / ((double)n * at_once) + shortest / n);
        const double cost = (double)((units + at_once - 1) / at_once) * (n == 1 ? TC_FIXED : TC_MERGE) + span * TC_BLOCK;
        if (!*parts || cost < (*parts == 1 ? 0.95 * best : best)) {
            best = cost;
            *parts = n;
        }
    }
    return best;
}

// How many blocks share the keys of a tile of queries in acv_attention_tc, by the time of the rounds of blocks that come one after the
// other; beside it (times 16), where they go by a launch of their own, the same for the groups' odd heads.  total, longest, shortest:
// key tiles of all tiles of queries, of the one that sees most, of the one that sees least; limit > 0: none sees more.
ACV_API int acv_attention_tc_parts(int n_tiles, int total, int longest, int shortest, int NH, int NKV, int limit, int sms) {
    if (n_tiles <= 0 || NKV <= 0 || NH < NKV || NH % NKV || longest <= 0) return ACV_ERR_SIZE;
    if (limit > 0 && limit < longest) {
        total = (int)std::min<long long>(total, (long long)n_tiles * limit);
        longest = limit;
        shortest = std::min(shortest, limit);
    }
    const int n_rep = NH / NKV, pairs = n_rep / 2, odd = n_rep % 2;
    const long long each = (long long)n_tiles * NKV;
    int parts, a, b;
    if (n_rep == 1) {       // one head to a block throughout
        tc_parts(each, (double)total * NKV * TC_ODD, longest * TC_ODD, shortest * TC_ODD, sms, longest, &parts);
        return parts;
    }
    const double cost = tc_parts(each * (pairs + odd), (double)total * NKV * (pairs + TC_ODD * odd), longest, shortest * (odd ? TC_ODD : 1.), sms, longest, &parts);
    if (odd) {
        const double both = tc_parts(each * pairs, (double)total * NKV * pairs, longest, shortest, sms, longest, &a) +
                            tc_parts(each, (double)total * NKV * TC_ODD, longest * TC_ODD, shortest * TC_ODD, sms, longest, &b);
        if (both + 3. < 0.95 * cost) return a + 16 * b;
    }
    return parts;
}
