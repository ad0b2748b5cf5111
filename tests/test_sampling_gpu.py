"""The sampling kernels against the plain sampler."""

from __future__ import annotations

import math

import pytest
import torch

import plain_qwen3

pytestmark = pytest.mark.gpu


def run_sample(logits, temperature, top_k, top_p, min_p, seeds, counters, logprobs=False):
    from acvram_b200.kernels import ops
    R = logits.shape[0]
    dev = "cuda"
    f = lambda v: torch.tensor(v, dtype=torch.float32, device=dev)
    out = torch.empty(R, dtype=torch.int32, device=dev)
    lp = torch.empty(R, dtype=torch.float32, device=dev) if logprobs else None
    ops.sample(logits, f(temperature), torch.tensor(top_k, dtype=torch.int32, device=dev), f(top_p), f(min_p),
               torch.tensor(seeds, dtype=torch.int64, device=dev), torch.tensor(counters, dtype=torch.int64, device=dev),
               out, lp)
    return out.tolist(), (lp.tolist() if logprobs else None)


@pytest.mark.parametrize("V", [331, 4097, 151936])
def test_sample_matches_plain(V):
    g = torch.Generator().manual_seed(V)
    cases = [(0.7, 0, 1.0, 0.0), (1.0, 40, 1.0, 0.0), (1.3, 0, 0.8, 0.0), (0.5, 0, 1.0, 0.05), (0.9, 100, 0.9, 0.01),
             (1.0, 1, 1.0, 0.0), (1.0, 0, 1e-6, 0.0), (0.0, 5, 0.5, 0.1)]
    R = len(cases)
    logits = (torch.randn(R, V, generator=g) * 2.5).cuda()
    seeds = [11 * i + 3 for i in range(R)]
    for counter in (0, 1, 17):
        got, lps = run_sample(logits, [c[0] for c in cases], [c[1] for c in cases], [c[2] for c in cases],
                              [c[3] for c in cases], seeds, [counter] * R, logprobs=True)
        for i, (temp, k, p, mp) in enumerate(cases):
            row = logits[i].cpu()
            if temp <= 0:
                assert got[i] == int(row.argmax())
                continue
            scaled = plain_qwen3.filtered_distribution(row, temp, k, mp, p)
            want = plain_qwen3.draw(scaled, plain_qwen3.philox_uniform(seeds[i], counter))
            assert got[i] == want, f"case {i} counter {counter}"
            assert torch.isfinite(scaled[got[i]]), "a dropped token was drawn"
            assert abs(lps[i] - float(torch.log_softmax(scaled, -1)[got[i]])) < 1e-3


@pytest.mark.parametrize("V", [16384, 16389, 40000])
@pytest.mark.parametrize("kind", ["equal", "two", "spread", "negative", "holes"])
def test_wide_rows_cut_where_the_plain_sampler_cuts(V, kind):
    """Rows for which the cut's bits are all of one kind: one value, two values, magnitudes from 1e-30 to 1e3, all below
    zero, -inf in places; a top-k at a tie keeps every equal value."""
    g = torch.Generator().manual_seed(V)
    row = {"equal": lambda: torch.full((V,), 1.5), "two": lambda: torch.where(torch.rand(V, generator=g) < 0.5, 1.0, 1.0000001),
           "spread": lambda: torch.randn(V, generator=g) * 10.0 ** (torch.rand(V, generator=g) * 33 - 30),
           "negative": lambda: -torch.rand(V, generator=g) * 20 - 1e-3,
           "holes": lambda: torch.randn(V, generator=g).masked_fill(torch.rand(V, generator=g) < 0.7, float("-inf"))}[kind]()
    cases = [(1.0, 7, 1.0, 0.0), (1.0, 0, 0.5, 0.0), (0.7, 1000, 0.9, 0.0), (1.0, V - 1, 0.99, 0.001), (1.0, 1, 0.3, 0.0)]
    R = len(cases)
    got, _ = run_sample(row.repeat(R, 1).cuda(), *[[c[j] for c in cases] for j in (0, 1, 2, 3)], list(range(R)), [3] * R)
    for i, (temp, k, p, mp) in enumerate(cases):
        x = (row / temp).double()
        weight = (x - x.max()).exp()
        keep = x >= x.topk(k).values[-1] if 0 < k < V else torch.ones(V, dtype=torch.bool)
        keep &= weight >= mp
        values, at = torch.unique(x[keep], return_inverse=True)         # ascending; equal values stay or go together
        mass = torch.zeros(len(values), dtype=torch.float64).index_add_(0, at, weight[keep])
        above = mass.flip(0).cumsum(0).flip(0) - mass
        if p < 1.0:         # a value goes when the mass above it exceeds p
            keep &= x >= values[above <= p * mass.sum() * (1 + 1e-6)][0]
        assert keep[got[i]], f"case {i}: a dropped token was drawn"
        # (where the draw falls between two tokens by less than the sums' rounding either may come)
        cdf = torch.where(keep, weight, 0.0).cumsum(0) / weight[keep].sum()
        u = plain_qwen3.philox_uniform(i, 3)
        before = float(cdf[got[i]] - weight[got[i]] / weight[keep].sum())
        assert before - 1e-4 <= u <= float(cdf[got[i]]) + 1e-4, f"case {i}"


@pytest.mark.parametrize("V", [16384, 151936])
@pytest.mark.parametrize("kind", ["cold", "hot", "crowded", "far", "lowest"])
def test_wide_rows_whose_cut_is_searched_near_the_maximum(V, kind):
    """The search by distance from the maximum: two passes and the lists, three, more candidates than a list holds, a cut in the
    bin of all that is far, half of the row at the type's lowest value; a draw just inside the kept mass, whatever the seed."""
    g = torch.Generator().manual_seed(V + 1)
    x = torch.randn(V, generator=g)
    row = {"cold": lambda: x * 9, "hot": lambda: x * 0.01, "crowded": lambda: (x * 40).round() / 40,
           "far": lambda: torch.cat([x[: V // 2], x[V // 2:] * 1e-3 - 60.0]), "lowest": lambda: torch.where(x < 0, torch.finfo(torch.float32).min, x)}[kind]()
    cases = [(1.0, 50, 1.0, 0.0), (1.0, 0, 0.9, 0.0), (1.0, V // 2 + 1000, 1.0, 0.0), (1.0, V - 3, 0.9995, 0.0), (1.0, 300, 0.95, 0.01), (1.0, 64, 1.0, 0.0)]
    R = len(cases)
    for counter in range(3):
        got, _ = run_sample(row.repeat(R, 1).cuda(), *[[c[j] for c in cases] for j in (0, 1, 2, 3)], list(range(R)), [counter] * R)
        for i, (_, k, p, mp) in enumerate(cases):
            z = row.double()
            weight = (z - z.max()).exp()
            keep = z >= z.topk(k).values[-1] if 0 < k < V else torch.ones(V, dtype=torch.bool)
            keep &= weight >= mp
            if p < 1.0:
                values, at = torch.unique(z[keep], return_inverse=True)
                mass = torch.zeros(len(values), dtype=torch.float64).index_add_(0, at, weight[keep])
                above = mass.flip(0).cumsum(0).flip(0) - mass
                keep &= z >= values[above <= p * mass.sum() * (1 + 1e-6)][0]
            assert keep[got[i]], f"case {i}: a dropped token was drawn"
            cdf = torch.where(keep, weight, 0.0).cumsum(0) / weight[keep].sum()
            u = plain_qwen3.philox_uniform(i, counter)
            before = float(cdf[got[i]] - weight[got[i]] / weight[keep].sum())
            assert before - 1e-4 <= u <= float(cdf[got[i]]) + 1e-4, f"case {i}"


@pytest.mark.parametrize("kind", ["spread", "ties", "clumped", "below"])
@pytest.mark.parametrize("V", [16384, 50001])
def test_wide_rows_of_which_a_top_k_leaves_few(V, kind):
    """The cut and the draw on the entries that a small top-k leaves: one, a list's share and one more, the most and one more;
    many of one value; all in one part of the row; a probability floor that leaves the maximum alone.  The draw is the kept
    mass's at the seed's point (a float sum of at most V weights is good to 1e-4 of it), and its log-probability is the share's."""
    g = torch.Generator().manual_seed(V + 2)
    x = torch.randn(V, generator=g)
    row = {"spread": lambda: x * 2, "ties": lambda: (x * 4).round() / 2, "clumped": lambda: torch.where(torch.arange(V) < 500, x + 6.0, x),
           "below": lambda: torch.where(torch.arange(V) == V - 1, 30.0, x)}[kind]()
    cases = [(k, p, mp) for k in (1, 2, 63, 64, 65, 256, 257) for p, mp in ((1.0, 0.0), (0.9, 0.0), (0.3, 0.05))]
    for counter in range(3):
        got, logprob = run_sample(row.repeat(len(cases), 1).cuda(), [1.0] * len(cases), *[[c[j] for c in cases] for j in (0, 1, 2)],
                                  list(range(len(cases))), [counter] * len(cases), logprobs=True)
        for i, (k, p, mp) in enumerate(cases):
            z = row.double()
            weight = (z - z.max()).exp()
            keep = (z >= z.topk(k).values[-1]) & (weight >= mp)
            if p < 1.0:
                values, at = torch.unique(z[keep], return_inverse=True)
                mass = torch.zeros(len(values), dtype=torch.float64).index_add_(0, at, weight[keep])
                above = mass.flip(0).cumsum(0).flip(0) - mass
                keep &= z >= values[above <= p * mass.sum() * (1 + 1e-6)][0]
            assert keep[got[i]], f"case {cases[i]}: a dropped token was drawn"
            share = weight / weight[keep].sum()
            upto = float(torch.where(keep, share, 0.0).cumsum(0)[got[i]])
            u = plain_qwen3.philox_uniform(i, counter)
            assert upto - float(share[got[i]]) - 1e-4 <= u <= upto + 1e-4, f"case {cases[i]}"
            assert abs(float(logprob[i]) - math.log(float(share[got[i]]))) < 1e-4, f"case {cases[i]}"


@pytest.mark.parametrize("at", [(100, 104), (104, 100), (100, 2040), (0, 63)])
def test_a_wide_row_with_a_logit_that_is_no_number_gives_a_kept_token(at):
    """Top-k 2 of a row whose largest entries are NaN and a number, in the same part of the row: the number is drawn."""
    row = torch.zeros(16384)
    row[at[0]], row[at[1]] = float("nan"), 5.0
    got, _ = run_sample(row[None].cuda(), [1.0], [2], [1.0], [0.0], [7], [3])
    assert list(got) == [at[1]]


def test_draws_follow_the_distribution():
    """Many counters on one row: the empirical frequencies approach the kept probabilities."""
    V = 50
    g = torch.Generator().manual_seed(1)
    row = torch.randn(V, generator=g) * 2
    n = 4000
    logits = row.repeat(n, 1).cuda()
    got, _ = run_sample(logits, [0.8] * n, [10] * n, [1.0] * n, [0.0] * n, [5] * n, list(range(n)))
    probs = torch.softmax(plain_qwen3.filtered_distribution(row, 0.8, 10, 0.0, 1.0), -1)
    freq = torch.bincount(torch.tensor(got), minlength=V).float() / n
    assert (freq[probs == 0] == 0).all()
    assert (freq - probs).abs().max() < 0.03


def test_penalties():
    from acvram_b200.kernels import ops
    V = 64
    g = torch.Generator().manual_seed(2)
    logits = torch.randn(2, V, generator=g)
    hist = [[3, 3, 9, 11, 3], [5]]
    want = torch.stack([plain_qwen3.penalised(logits[0], hist[0], 1.3, 0.5, 0.2),
                        plain_qwen3.penalised(logits[1], hist[1], 1.0, 0.0, 0.7)])
    dev = logits.cuda()
    rows = torch.tensor([0, 0, 0, 1], dtype=torch.int32).cuda()
    toks = torch.tensor([3, 9, 11, 5], dtype=torch.int32).cuda()
    cnts = torch.tensor([3, 1, 1, 1], dtype=torch.int32).cuda()
    f = lambda v: torch.tensor(v, dtype=torch.float32).cuda()
    ops.apply_penalties(dev, rows, toks, cnts, f([1.3, 1.0]), f([0.5, 0.0]), f([0.2, 0.7]))
    torch.testing.assert_close(dev.cpu(), want, rtol=1e-6, atol=1e-6)


def test_sampler_object_mixes_greedy_and_sampled_rows():
    from acvram_b200.sampling import Sampler, SamplingParams
    V = 300
    g = torch.Generator().manual_seed(3)
    logits = (torch.randn(3, V, generator=g) * 2).cuda()
    params = [SamplingParams(temperature=0.0), SamplingParams(temperature=0.8, top_k=20, seed=4),
              SamplingParams(temperature=0.0, repetition_penalty=50.0)]
    best = int(logits[2].argmax())
    toks, _ = Sampler("cuda")(logits, params, [(), (), [best]], [1, 4, 2], [0, 6, 0])
    toks = toks.tolist()
    assert toks[0] == int(logits[0].argmax())
    scaled = plain_qwen3.filtered_distribution(logits[1].cpu(), 0.8, 20, 0.0, 1.0)
    assert toks[1] == plain_qwen3.draw(scaled, plain_qwen3.philox_uniform(4, 6))
    assert toks[2] != best, "the repetition penalty moved the greedy choice"


@pytest.mark.parametrize("V,k", [(331, 5), (4097, 1), (151936, 20), (7, 7), (5, 8)])
def test_top_logprobs_kernel(V, k):
    """The k most probable tokens of each row with logit - logsumexp, against a sort in float64; equal logits
    come lowest id first; a row shorter than k ends with id -1 and -inf."""
    from acvram_b200.kernels import ops
    g = torch.Generator().manual_seed(V + k)
    logits = (torch.randn(6, V, generator=g) * 3.0)
    logits[1, : min(V, 4)] = 2.5                    # equal values among the largest
    logits[2, V // 2] = float("-inf")
    if V > 100:
        logits[3] = torch.round(logits[3])          # many equal values
    ids, lp = ops.top_logprobs(logits.cuda(), k)
    ids, lp = ids.cpu(), lp.cpu()
    ref = torch.log_softmax(logits.double(), dim=-1)
    for r in range(6):
        order = sorted(range(V), key=lambda i: (-float(logits[r, i]), i))
        order = [i for i in order if logits[r, i] != float("-inf")][:k]
        assert ids[r, :len(order)].tolist() == order
        torch.testing.assert_close(lp[r, :len(order)].double(), ref[r, order], rtol=1e-5, atol=1e-5)
        assert all(int(i) == -1 for i in ids[r, len(order):]) and all(v == float("-inf") for v in lp[r, len(order):])
