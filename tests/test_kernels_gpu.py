"""Each CUDA kernel alone against its plain PyTorch reference, at sizes other than the engine's."""

from __future__ import annotations

import pytest
import torch

import kernel_refs as ref
from acvram_b200.kernels.ops import QUERY_TILE

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16]


def tol(dtype):
    return dict(rtol=2e-5, atol=2e-5) if dtype == torch.float32 else dict(rtol=1.6e-2, atol=1.6e-2)


@pytest.fixture(scope="module")
def ops():
    from acvram_b200.kernels import ops
    ops.library()
    return ops


def rnd(*shape, dtype=torch.float32, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,V,T", [(72, 331, 9), (4096, 1000, 3), (50, 77, 1)])
def test_embed(ops, dtype, H, V, T):
    table = rnd(V, H, dtype=dtype)
    tok = torch.randint(0, V, (T,), device="cuda", dtype=torch.int32)
    out = torch.empty(T, H, device="cuda", dtype=dtype)
    ops.embed(table, tok, out)
    assert torch.equal(out, table[tok.long()])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,H,eps", [(5, 72, 1e-6), (3, 4096, 1e-5), (2, 5120, 1e-6), (1, 13000, 1e-5), (17, 50, 1e-3)])
def test_add_rmsnorm(ops, dtype, T, H, eps):
    x = rnd(T, H, dtype=dtype, seed=1)
    d = rnd(T, H, dtype=dtype, seed=2)
    w = 1 + 0.1 * rnd(H, seed=3)
    # with the residual sum
    x1, x2 = x.clone(), x.clone()
    o1 = ops.add_rmsnorm(x1, d, w, eps, torch.empty_like(x))
    o2 = ref.add_rmsnorm(x2, d, w, eps, torch.empty_like(x))
    torch.testing.assert_close(x1, x2, **tol(dtype))
    torch.testing.assert_close(o1, o2, **tol(dtype))
    # without, and on chosen rows only
    rows = torch.tensor([T - 1, 0], device="cuda", dtype=torch.int32)
    x3 = x.clone()
    o3 = ops.add_rmsnorm(x3, d, w, eps, torch.empty(2, H, device="cuda", dtype=dtype), rows)
    o4 = ref.add_rmsnorm(x.clone(), d, w, eps, torch.empty(2, H, device="cuda", dtype=dtype), rows)
    assert torch.equal(x3, x), "the rows form must leave x as it is"
    torch.testing.assert_close(o3, o4, **tol(dtype))
    o5 = ops.add_rmsnorm(x.clone(), None, w, eps, torch.empty_like(x))
    o6 = ref.add_rmsnorm(x.clone(), None, w, eps, torch.empty_like(x))
    torch.testing.assert_close(o5, o6, **tol(dtype))


def test_rmsnorm_breaking_arm(ops):
    """The comparison can see a fault: a wrong eps moves the result beyond the tolerance."""
    x = rnd(4, 96, scale=0.01, seed=4)
    w = torch.ones(96, device="cuda")
    good = ops.add_rmsnorm(x.clone(), None, w, 1e-6, torch.empty_like(x))
    bad = ref.add_rmsnorm(x.clone(), None, w, 1e-4, torch.empty_like(x))
    assert (good - bad).abs().max() > 1e-2


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,I", [(7, 176), (2, 12288), (1, 5), (33, 1000)])
def test_swiglu(ops, dtype, T, I):
    gu = rnd(T, 2 * I, dtype=dtype, scale=3.0, seed=5)
    gu[0, 0] = 80.0   # extremes: exp(-g) under- and overflows
    gu[0, 1] = -80.0
    o1 = ops.swiglu(gu, torch.empty(T, I, device="cuda", dtype=dtype))
    o2 = ref.swiglu(gu, torch.empty(T, I, device="cuda", dtype=dtype))
    torch.testing.assert_close(o1, o2, **tol(dtype))
    assert torch.isfinite(o1.float()).all()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T,N", [(1, 17), (9, 331), (300, 4096)])
def test_add_bias(ops, dtype, T, N):
    out = rnd(T, N + 5, dtype=dtype, seed=21)[:, :N]          # a row stride that is not the width
    bias = rnd(N, seed=22)
    want = out.clone()
    ref.add_bias(want, bias)
    ops.add_bias(out, bias)
    torch.testing.assert_close(out, want, **tol(dtype))


def test_table_update(ops):
    """The (row, column, page) triples of a step reach the block table on the device; what lies outside is skipped."""
    table = torch.full((5, 7), -1, dtype=torch.int32, device="cuda")
    triples = torch.tensor([[0, 0, 11], [4, 6, 12], [2, 3, 14], [5, 0, 15], [0, 7, 16], [-1, 2, 17], [1, 1, 99]],
                           dtype=torch.int32, device="cuda").reshape(-1)
    ops.table_update(table, triples, 6)             # the seventh triple is not part of the step
    want = torch.full((5, 7), -1, dtype=torch.int32)
    want[0, 0], want[4, 6], want[2, 3] = 11, 12, 14
    assert torch.equal(table.cpu(), want)


def _paged_setup(B, lens, NKV, D, page, dtype, n_pages, seed, shuffle=True):
    """Random block tables over a shuffled pool; returns (k_pages, v_pages, table[B, W])."""
    g = torch.Generator().manual_seed(seed)
    W = max((l + page - 1) // page for l in lens)
    perm = torch.randperm(n_pages, generator=g) if shuffle else torch.arange(n_pages)
    table = torch.full((B, W), -1, dtype=torch.int32)
    used = 0
    for b, l in enumerate(lens):
        n = (l + page - 1) // page
        table[b, :n] = perm[used:used + n].to(torch.int32)
        used += n
    assert used <= n_pages
    kp = torch.zeros(n_pages, NKV, page, D, device="cuda", dtype=dtype)
    vp = torch.zeros_like(kp)
    return kp, vp, table.cuda()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("NH,NKV,D,rot,page", [(5, 1, 48, 48, 16), (6, 2, 32, 32, 8), (8, 8, 64, 32, 4), (4, 2, 128, 128, 16),
                                              (3, 3, 16, 16, 32)])
def test_qk_norm_rope_append(ops, dtype, NH, NKV, D, rot, page):
    lens = [19, 3, 40]
    q_lens = [5, 3, 1]   # the last tokens of each request are this step's
    B = len(lens)
    kp, vp, table = _paged_setup(B, lens, NKV, D, page, dtype, 16, seed=7)
    kp2, vp2 = kp.clone(), vp.clone()
    pos = torch.cat([torch.arange(l - q, l) for l, q in zip(lens, q_lens)]).to(torch.int32).cuda()
    seq = torch.cat([torch.full((q,), b) for b, q in enumerate(q_lens)]).to(torch.int32).cuda()
    T = pos.numel()
    qkv = rnd(T, (NH + 2 * NKV) * D, dtype=dtype, seed=8)
    qw, kw = 1 + 0.1 * rnd(D, seed=9), 1 + 0.1 * rnd(D, seed=10)
    inv = 1.0 / (10000.0 ** (torch.arange(0, rot, 2, dtype=torch.float32) / rot))
    ang = torch.outer(torch.arange(64, dtype=torch.float32), inv)
    cs = torch.cat((ang.cos(), ang.sin()), -1).cuda()
    a, b = qkv.clone(), qkv.clone()
    ops.qk_norm_rope_append(a, NH, NKV, D, qw, kw, 1e-6, cs, pos, seq, table, kp, vp)
    ref.qk_norm_rope_append(b, NH, NKV, D, qw, kw, 1e-6, cs, pos, seq, table, kp2, vp2)
    torch.testing.assert_close(a[:, :NH * D], b[:, :NH * D], **tol(dtype))
    torch.testing.assert_close(kp, kp2, **tol(dtype))
    torch.testing.assert_close(vp, vp2, **tol(dtype))
    # steps alone: norm only (no table, no pages), then append only
    c, d = qkv.clone(), qkv.clone()
    ops.qk_norm_rope_append(c, NH, NKV, D, qw, kw, 1e-6, None, pos, seq, None, None, None)
    ref.qk_norm_rope_append(d, NH, NKV, D, qw, kw, 1e-6, None, pos, seq, None, None, None)
    torch.testing.assert_close(c, d, **tol(dtype))
    kp3, vp3 = torch.zeros_like(kp), torch.zeros_like(vp)
    ops.qk_norm_rope_append(c, NH, NKV, D, None, None, 0.0, None, pos, seq, table, kp3, vp3)
    kp4, vp4 = torch.zeros_like(kp), torch.zeros_like(vp)
    ref.qk_norm_rope_append(d, NH, NKV, D, None, None, 0.0, None, pos, seq, table, kp4, vp4)
    torch.testing.assert_close(kp3, kp4, **tol(dtype))
    torch.testing.assert_close(vp3, vp4, **tol(dtype))


def test_append_skips_negative_page(ops):
    """A page index < 0 writes nothing (it must not wrap to the last page)."""
    NH, NKV, D, page = 2, 1, 16, 4
    kp = torch.zeros(4, NKV, page, D, device="cuda")
    vp = torch.zeros_like(kp)
    table = torch.full((1, 2), -1, dtype=torch.int32, device="cuda")
    qkv = rnd(1, (NH + 2 * NKV) * D, seed=11)
    pos = torch.tensor([5], dtype=torch.int32, device="cuda")
    seq = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.qk_norm_rope_append(qkv, NH, NKV, D, None, None, 0.0, None, pos, seq, table, kp, vp)
    assert kp.abs().sum() == 0 and vp.abs().sum() == 0


def _attention_case(ops, fn, dtype, NH, NKV, D, page, lens, q_lens, window, seed, spike=None):
    B = len(lens)
    n_pages = sum((l + page - 1) // page for l in lens) + 3
    kp, vp, table = _paged_setup(B, lens, NKV, D, page, dtype, n_pages, seed)
    # fill the pages of each request with random keys and values
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    for b, l in enumerate(lens):
        for j in range(l):
            pg = int(table[b, j // page])
            kp[pg, :, j % page] = torch.randn(NKV, D, device="cuda", generator=g).to(dtype)
            vp[pg, :, j % page] = torch.randn(NKV, D, device="cuda", generator=g).to(dtype)
    pos = torch.cat([torch.arange(l - q, l) for l, q in zip(lens, q_lens)]).to(torch.int32).cuda()
    seq = torch.cat([torch.full((q,), b) for b, q in enumerate(q_lens)]).to(torch.int32).cuda()
    T = pos.numel()
    q = rnd(T, (NH + 2 * NKV) * D, dtype=dtype, seed=seed + 2)
    if spike is not None:
        # make one far key dominate for the last query of request 0: a kernel that loses that
        # key (a page's edge, a tile's edge) is far off, not a little
        b, j = spike
        pg = int(table[b, j // page])
        last = sum(q_lens[:b + 1]) - 1
        for h in range(NH):
            kv = h // (NH // NKV)
            q[last, h * D:(h + 1) * D] = (kp[pg, kv, j % page].float() * 4.0).to(dtype)
    out1 = torch.zeros(T, NH * D, device="cuda", dtype=dtype)
    out2 = torch.zeros_like(out1)
    fn(q, out1, kp, vp, pos, seq, table, NH, NKV, D, D ** -0.5, window)
    ref.attention_generic(q, out2, kp, vp, pos, seq, table, NH, NKV, D, D ** -0.5, window)
    return out1, out2


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("NH,NKV,D,page,window", [(5, 1, 48, 16, 0), (6, 2, 32, 8, 0), (4, 4, 16, 4, 0), (8, 2, 128, 16, 0),
                                                 (4, 2, 64, 16, 21), (6, 3, 80, 8, 7), (2, 1, 256, 16, 0)])
def test_attention_generic(ops, dtype, NH, NKV, D, page, window):
    o1, o2 = _attention_case(ops, ops.attention_generic, dtype, NH, NKV, D, page, lens=[150, 33, 1, 64],
                             q_lens=[37, 33, 1, 2], window=window, seed=20)
    torch.testing.assert_close(o1, o2, **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
def test_attention_generic_far_key(ops, dtype):
    """One far key among hundreds carries the answer."""
    for j in (0, 15, 16, 255, 256, 300):
        o1, o2 = _attention_case(ops, ops.attention_generic, dtype, 4, 2, 64, 16, lens=[301, 40], q_lens=[1, 3],
                                 window=0, seed=30 + j, spike=(0, j))
        torch.testing.assert_close(o1, o2, **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("q_lens", [(1, 1, 1), (63,), (64,), (1, 64, 1, 1), (65, 2, 1, 33), (1, 130, 1)])
@pytest.mark.parametrize("NH,NKV,D,DV,window,keep", [(3, 3, 64, 64, 0, 0), (4, 2, 128, 64, 33, 5), (9, 3, 20, 36, 0, 0), (16, 2, 32, 256, 40, 70),
                                                    (5, 1, 136, 132, 31, 0)])
def test_attention_generic_options(ops, dtype, q_lens, NH, NKV, D, DV, window, keep):
    """Steps of one-token requests, of portions and of both, around the edges of the kernels' tiles (64 tokens, 32 keys),
    with every option, against float64; a value that no query sees is not a number and must not reach a result."""
    page, B = 8, len(q_lens)
    lens = [q + (0 if i % 3 == 1 else 37 * (i + 1)) for i, q in enumerate(q_lens)]
    n_pages = sum(-(-l // page) for l in lens) + 2
    perm = torch.randperm(n_pages, generator=torch.Generator().manual_seed(3)).tolist()
    table = torch.full((B, max(-(-l // page) for l in lens)), -1, dtype=torch.int32)
    kp, vp = rnd(n_pages, NKV, page, D, dtype=dtype, seed=50), rnd(n_pages, NKV, page, DV, dtype=dtype, seed=51)
    for b, l in enumerate(lens):
        for i in range(-(-l // page)):
            table[b, i] = perm.pop()
        if l % page:
            vp[int(table[b, l // page]), :, l % page:] = float("nan")      # behind the request's last key
    table = table.cuda()
    T = sum(q_lens)
    pos = torch.cat([torch.arange(l - q, l) for l, q in zip(lens, q_lens)]).to(torch.int32).cuda()
    seq = torch.repeat_interleave(torch.arange(B), torch.tensor(q_lens)).to(torch.int32).cuda()
    q, gate = rnd(T, NH * D + 4, dtype=dtype, seed=52)[:, :NH * D], rnd(T, NH * DV, dtype=dtype, seed=53)
    sinks, slopes = rnd(NH, seed=54), rnd(NH, seed=55).abs() * 0.1
    out = torch.full((T, NH * DV), float("nan"), device="cuda", dtype=dtype)
    ops.attention_generic(q, out, kp, vp, pos, seq, table, NH, NKV, D, D ** -0.5, window, value_dim=DV if DV != D else 0, keep_first=keep,
                          sinks=sinks, slopes=slopes, gate=gate)
    want, at = torch.empty(T, NH, DV, dtype=torch.float64, device="cuda"), 0
    for b, (l, n) in enumerate(zip(lens, q_lens)):
        j = torch.arange(l, device="cuda")
        k, v = (x[table[b, j // page].long(), :, j % page].double().repeat_interleave(NH // NKV, 1) for x in (kp, vp))
        d = pos[at:at + n, None].long() - j
        hidden = (d < 0) | ((d >= window) & (j[None] >= keep) if window else torch.zeros_like(d, dtype=torch.bool))
        s = torch.einsum("qhd,khd->hqk", q[at:at + n].double().view(n, NH, D), k) * D ** -0.5 - slopes.double()[:, None, None] * d
        s = torch.cat([s.masked_fill(hidden, -float("inf")), sinks.double()[:, None, None].expand(NH, n, 1)], -1).softmax(-1)[:, :, :-1]
        want[at:at + n] = torch.einsum("hqk,khd->qhd", s, v)
        at += n
    want = want.reshape(T, NH * DV) * torch.sigmoid(gate.double())
    torch.testing.assert_close(out.double(), want, **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("NH,NKV,D,DV,window,keep", [(4, 2, 64, 64, 0, 0), (3, 3, 20, 36, 0, 0), (9, 3, 128, 128, 0, 0), (8, 1, 136, 132, 0, 0),
                                                    (4, 2, 128, 64, 300, 45), (6, 6, 64, 64, 33, 0), (16, 2, 32, 256, 40, 70)])
def test_attention_generic_one_order_of_sums(ops, dtype, NH, NKV, D, DV, window, keep):
    """A token's result has the same bits whatever else is in the step and however its prompt was cut: as part of one
    portion, of portions of odd lengths beside other requests, as one token among a few (where several CTAs share its keys) or
    among many."""
    page, lens = 8, [1300, 70, 33, 1, 400]
    B, per = len(lens) + 80, 1304 // page
    g = torch.Generator(device="cuda").manual_seed(4)
    table = torch.randperm(len(lens) * per, device="cuda", generator=g).to(torch.int32).reshape(-1, per)
    table = torch.cat([table, table[3:4].expand(80, per)])          # 80 further requests of one key to fill a step with
    kp, vp = rnd(len(lens) * per, NKV, page, D, dtype=dtype, seed=73), rnd(len(lens) * per, NKV, page, DV, dtype=dtype, seed=74)
    sinks, slopes = rnd(NH, seed=75), rnd(NH, seed=76).abs() * 0.05
    lens += [1] * 80
    qs = {b: rnd(lens[b], NH * D, dtype=dtype, seed=80 + b) for b in range(B)}
    gates = {b: rnd(lens[b], NH * DV, dtype=dtype, seed=200 + b) for b in range(B)}

    def step(parts, singles=False):        # (request, first token, end) of each portion
        cat = lambda x: torch.cat([x[b][i:j] for b, i, j in parts])
        pos = torch.cat([torch.arange(i, j) for _, i, j in parts]).to(torch.int32).cuda()
        seq = torch.repeat_interleave(torch.tensor([b for b, _, _ in parts]), torch.tensor([j - i for _, i, j in parts])).to(torch.int32).cuda()
        out = torch.full((len(pos), NH * DV), float("nan"), device="cuda", dtype=dtype)
        ops.attention_generic(cat(qs), out, kp, vp, pos, seq, table, NH, NKV, D, D ** -0.5, window, value_dim=DV if DV != D else 0,
                              keep_first=keep, sinks=sinks, slopes=slopes, gate=cat(gates), singles=singles)
        return dict(zip(parts, out.split([j - i for _, i, j in parts])))

    few, many = [(b, 0, 1) for b in range(5, 8)], [(b, 0, 1) for b in range(5, 85)]
    whole = {b: step([(b, 0, lens[b])] + many)[(b, 0, lens[b])] for b in range(5)}
    assert not any(w.isnan().any() for w in whole.values())
    for b, cuts in ((0, [0, 1, 2, 5, 64, 131, 700, 701, 1299, 1300]), (1, [0, 1, 35, 69, 70]), (2, [0, 32, 33]), (4, [0, 3, 80, 399, 400])):
        for i, j in zip(cuts, cuts[1:]):
            for others in ([], few, many, [(3, 0, 1), ((b + 1) % 5, 0, min(66, lens[(b + 1) % 5]))]):
                got = step(others[:1] + [(b, i, j)] + others[1:])[(b, i, j)]
                assert torch.equal(got, whole[b][i:j]), (b, i, j, len(others))
            assert torch.equal(step([(b, i, j)], singles=True)[(b, i, j)], whole[b][i:j]), (b, i, j)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("q_lens,D", [((1, 1, 1), 64), ((1,) * 40, 64), ((70, 2), 64), ((70, 1, 1), 64), ((1, 70), 260)])
def test_attention_generic_scores_that_are_no_finite_numbers(ops, dtype, q_lens, D):
    """Infinities and NaN, for tokens one by one, for portions and for the general kernel (head size 260): a query or a key
    that is no number, or a score of +inf, leaves a result that is none, in its own head and request alone; keys of score
    -inf weigh nothing, be it one, a whole tile of keys or all of them (a result of zeros)."""
    page, B, NH, NKV = 16, len(q_lens), 4, 2
    lens = [100 + n for n in q_lens]
    per = -(-max(lens) // page)
    table = torch.arange(B * per, dtype=torch.int32).reshape(B, per).cuda()
    k, v = rnd(B, per * page, NKV, D, dtype=dtype, seed=70), rnd(B, per * page, NKV, D, dtype=dtype, seed=71)
    q = rnd(sum(q_lens), NH, D, dtype=dtype, seed=72)
    q[:, :, 0] = q[:, :, 0].abs() + 0.1                # a key's first element decides the sign of an infinite score
    first = [sum(q_lens[:b]) for b in range(B)]
    q[first[0], 1, 5] = float("nan")                    # one query head of one token
    k[0, 40, 1, 3] = float("nan")                       # one key of the other kv-head: every token behind it
    k[1, 0:40, 0, 0] = -float("inf")                    # a tile and more
    k[1, :, 1, 0] = -float("inf")                       # every key
    if B > 2:
        k[2, 50, 0, 0] = float("inf")
        k[2, 64:96, 1, 0] = -float("inf")
    pages = lambda x: x.reshape(B * per, page, NKV, D).transpose(1, 2).contiguous()
    pos = torch.cat([torch.arange(l - n, l) for l, n in zip(lens, q_lens)]).to(torch.int32).cuda()
    seq = torch.repeat_interleave(torch.arange(B), torch.tensor(q_lens)).to(torch.int32).cuda()
    out = torch.full((sum(q_lens), NH * D), 7.0, device="cuda", dtype=dtype)
    ops.attention_generic(q.reshape(-1, NH * D), out, pages(k), pages(v), pos, seq, table, NH, NKV, D, D ** -0.5)
    for b in range(B):
        rows = slice(first[b], first[b] + q_lens[b])
        kk, vv = (x[b].double().repeat_interleave(NH // NKV, 1) for x in (k, v))
        s = torch.einsum("qhd,khd->hqk", q[rows].double(), kk) * D ** -0.5
        s = s.masked_fill(torch.arange(per * page, device="cuda") > pos[rows, None], -float("inf"))
        want = torch.einsum("hqk,khd->qhd", s.softmax(-1), vv)
        want[(s == -float("inf")).all(-1).T] = 0.0
        torch.testing.assert_close(out[rows].double(), want.reshape(-1, NH * D), equal_nan=True, **tol(dtype))


def _attention_generic_us(ops, q_lens, NH=16, NKV=8, D=128, keys=500, page=16):
    """Microseconds of a float32 step of portions that end at `keys` keys each."""
    B, T, per = len(q_lens), sum(q_lens), -(-keys // page)
    kp, vp = rnd(B * per, NKV, page, D, seed=77), rnd(B * per, NKV, page, D, seed=78)
    table = torch.arange(B * per, device="cuda", dtype=torch.int32).reshape(B, per)
    q, out = rnd(T, NH * D, seed=79), torch.empty(T, NH * D, device="cuda")
    pos = torch.cat([torch.arange(keys - n, keys) for n in q_lens]).to(torch.int32).cuda()
    seq = torch.repeat_interleave(torch.arange(B), torch.tensor(q_lens)).to(torch.int32).cuda()
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = float("inf")
    for _ in range(6):          # (the first pass warms up; the shortest of the others)
        torch.cuda.synchronize()
        start.record()
        for _ in range(10):
            ops.attention_generic(q, out, kp, vp, pos, seq, table, NH, NKV, D, D ** -0.5)
        end.record()
        torch.cuda.synchronize()
        best = min(best, start.elapsed_time(end) * 100.0)
    return best


@pytest.mark.parametrize("q_lens,times", [([1] * 65, 2.0), ([2] * 33, 4.0), ([5] * 14, 4.0)])
def test_attention_generic_has_no_cliff_past_64_tokens(ops, q_lens, times):
    """A step a little over the size where the kernels change hands costs about what one a little under it does (65
    requests: 1.1 times the 64, four times when a CTA walked eight of them; 33 portions of two tokens 1.8 times, eleven
    times when a CTA walked sixteen of them)."""
    assert _attention_generic_us(ops, q_lens) < times * _attention_generic_us(ops, [1] * 64)


@pytest.mark.parametrize("in_dtype,out_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32),
                                                (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("M,N,K", [(1, 331, 80), (7, 100, 72), (65, 130, 200), (3, 1000, 4096), (128, 64, 16)])
def test_gemm_simt(ops, in_dtype, out_dtype, M, N, K):
    a = rnd(M, K, dtype=in_dtype, seed=40)
    w = rnd(N, K, dtype=in_dtype, scale=0.05, seed=41)
    out = ops.gemm_simt(a, w, torch.empty(M, N, device="cuda", dtype=out_dtype))
    want = (a.double() @ w.double().T)
    t = dict(rtol=1e-4, atol=1e-4) if out_dtype == torch.float32 else tol(out_dtype)
    torch.testing.assert_close(out.double(), want, **t)


def test_gemm_simt_rows_independent(ops):
    """A row's result does not depend on the other rows of the batch (bit for bit)."""
    a = rnd(37, 300, seed=42)
    w = rnd(91, 300, scale=0.05, seed=43)
    whole = ops.gemm_simt(a, w, torch.empty(37, 91, device="cuda"))
    one = ops.gemm_simt(a[5:6].contiguous(), w, torch.empty(1, 91, device="cuda"))
    assert torch.equal(whole[5:6], one)


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 32, 33, 64, 65, 129, 700])
@pytest.mark.parametrize("N,K", [(1, 1024), (129, 1029), (1030, 1100), (2500, 2080), (130, 9220)])
def test_gemm_split_one_order_of_sums(ops, M, N, K):
    """Float sums from K = 1024 on are made of bfloat16 parts: the kernel for few tokens (mma.sync) and every tile and
    sharing of K of the other (tcgen05) give a row the same bits, whatever its alignment.  Its error: a chunk of 32 k loses at most
    two cut-off additions (2^-23 of its absolute sum each), 2^-24 for the parts' products left out and for the small ones' sums;
    chunks and groups are added to nearest, no more than K / 256 + 2 chunks to a group and eight groups."""
    a = rnd(700, K, seed=46)
    w = rnd(N, K, scale=0.05, seed=47)
    one = ops.gemm_simt(a[:1], w, torch.empty(1, N, device="cuda"))
    got = ops.gemm_simt(a[:M], w, torch.full((M, N), float("nan"), device="cuda"))
    assert torch.equal(got[:1], one)
    # the same rows at strides of 16-byte pieces (which K may end within) and of none
    for pad in (-K % 4, -K % 4 + 1):
        x, y = torch.zeros(M, K + pad, device="cuda"), torch.zeros(N, K + pad, device="cuda")
        x[:, :K], y[:, :K] = a[:M], w
        assert torch.equal(ops.gemm_simt(x[:, :K], y[:, :K], torch.empty(M, N, device="cuda")), got)
    size = a[:M].double().abs() @ w.double().abs().T
    assert ((got.double() - a[:M].double() @ w.double().T).abs() <= (6 + K / 256 + 2 + 8) * 2.0 ** -24 * size).all()
    assert ops.gemm_status() == 0


@pytest.mark.parametrize("N,K", [(1500, 4100), (3600, 1029), (12000, 1100), (28500, 1024), (500, 1540)])
@pytest.mark.parametrize("odd", [0, 1])
def test_gemm_split_few_tokens_every_way(ops, N, K, odd):
    """Up to 16 tokens, whose parts come through the ring or lie in shared memory, two or three chunks side by side, in rows of
    16-byte pieces and without: the bits that seventeen have on the tiles' kernel."""
    pad = -K % 4 + odd
    x, y = torch.zeros(17, K + pad, device="cuda"), torch.zeros(N, K + pad, device="cuda")
    x[:, :K], y[:, :K] = rnd(17, K, seed=59), rnd(N, K, scale=0.05, seed=60)
    want = ops.gemm_simt(x[:, :K], y[:, :K], torch.full((17, N), float("nan"), device="cuda"))
    for M in (1, 2, 4, 5, 8, 9, 13, 16):
        assert torch.equal(ops.gemm_simt(x[:M, :K], y[:, :K], torch.full((M, N), float("nan"), device="cuda")), want[:M]), M


@pytest.mark.parametrize("M", [1, 9, 16, 17, 40, 130])
@pytest.mark.parametrize("a_size,w_size", [(1e-34, 1.0), (1.0, 1e-36), (1e-38, 1e3), (1e-42, 1.0), (1e-20, 1e-21), (1e-38, 1e30), (1e-44, 1e38), (1e14, 1e13), (1e33, 1e-30), (2e37, 1.0)])
def test_gemm_split_small_and_large_operands(ops, M, a_size, w_size):
    """Operands down to the smallest floats keep their 24 bits (their parts are scaled), and those that leave a float's range by
    the scale or as sums are made by multiply-adds.  The bound of ``test_gemm_split_one_order_of_sums`` (of plain chains of K / 8
    where those are), and half of the smallest float for a result that is one of the smallest."""
    K, N = 1030, 140
    a, w = rnd(M, K, seed=53) * a_size, rnd(N, K, scale=0.05, seed=54) * w_size
    got = ops.gemm_simt(a, w, torch.full((M, N), float("nan"), device="cuda")).double()
    size = a.double().abs() @ w.double().abs().T
    assert ((got - a.double() @ w.double().T).abs() <= (6 + K / 8 + 2 + 8) * 2.0 ** -24 * size + 2.0 ** -150).all()
    if a_size < 1e13:
        assert ((got - a.double() @ w.double().T).abs() <= (6 + K / 256 + 2 + 8) * 2.0 ** -24 * size + 2.0 ** -150).all()


@pytest.mark.parametrize("M", [16, 33, 64, 129, 700])
@pytest.mark.parametrize("N,K", [(129, 1029), (1030, 4100)])
@pytest.mark.parametrize("kind", ["spread", "cancelling", "one sign", "tiny"])
def test_gemm_split_every_row_by_itself(ops, M, N, K, kind):
    """Rows among many against the same rows one by one, bit by bit, over both octets of the kernel for few tokens and every part of
    the tiles of the other, where the units that make the sums could differ: terms of all sizes in one sum, terms that cancel,
    sums that grow throughout, values at the lower end."""
    g = torch.Generator(device="cuda").manual_seed(55)
    a, w = rnd(M, K, seed=56), rnd(N, K, scale=0.05, seed=57)
    if kind in ("spread", "tiny"):
        for t in (a, w):
            t *= 2.0 ** torch.randint(-20, 21, t.shape, device="cuda", generator=g)
    if kind == "tiny":
        a *= 2.0 ** -110
    if kind == "cancelling":            # each term and, somewhere behind it, nearly its opposite
        a[:, K // 2:2 * (K // 2)] = -a[:, :K // 2].flip(1)
        w[:, K // 2:2 * (K // 2)] = w[:, :K // 2].flip(1) * (1 + 2.0 ** -12 * rnd(N, K // 2, seed=58))
    if kind == "one sign":
        a, w = a.abs(), w.abs()
    got = ops.gemm_simt(a, w, torch.full((M, N), float("nan"), device="cuda"))
    for r in sorted({r for r in (0, 3, 7, 8, 11, 15, 16, 31, 32, 63, 64, 95, 96, 127, 128, M - 1) if r < M}):
        assert torch.equal(ops.gemm_simt(a[r:r + 1], w, torch.empty(1, N, device="cuda"))[0], got[r]), f"row {r}"
    for n in (2, 8, 9, 16, 17, 40):     # and among other numbers of rows
        if n < M:
            assert torch.equal(ops.gemm_simt(a[M - n:], w, torch.empty(n, N, device="cuda")), got[M - n:]), f"{n} rows"


@pytest.mark.parametrize("M", [3, 16, 40, 200])
def test_gemm_split_infinities_and_gate(ops, M):
    """Infinities, NaN and values near the largest have no finite parts: those outputs are what a chain of multiply-adds gives,
    the others keep their bits; the gate of the batched form."""
    K, N = 1030, 140
    a, w = rnd(M, K, seed=48), rnd(N, K, scale=0.05, seed=49)
    clean = ops.gemm_simt(a, w, torch.empty(M, N, device="cuda"))
    a[0, 5], a[1, 1029], w[7, 3], w[9, 1028], a[2, 17] = float("inf"), float("nan"), -float("inf"), float("nan"), 3.4e38
    w[:, 17] = 0.01
    got = ops.gemm_simt(a, w, torch.empty(M, N, device="cuda"))
    want = a.double() @ w.double().T
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[got.isinf()].double(), want[got.isinf()])
    torch.testing.assert_close(got[2, 10:].double(), want[2, 10:], rtol=1e-6, atol=0)
    w2, gate = rnd(2, N, K, scale=0.05, seed=50), rnd(M, 2, N, seed=51)
    x = rnd(M, 2, K, seed=52)
    out = ops.gemm_batched(x, w2, torch.empty(M, 2, N, device="cuda"), gate)
    want = torch.einsum("mbk,bnk->mbn", x.double(), w2.double()) * torch.sigmoid(gate.double())
    torch.testing.assert_close(out.double(), want, rtol=1e-5, atol=1e-5)
    assert clean.isfinite().all()


@pytest.mark.parametrize("M", [3, 16, 40, 500])
def test_gemm_split_gate_beside_infinities(ops, M):
    """The batched form's gate on results that leave with it and on those that are made again: infinities, a NaN, a sum out of the
    scale's range, a gate that closes and one that is none."""
    K, N = 1030, 140
    w, gate, x = rnd(2, N, K, scale=0.05, seed=61), rnd(M, 2, N, seed=62), rnd(M, 2, K, seed=63)
    x[0, 0, 5], x[1, 1, 1029], w[1, 7, 3], x[2, 0, 17] = float("inf"), float("nan"), -float("inf"), 3e30
    gate[0, 0, 3], gate[2, 0, 9], gate[2, 1, 11] = -float("inf"), float("inf"), float("nan")
    out = ops.gemm_batched(x, w, torch.full((M, 2, N), 7.0, device="cuda"), gate)
    want = torch.einsum("mbk,bnk->mbn", x.double(), w.double()) / (1 + torch.exp(-gate.double()))
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isinf(), want.isinf())
    ok = want.isfinite()
    torch.testing.assert_close(out[ok].double(), want[ok], rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("M", [1, 2, 4, 5, 8, 9, 16, 17, 33, 65, 129, 700])
@pytest.mark.parametrize("N,K", [(1, 4), (65, 33), (129, 256), (200, 2052), (1030, 260)])
def test_gemm_simt_one_order_of_sums(ops, M, N, K):
    """Every tile and every split of K (they follow M, N and K), and the form for rows that are no 16-byte pieces, give a
    row the same bits; its error is that of eight chains of K/8 (each at most K/8 roundings of its partial sums)."""
    a = rnd(700, K, seed=44)
    w = rnd(N, K, scale=0.05, seed=45)
    one = ops.gemm_simt(a[:1], w, torch.empty(1, N, device="cuda"))
    got = ops.gemm_simt(a[:M], w, torch.full((M, N), float("nan"), device="cuda"))
    wide = torch.zeros(M, K + 1, device="cuda")        # the same rows at a stride of no 16-byte pieces
    wide[:, :K] = a[:M]
    assert torch.equal(got[:1], one)
    assert torch.equal(ops.gemm_simt(wide[:, :K], w, torch.empty(M, N, device="cuda")), got)
    bound = (K / 8 + 4) * 2.0 ** -24 * (a[:M].double().abs() @ w.double().abs().T)
    assert ((got.double() - a[:M].double() @ w.double().T).abs() <= bound + 1e-30).all()


@pytest.mark.parametrize("R,V", [(1, 331), (5, 151936), (3, 1000), (64, 4097)])
def test_argmax(ops, R, V):
    lg = rnd(R, V, seed=50)
    lg[0, V - 1] = lg[0, 3] = 50.0   # equal maxima: the lowest index wins
    out = ops.argmax(lg, torch.empty(R, device="cuda", dtype=torch.int32))
    assert out.tolist() == lg.argmax(-1).tolist()
    assert out[0].item() == 3


# ----------------------------------------------------------------------------- tensor-core attention (bfloat16)
class _Ctx:
    pass


def _tc_case(ops, NH, NKV, D, page, lens, q_lens, window, seed, n_splits=None, spike=None, k_growth=0.0):
    """A mixed batch through ops.attention (decode kernel for one-token requests, tile kernel for portions)."""
    dtype = torch.bfloat16
    B = len(lens)
    n_pages = sum((l + page - 1) // page for l in lens) + 3
    kp, vp, table = _paged_setup(B, lens, NKV, D, page, dtype, n_pages, seed)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    for b, l in enumerate(lens):
        for j in range(l):
            pg = int(table[b, j // page])
            kp[pg, :, j % page] = (torch.randn(NKV, D, device="cuda", generator=g) * (1.0 + k_growth * j)).to(dtype)
            vp[pg, :, j % page] = torch.randn(NKV, D, device="cuda", generator=g).to(dtype)
    ctx = _Ctx()
    ctx.positions = torch.cat([torch.arange(l - q, l) for l, q in zip(lens, q_lens)]).to(torch.int32).cuda()
    ctx.seq_of_token = torch.cat([torch.full((q,), b) for b, q in enumerate(q_lens)]).to(torch.int32).cuda()
    cu = [0]
    for q in q_lens:
        cu.append(cu[-1] + q)
    ctx.cu_q = torch.tensor(cu, dtype=torch.int32).cuda()
    ctx.kv_len = torch.tensor(lens, dtype=torch.int32).cuda()
    dec = [b for b, q in enumerate(q_lens) if q == 1]
    tiles = [(b, s) for b, q in enumerate(q_lens) if q > 1 for s in range(0, q, QUERY_TILE)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32).cuda()
    ctx.work = {"dec_tokens": i32([cu[b] for b in dec]), "dec_seqs": i32(dec), "n_dec": len(dec),
                "tile_seq": i32([t[0] for t in tiles]), "tile_q0": i32([t[1] for t in tiles]), "n_tiles": len(tiles),
                "max_dec_kv": max([lens[b] for b in dec], default=0), "n_splits": n_splits}
    T = cu[-1]
    q = rnd(T, (NH + 2 * NKV) * D, dtype=dtype, seed=seed + 2)
    if spike is not None:
        b, j = spike
        pg = int(table[b, j // page])
        last = cu[b + 1] - 1
        for h in range(NH):
            q[last, h * D:(h + 1) * D] = (kp[pg, h // (NH // NKV), j % page].float() * 3.0).to(dtype)
    out1 = torch.full((T, NH * D), 7.0, device="cuda", dtype=dtype)
    out2 = torch.zeros_like(out1)
    assert ops.tensor_core_attention_takes(dtype, NH, NKV, D)
    ops.attention(q, out1, kp, vp, ctx, table, NH, NKV, D, D ** -0.5, window)
    ref.attention_generic(q, out2, kp, vp, ctx.positions, ctx.seq_of_token, table, NH, NKV, D, D ** -0.5, window)
    return out1, out2


@pytest.mark.parametrize("NH,NKV,D,page", [(8, 2, 128, 16), (6, 2, 64, 8), (5, 1, 64, 16), (16, 1, 128, 32), (4, 4, 128, 4),
                                          (3, 3, 64, 16)])
@pytest.mark.parametrize("n_splits", [1, 2, 5, 8, None])
def test_attention_decode_kernel(ops, NH, NKV, D, page, n_splits):
    o1, o2 = _tc_case(ops, NH, NKV, D, page, lens=[1, 77, 300, 64, 65, 513], q_lens=[1] * 6, window=0, seed=60,
                      n_splits=n_splits)
    torch.testing.assert_close(o1, o2, **tol(torch.bfloat16))


@pytest.mark.parametrize("NH,NKV,D,page", [(8, 2, 128, 16), (6, 2, 64, 8), (5, 1, 64, 16), (4, 4, 128, 4)])
def test_attention_chunk_kernel(ops, NH, NKV, D, page):
    # whole prompts, portions after a cached prefix, a portion of two tokens, tiles that end mid-way
    o1, o2 = _tc_case(ops, NH, NKV, D, page, lens=[150, 33, 200, 64, 130, 2], q_lens=[150, 2, 71, 64, 65, 2], window=0,
                      seed=61)
    torch.testing.assert_close(o1, o2, **tol(torch.bfloat16))


@pytest.mark.parametrize("D,spread", [(128, 0.0), (128, 1.0), (128, 40.0), (128, 4000.0), (64, 40.0)])
def test_prompt_attention_exponentials_of_every_size(ops, D, spread):
    """Scores that are all equal, that differ by a few units and that differ by thousands (exponentials of which almost all
    vanish, far below where the smallest float lies), each column of a tile by whichever unit takes its exponential."""
    NH, NKV, page, n = 2, 1, 64, 256
    kp, vp = torch.zeros(4, NKV, page, D, device="cuda", dtype=torch.bfloat16), rnd(4, NKV, page, D, dtype=torch.bfloat16, seed=56)
    kp[..., 0] = rnd(4, NKV, page, dtype=torch.bfloat16, seed=57)
    q = torch.zeros(n, (NH + 2 * NKV) * D, device="cuda", dtype=torch.bfloat16)
    q[:, 0:NH * D:D] = spread
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    call = lambda q: ops.attention_tc(q, torch.full((n, NH * D), 7.0, device="cuda", dtype=torch.bfloat16), kp, vp, i32([0, 0]), i32([128, 0]), 2,
                                      i32([0, n]), i32([n]), i32([[0, 1, 2, 3]]), NH, NKV, D, 1.0, 0)
    got = call(q)
    s = spread * kp[:, 0, :, 0].reshape(1, n).double() + torch.full((n, n), -float("inf"), device="cuda", dtype=torch.float64).triu(1)
    want = (s.softmax(-1) @ vp[:, 0].reshape(n, D).double()).repeat(1, NH)
    torch.testing.assert_close(got.double(), want, **tol(torch.bfloat16))
    q[70, :D] = float("nan")            # a query that is no number stays none, and alone
    bad = call(q).isnan()
    assert bad[70, :D].all() and int(bad.sum()) == D


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("window", [0, 20])
def test_prompt_attention_gives_no_weight_to_keys_that_are_not_seen(ops, D, window):
    """Values of 1e38 at tokens behind a query, or in front of its window, in the same tile: a weight of the smallest float
    instead of 0 would show."""
    NH, NKV, page, n = 2, 1, 64, 256
    kp, vp = rnd(4, NKV, page, D, dtype=torch.bfloat16, seed=65), rnd(4, NKV, page, D, dtype=torch.bfloat16, seed=66)
    q = rnd(n, (NH + 2 * NKV) * D, dtype=torch.bfloat16, seed=67)
    vp[1, :, 36:] = 1e38            # tokens 100 to 127
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    out = torch.full((n, NH * D), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.attention_tc(q, out, kp, vp, i32([0, 0]), i32([128, 0]), 2, i32([0, n]), i32([n]), i32([[0, 1, 2, 3]]), NH, NKV, D, D ** -0.5, window)
    d = torch.arange(n, device="cuda")[:, None] - torch.arange(n, device="cuda")
    s = torch.einsum("qhd,kd->hqk", q[:, :NH * D].double().view(n, NH, D), kp[:, 0].reshape(n, D).double()) * D ** -0.5
    s = s.masked_fill((d < 0) | ((d >= window) if window else torch.zeros_like(d, dtype=torch.bool)), -float("inf"))
    want = torch.einsum("hqk,kd->qhd", s.softmax(-1), vp[:, 0].reshape(n, D).double()).reshape(n, NH * D)
    rows = (torch.arange(n) < 100) | ((torch.arange(n) >= 127 + window) if window else torch.zeros(n, dtype=torch.bool))
    torch.testing.assert_close(out[rows].double(), want[rows], **tol(torch.bfloat16))


@pytest.mark.parametrize("window", [1, 7, 64, 100])
def test_tensor_core_attention_window_and_mixed_batch(ops, window):
    o1, o2 = _tc_case(ops, 8, 2, 128, 16, lens=[150, 90, 300, 17, 64], q_lens=[150, 1, 70, 1, 2], window=window, seed=62)
    torch.testing.assert_close(o1, o2, **tol(torch.bfloat16))


def test_tensor_core_attention_far_key(ops):
    """One far key among hundreds carries the answer: at a page's edge, a tile's edge, a split's edge."""
    for j in (0, 15, 16, 63, 64, 127, 128, 447, 448, 600):
        for q_lens in ([1, 1], [5, 3]):
            o1, o2 = _tc_case(ops, 4, 2, 128, 16, lens=[601, 40], q_lens=q_lens, window=0, seed=70 + j, spike=(0, j))
            torch.testing.assert_close(o1, o2, **tol(torch.bfloat16))


def test_decode_kernel_twice_leaves_its_counters_clean(ops):
    """The split counters go back to zero, so a second call with other shapes is right too."""
    for seed, lens in ((80, [500, 300]), (81, [129, 700, 90])):
        o1, o2 = _tc_case(ops, 8, 2, 128, 16, lens=lens, q_lens=[1] * len(lens), window=0, seed=seed, n_splits=4)
        torch.testing.assert_close(o1, o2, **tol(torch.bfloat16))


def _decode_direct(ops, NH, NKV, D, page, lens, n_splits, cluster_merge, seed, spike=None):
    """The split-KV kernel called by itself (every page filled at random), against the float32 reference."""
    dtype = torch.bfloat16
    B = len(lens)
    n_pages = sum((l + page - 1) // page for l in lens) + 3
    kp, vp, table = _paged_setup(B, lens, NKV, D, page, dtype, n_pages, seed)
    kp.copy_(rnd(*kp.shape, dtype=dtype, seed=seed + 1))
    vp.copy_(rnd(*vp.shape, dtype=dtype, seed=seed + 2))
    q = rnd(B, (NH + 2 * NKV) * D, dtype=dtype, seed=seed + 3)
    if spike is not None:
        b, j = spike
        pg = int(table[b, j // page])
        for h in range(NH):
            q[b, h * D:(h + 1) * D] = (kp[pg, h // (NH // NKV), j % page].float() * 3.0).to(dtype)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32).cuda()
    kv_len, ar = i32(lens), i32(list(range(B)))
    out1 = torch.full((B, NH * D), 7.0, device="cuda", dtype=dtype)
    out2 = torch.zeros_like(out1)
    splits = n_splits or ops.decode_plan(B, NH, NKV, D, page, max(lens))[0]
    ops.attention_decode(q, out1, kp, vp, ar, ar, B, kv_len, table, NH, NKV, D, D ** -0.5, 0, splits, max(lens),
                         cluster_merge=cluster_merge)
    ref.attention_generic(q, out2, kp, vp, i32([l - 1 for l in lens]), ar, table, NH, NKV, D, D ** -0.5, 0)
    return out1, out2, splits


@pytest.mark.parametrize("n_splits", [3, 9, 16])
def test_decode_attention_merge_through_scratch_memory(ops, n_splits):
    """Partial results in scratch memory and the merge by the CTA that arrives last (what more than 8 splits, i.e.
    long contexts, use; up to 8 splits ordinarily merge inside a cluster): twice in a row with different shapes,
    so that a counter that did not return to zero or a partial result left over from the first call would show."""
    for seed, NH, NKV, D, page, lens in ((82, 8, 2, 128, 16, [700, 300, 1, 2100]), (83, 6, 2, 64, 8, [129, 1500, 90]),
                                         (84, 8, 2, 128, 16, [640, 33])):
        o1, o2, _ = _decode_direct(ops, NH, NKV, D, page, lens, n_splits, cluster_merge=False, seed=seed)
        torch.testing.assert_close(o1, o2, **tol(torch.bfloat16))


@pytest.mark.parametrize("n_splits", [2, 6, 8])
def test_decode_attention_merge_inside_clusters(ops, n_splits):
    """The splits of a request are the CTAs of a cluster: rank 0 keeps its own partial result, the others write theirs
    where rank 0's queries lay.  One far key carries the answer of request 0, in rank 0's part, at the edges of the
    parts and in the last one; 4 and 16 query heads to a kv-head (the partial results are smaller and larger than the
    queries' buffer)."""
    for NH, NKV in ((8, 2), (16, 1)):
        lens = [3000, 517, 40]
        per = -(-max(lens) // n_splits)
        for j in (0, 7, per - 1, per, 2999):
            o1, o2, _ = _decode_direct(ops, NH, NKV, 128, 16, lens, n_splits, cluster_merge=True, seed=90 + j % 5, spike=(0, j))
            torch.testing.assert_close(o1, o2, **tol(torch.bfloat16))


def test_decode_attention_long_context_chooses_many_splits(ops):
    """About 60 000 keys: the split count that serving computes is above 8, the merge goes through scratch memory
    and block-table entries beyond the part cached in shared memory are read; one far key at a split's edge carries
    the answer for request 0."""
    lens = [60000, 517]
    n, in_clusters = ops.decode_plan(len(lens), 8, 2, 128, 16, max(lens))
    assert n > 8 and not in_clusters
    per = -(-max(lens) // n)
    for j in (per - 1, per, 5 * per, 59999, 0):
        o1, o2, splits = _decode_direct(ops, 8, 2, 128, 16, lens, None, cluster_merge=True, seed=85 + j % 7, spike=(0, j))
        assert splits == n
        torch.testing.assert_close(o1, o2, **tol(torch.bfloat16))


# ----------------------------------------------------------------------------- tcgen05 matrix product
GEMM_SHAPES = [
    # (M, N, K): decode-like (swapped roles) and prefill-like, with edges that fill no tile
    (1, 256, 128), (8, 6144, 4096), (5, 331, 72), (16, 128, 64), (17, 200, 264), (64, 1000, 512), (100, 384, 200),
    (128, 256, 4096), (129, 256, 128), (300, 520, 136), (2048, 512, 1024), (515, 4096, 256),
]


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_tc(ops, M, N, K, out_dtype):
    x = rnd(M, K, dtype=torch.bfloat16, seed=90)
    w = rnd(N, K, dtype=torch.bfloat16, scale=0.05, seed=91)
    out = torch.full((M, N), 3.0, device="cuda", dtype=out_dtype)
    ops.gemm_tc(x, w, out)
    want = x.double() @ w.double().T
    assert ops.gemm_status() == 0
    t = dict(rtol=1e-4, atol=1e-4) if out_dtype == torch.float32 else tol(torch.bfloat16)
    torch.testing.assert_close(out.double(), want, **t)


@pytest.mark.parametrize("M,K", [(8, 512), (1, 4096), (300, 256)])
def test_gemm_tc_at_the_real_vocabulary(ops, M, K):
    """The output head of the real models: 151 936 rows of weights, float32 logits (1187 tiles of 128 rows)."""
    N = 151936
    x = rnd(M, K, dtype=torch.bfloat16, seed=98)
    w = rnd(N, K, dtype=torch.bfloat16, scale=0.05, seed=99)
    out = torch.full((M, N), 3.0, device="cuda", dtype=torch.float32)
    ops.gemm_tc(x, w, out, static_weights=True)
    assert ops.gemm_status() == 0
    for n0 in range(0, N, 32768):        # the reference in pieces: a double copy of the whole weight is not needed
        want = x.double() @ w[n0:n0 + 32768].double().T
        torch.testing.assert_close(out[:, n0:n0 + 32768].double(), want, rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("plan", [(1, 16, 1), (1, 16, 4), (1, 32, 3), (1, 64, 2), (1, 128, 5), (0, 64, 1), (0, 128, 2),
                                  (0, 256, 1), (0, 256, 3), (0, 160, 1), (0, 192, 1), (0, 224, 1), (0, 160, 2),
                                  (0, 256, 1, 6, 4), (0, 256, 1, 2, 4)])          # the last two: pairs of CTAs on 256 x 256
def test_gemm_tc_every_tile_shape_and_split(ops, plan):
    M, N, K = (50 if plan[0] else 300), 700, 1160
    if plan[0] and M > plan[1]:
        M = plan[1] - 3
    x = rnd(M, K, dtype=torch.bfloat16, seed=92)
    w = rnd(N, K, dtype=torch.bfloat16, scale=0.05, seed=93)
    for out_dtype in (torch.float32, torch.bfloat16):
        out = torch.zeros(M, N, device="cuda", dtype=out_dtype)
        ops.gemm_tc(x, w, out, plan)
        assert ops.gemm_status() == 0
        t = dict(rtol=1e-4, atol=1e-4) if out_dtype == torch.float32 else tol(torch.bfloat16)
        torch.testing.assert_close(out.double(), x.double() @ w.double().T, **t)


@pytest.mark.parametrize("M,N,K", [
    # one shape for every way that the plans split and share a product: few tokens with 7, 6, 5, 4, 3 and 2 splits and with two or
    # three CTAs an SM, 65 to 128 tokens in tiles of 64 and 128 or on the rows, more tokens with two CTAs to a tile
    (3, 1024, 3072), (9, 2560, 4096), (20, 2048, 3072), (30, 2560, 3072), (25, 3072, 8192), (33, 1024, 3072), (64, 2560, 9728), (40, 5120, 8192),
    (50, 6144, 1024), (60, 12288, 1088), (12, 12288, 1088), (20, 12288, 1088), (5, 16384, 1088), (16, 34816, 512), (7, 41472, 256), (65, 1024, 1032),
    (100, 2560, 2048), (128, 4096, 1024), (128, 7168, 1088), (80, 12288, 1024), (70, 19456, 640), (127, 24576, 512), (66, 256, 512),
    (129, 4096, 3072), (200, 2560, 4104), (300, 2056, 3080), (257, 5120, 8192), (300, 4096, 8200), (512, 24576, 512)])
@pytest.mark.parametrize("form", ["float", "bias", "unary", "swiglu"])
def test_gemm_tc_as_planned(ops, M, N, K, form):
    """Every epilogue behind every plan, with rows and a K that fill no tile; rows that lie further apart than they are long."""
    x = rnd(M, K + 8, dtype=torch.bfloat16, seed=58)[:, :K]
    w = rnd(N, K, dtype=torch.bfloat16, scale=0.05, seed=59)
    bias = rnd(N, seed=60)
    want = x.double() @ w.double().T
    if form == "float":
        out = ops.gemm_tc(x, w, torch.full((M, N), 7.0, device="cuda"))
        torch.testing.assert_close(out.double(), want, rtol=1e-4, atol=1e-3)
    elif form == "swiglu":
        out = ops.gemm_tc(x, w, torch.full((M, N // 2), 7.0, device="cuda", dtype=torch.bfloat16), swiglu_pairs=True, bias=bias)
        want = (want + bias.double()).bfloat16().double()
        gate = want[:, ::2]
        torch.testing.assert_close(out.double(), (gate * torch.sigmoid(gate)).bfloat16().double() * want[:, 1::2], rtol=2.4e-2, atol=2.4e-2)
    else:
        out = ops.gemm_tc(x, w, torch.full((M, N), 7.0, device="cuda", dtype=torch.bfloat16), bias=bias, unary="silu" if form == "unary" else None)
        want = want + bias.double()
        torch.testing.assert_close(out.double(), want * torch.sigmoid(want) if form == "unary" else want, **tol(torch.bfloat16))
    assert ops.gemm_status() == 0


def test_a_split_product_of_many_tokens_inside_a_capture(ops):
    """The router's plan for long steps, in a graph that nothing of its size ran before, twice in a row: the first product's
    counters and partial sums are not the second's."""
    x, w = rnd(8200, 2048, dtype=torch.bfloat16, seed=63), rnd(64, 2048, dtype=torch.bfloat16, scale=0.05, seed=64)
    one, two = (torch.full((8200, 64), 7.0, device="cuda") for _ in range(2))
    ops.gemm_tc(x[:4], w, one[:4])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.gemm_tc(x, w, one, plan=(0, 128, 8, 4, 0))
        ops.gemm_tc(x[:600], w, two[:600], plan=(0, 128, 8, 4, 0))
    for _ in range(3):
        one.fill_(7.0)
        two.fill_(7.0)
        graph.replay()
        want = x.double() @ w.double().T
        torch.testing.assert_close(one.double(), want, rtol=1e-4, atol=1e-3)
        torch.testing.assert_close(two[:600].double(), want[:600], rtol=1e-4, atol=1e-3)
    assert ops.gemm_status() == 0


@pytest.mark.parametrize("M,N,K", [(129, 3072, 4096), (200, 512, 4096), (256, 4608, 8192)])
def test_clamped_unit_keeps_its_tokens_on_the_rows(ops, M, N, K):
    """The product with the clamped gated unit has no form for shared tiles: sizes for which a plain product takes one."""
    assert ops.gemm_tc_plan(M, N, K, 148)[:3] != ops.gemm_tc_plan(M, N, K, 148, rows=True)[:3]
    x, w = rnd(M, K, dtype=torch.bfloat16, seed=61), rnd(N, K, dtype=torch.bfloat16, scale=0.02, seed=62)
    out = ops.linear_bf16_glu(x, w, torch.empty(M, N // 2, device="cuda", dtype=torch.bfloat16), 2.0, 1.7)
    z = x.double() @ w.double().T
    g, u = z[:, ::2].clamp(max=2.0), z[:, 1::2].clamp(-2.0, 2.0)
    torch.testing.assert_close(out.double(), g * torch.sigmoid(1.7 * g) * (u + 1), **tol(torch.bfloat16))


@pytest.mark.parametrize("M,plan", [(8, None), (8, (1, 16, 4, 4, 0)), (300, None), (300, (0, 256, 1, 4, 4))])
def test_gemm_tc_wait_that_runs_out_leaves_its_code_and_returns(ops, M, plan):
    """A bounded wait made to run out, without a fault: the product is told to poll each barrier a few thousand
    times at most and never to load one k-block.  It has to give up, free what it holds and return, with the
    wait's code in the status word; after the counters are cleared the next launch of the same shape is right.
    M = 8: swapped roles, the splits of K as a cluster / through the work space; M = 300: tokens on the rows, a CTA
    or a pair of CTAs to a tile (in a pair both CTAs' waits run out, each by itself)."""
    N, K = 512, 4096
    x = rnd(M, K, dtype=torch.bfloat16, seed=190)
    w = rnd(N, K, dtype=torch.bfloat16, scale=0.05, seed=191)
    want = x.double() @ w.double().T
    assert ops.gemm_status() == 0
    ops.gemm_tc_test_fault(1 << 12, 5)
    ops.gemm_tc(x, w, torch.zeros(M, N, device="cuda", dtype=torch.float32), plan)
    torch.cuda.synchronize()                 # returns: the kernel ended by itself
    assert ops.gemm_status() in (1, 2, 3, 4)
    ops.reset_after_failure()
    assert ops.gemm_status() == 0
    for _ in range(2):
        out = torch.zeros(M, N, device="cuda", dtype=torch.float32)
        ops.gemm_tc(x, w, out, plan)
        torch.testing.assert_close(out.double(), want, rtol=1e-4, atol=1e-4)
    assert ops.gemm_status() == 0


def test_gemm_tc_strided_rows_and_repeat(ops):
    """x as a column slice of a wider matrix (row stride > K), twice in a row (split counters return to zero)."""
    big = rnd(40, 1024, dtype=torch.bfloat16, seed=94)
    x = big[:, 256:768]
    w = rnd(384, 512, dtype=torch.bfloat16, scale=0.05, seed=95)
    for _ in range(2):
        out = torch.zeros(40, 384, device="cuda", dtype=torch.float32)
        ops.gemm_tc(x, w, out, (1, 64, 4))
        torch.testing.assert_close(out.double(), x.double() @ w.double().T, rtol=1e-4, atol=1e-4)
    assert ops.gemm_status() == 0


def test_gemm_tc_rows_do_not_depend_on_the_batch(ops):
    """The same token gives the same output row alone and among others (same tile shape and split)."""
    x = rnd(16, 512, dtype=torch.bfloat16, seed=96)
    w = rnd(640, 512, dtype=torch.bfloat16, scale=0.05, seed=97)
    whole = ops.gemm_tc(x, w, torch.zeros(16, 640, device="cuda", dtype=torch.float32), (1, 16, 2))
    one = ops.gemm_tc(x[3:4], w, torch.zeros(1, 640, device="cuda", dtype=torch.float32), (1, 16, 2))
    assert torch.equal(whole[3:4], one)


@pytest.mark.parametrize("plan", [None, (1, 16, 1), (1, 16, 3), (1, 64, 2), (0, 256, 1), (0, 128, 2), (0, 64, 1), (0, 256, 1, 6, 4)])
@pytest.mark.parametrize("M,I,K", [(8, 352, 512), (40, 1000, 264), (300, 520, 1160)])
def test_gemm_tc_fused_swiglu(ops, plan, M, I, K):
    """The paired epilogue equals the stacked product followed by the SwiGLU kernel, bit for bit."""
    if plan is not None and plan[0] == 1 and M > plan[1]:
        pytest.skip("more tokens than the tile's narrow side")
    x = rnd(M, K, dtype=torch.bfloat16, seed=98)
    wg = rnd(I, K, dtype=torch.bfloat16, scale=0.05, seed=99)
    wu = rnd(I, K, dtype=torch.bfloat16, scale=0.05, seed=100)
    pairs = torch.stack([wg, wu], dim=1).reshape(2 * I, K).contiguous()
    got = ops.gemm_tc(x, pairs, torch.zeros(M, I, device="cuda", dtype=torch.bfloat16), plan, swiglu_pairs=True)
    gu = ops.gemm_tc(x, torch.cat([wg, wu]).contiguous(), torch.zeros(M, 2 * I, device="cuda", dtype=torch.bfloat16), plan)
    want = ops.swiglu(gu, torch.zeros(M, I, device="cuda", dtype=torch.bfloat16))
    assert ops.gemm_status() == 0
    assert torch.equal(got, want)
    torch.testing.assert_close(got, ref.swiglu((x.float() @ torch.cat([wg, wu]).float().T).bfloat16(),
                                               torch.zeros(M, I, device="cuda", dtype=torch.bfloat16)), **tol(torch.bfloat16))


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("N,K", [(16, 64), (48, 192), (4096, 1024), (80, 4160), (96, 4096), (19456, 640), (6144, 2560), (66000, 512)])
def test_gemm_rows(ops, monkeypatch, M, N, K):
    """Products of up to 32 tokens with weights written long before: sixteen or 32 rows to a block, one round of blocks and
    several, K that leaves warps without a chunk and K that their rings go round in; plain in both types, and (gate, up) pairs.
    The kernel takes all of these sizes, also those at which the tiled one is faster and the rule sends them there."""
    assert not ops.gemm_rows_pays(33, N, K, 148)
    monkeypatch.setattr(ops, "gemm_rows_pays", lambda M, N, K, sms: M <= 32)
    wide = rnd(M, K + 64, dtype=torch.bfloat16, seed=260)
    x = wide[:, 64:]
    w = rnd(N, K, dtype=torch.bfloat16, scale=0.05, seed=261)
    want = x.double() @ w.double().T
    out = ops.gemm_tc(x, w, torch.full((M, N), 3.0, device="cuda"), static_weights=True)
    torch.testing.assert_close(out.double(), want, rtol=1e-4, atol=1e-4)
    # (more than a rounding to bfloat16 apart only where a float sum lies at a boundary: one unit in the last place)
    out = ops.gemm_tc(x, w, torch.full((M, N), 3.0, device="cuda", dtype=torch.bfloat16), static_weights=True)
    torch.testing.assert_close(out.double(), want, rtol=2.0 ** -8, atol=1e-4)
    got = ops.gemm_tc(x, w, torch.full((M, N // 2), 3.0, device="cuda", dtype=torch.bfloat16), swiglu_pairs=True, static_weights=True)
    gate, up = out.double()[:, 0::2], out.double()[:, 1::2]
    torch.testing.assert_close(got.double(), gate * torch.sigmoid(gate) * up, rtol=2.0 ** -6, atol=1e-4)


@pytest.mark.parametrize("NH,NKV,D,T,K", [(16, 8, 128, 8, 1024), (32, 8, 128, 5, 640), (4, 4, 128, 1, 512), (6, 2, 64, 16, 128), (5, 1, 64, 9, 2112), (3, 1, 128, 13, 192)])
@pytest.mark.parametrize("normed,rotated", [(True, True), (False, True), (True, False)])
def test_gemm_rows_qkv(ops, NH, NKV, D, T, K, normed, rotated):
    """The projection of few tokens whose blocks share a head's norm through their cluster, against the product followed by
    the rotation kernel (sums in another order: a rounding may move here and there)."""
    page, per_request, N = 16, 10, (NH + 2 * NKV) * D
    x = rnd(T, K, dtype=torch.bfloat16, seed=262)
    w = rnd(N, K, dtype=torch.bfloat16, scale=0.05, seed=263)
    qw = (1.0 + 0.1 * rnd(D, seed=264)) if normed else None
    kw = (1.0 + 0.1 * rnd(D, seed=265)) if normed else None
    ang = torch.rand(200, D // 2, device="cuda") * 6.28
    cos_sin = torch.cat([ang.cos(), ang.sin()], dim=1).contiguous() if rotated else None
    seq = torch.tensor([i % 3 for i in range(T)], dtype=torch.int32, device="cuda")
    pos = torch.tensor([(7 * i + 3) % 150 for i in range(T)], dtype=torch.int32, device="cuda")
    table = torch.randperm(32, device="cuda").to(torch.int32)[:3 * per_request].view(3, per_request).contiguous()
    if T > 2:
        table[int(seq[2]), int(pos[2]) // page] = -1
    kp1 = torch.zeros(32, NKV, page, D, device="cuda", dtype=torch.bfloat16)
    vp1, kp2, vp2 = torch.zeros_like(kp1), torch.zeros_like(kp1), torch.zeros_like(kp1)
    assert ops.gemm_rows_pays(T, N, K, 148)
    want = ops.gemm_tc(x, w, torch.zeros(T, N, device="cuda", dtype=torch.bfloat16), static_weights=True)
    ops.qk_norm_rope_append(want, NH, NKV, D, qw, kw, 1e-6, cos_sin, pos, seq, table, kp1, vp1)
    got = torch.zeros(T, N, device="cuda", dtype=torch.bfloat16)
    ops.gemm_tc_qkv(x, w, got, NH, NKV, D, qw, kw, 1e-6, cos_sin, pos, seq, table, kp2, vp2, static_weights=True)
    for a, b in ((got[:, :NH * D], want[:, :NH * D]), (kp2, kp1), (vp2, vp1)):
        torch.testing.assert_close(a, b, **tol(torch.bfloat16))
        assert (a != b).float().mean() < 0.02
    assert not got[:, NH * D:].any()


@pytest.mark.parametrize("M,N,K", [(2100, 2304, 200), (5000, 520, 136), (257, 256, 64), (256, 4104, 72), (9000, 264, 4096)])
def test_gemm_tc_pairs_of_ctas(ops, M, N, K):
    """Tiles of 256 x 256 on pairs of CTAs (tcgen05 cta_group::2): more tiles than pairs (a pair walks several, the
    accumulator buffers alternate), groups of tile rows of which the last is short, edges that fill no tile, one
    k-block and many; and the plan picks this form by itself for a prompt's shapes."""
    x = rnd(M, K, dtype=torch.bfloat16, seed=196)
    w = rnd(N, K, dtype=torch.bfloat16, scale=0.05, seed=197)
    want = x.double() @ w.double().T
    for out_dtype in (torch.float32, torch.bfloat16):
        out = torch.full((M, N), 3.0, device="cuda", dtype=out_dtype)
        ops.gemm_tc(x, w, out, (0, 256, 1, 6, ops.GEMM_PAIR), static_weights=out_dtype == torch.bfloat16)
        assert ops.gemm_status() == 0
        t = dict(rtol=1e-4, atol=1e-4) if out_dtype == torch.float32 else tol(torch.bfloat16)
        torch.testing.assert_close(out.double(), want, **t)
    assert ops.gemm_tc_plan(2048, 4096, 4096, 148)[4:] == (ops.GEMM_PAIR,)
    assert len(ops.gemm_tc_plan(1056, 34816, 5120, 148)) == 4       # 1280 rows of pair tiles for 1056 tokens: not worth it


def test_tensor_core_attention_growing_scores(ops):
    """Keys whose scores grow along a long prompt: the running maximum moves in every tile of keys, far enough
    that the rows of O are rescaled again and again (and by different amounts in the rows of one warp)."""
    for q_lens, lens in (([700, 130], [700, 400]), ([257, 2], [900, 514])):
        o1, o2 = _tc_case(ops, 6, 2, 128, 16, lens=lens, q_lens=q_lens, window=0, seed=91, k_growth=1.0 / 20.0)
        torch.testing.assert_close(o1, o2, **tol(torch.bfloat16))


@pytest.mark.parametrize("parts", [(2, 0), (3, 0), (8, 0), (1, 2), (2, 3)])
@pytest.mark.parametrize("NH,NKV,D,window,keep,extra", [(10, 2, 128, 0, 0, ""), (4, 2, 64, 0, 0, "sinks"), (6, 2, 128, 300, 0, "gate"), (3, 3, 64, 200, 70, "float"), (10, 2, 64, 0, 0, "slopes")])
def test_tensor_core_attention_with_keys_shared_out(ops, parts, NH, NKV, D, window, keep, extra):
    """A tile's key tiles over a cluster's blocks (more blocks than key tiles among them, pairs of heads and heads without a
    partner, the odd heads by a launch of their own) against one block: the same softmax with its weights taken relative to
    another maximum, so a weight's rounding to bfloat16 may fall differently."""
    if parts[1] and (NH // NKV % 2 == 0 or NH // NKV < 3):
        pytest.skip("no odd heads beside pairs")
    import numpy as np
    q_lens, lens, page = [300, 2, 129, 40], [1100, 2, 129, 900], 16
    cu = np.concatenate([[0], np.cumsum(q_lens)]).astype(np.int32)
    arrays, values = ops.attention_work(q_lens, lens, cu)
    T, per = int(cu[-1]), max(lens) // page + 1
    d = lambda a: torch.as_tensor(np.asarray(a, dtype=np.int32), device="cuda")
    q = rnd(T, (NH + 2 * NKV) * D, dtype=torch.bfloat16, seed=270)
    kp, vp = (rnd(4 * per, NKV, page, D, dtype=torch.bfloat16, seed=s) for s in (271, 272))
    table = torch.randperm(4 * per, device="cuda").to(torch.int32).view(4, per).contiguous()
    table[3, 3] = -1            # a page that is not held
    more = {"sinks": {"sinks": rnd(NH, seed=273)}, "slopes": {"slopes": rnd(NH, seed=274).abs() * 0.01},
            "gate": {"gate": rnd(T, NH * D, dtype=torch.bfloat16, seed=275)}}.get(extra, {})
    run = lambda p: ops.attention_tc(q, torch.full((T, NH * D), 7.0, device="cuda", dtype=torch.float32 if extra == "float" else torch.bfloat16),
                                     kp, vp, d(arrays["tile_seq"]), d(arrays["tile_q0"]), values["n_tiles"], d(cu), d(lens), table, NH, NKV, D,
                                     D ** -0.5, window, keep_first=keep, parts=p, **more)
    torch.testing.assert_close(run(parts), run((1, 0)), **tol(torch.bfloat16))
    assert ops.gemm_status() == 0


@pytest.mark.parametrize("parts", [(2, 0), (3, 0), (8, 0), (1, 3)])
@pytest.mark.parametrize("NH,NKV,D", [(6, 2, 128), (5, 1, 64)])
@pytest.mark.parametrize("what", ["query", "first keys", "last keys", "all keys", "one key", "infinite query", "infinite key", "value"])
def test_shared_out_keys_keep_what_is_no_number(ops, parts, NH, NKV, D, what):
    """A query, keys or a value that are NaN or infinite leave the same entries of the result without a number whether one block
    sees all keys or a cluster shares them (a part whose scores are all NaN has no maximum, but it has a sum); the others are the
    plain softmax's."""
    if parts[1] and (NH // NKV % 2 == 0 or NH // NKV < 3):
        pytest.skip("no odd heads beside pairs")
    import numpy as np
    q_len, length, page = 140, 1100, 16
    arrays, values = ops.attention_work([q_len], [length], [0, q_len])
    per = length // page + 1
    d = lambda a: torch.as_tensor(np.asarray(a, dtype=np.int32), device="cuda")
    q = rnd(q_len, (NH + 2 * NKV) * D, dtype=torch.bfloat16, seed=276)
    kp, vp = (rnd(per, NKV, page, D, dtype=torch.bfloat16, seed=s) for s in (277, 278))
    nan, inf = float("nan"), float("inf")
    at = slice(0, 700 // page) if what == "first keys" else slice(700 // page, per) if what == "last keys" else slice(None)
    if what in ("query", "infinite query"):
        q[[0, 77, 139]] = nan if what == "query" else inf
    elif what in ("first keys", "last keys", "all keys"):
        kp[at] = nan
    elif what == "value":
        vp[3, :, 5] = nan
    else:
        kp[30, :, 7, 2] = nan if what == "one key" else inf
    run = lambda p: ops.attention_tc(q, torch.full((q_len, NH * D), 7.0, device="cuda", dtype=torch.float32), kp, vp, d(arrays["tile_seq"]), d(arrays["tile_q0"]),
                                     values["n_tiles"], d([0, q_len]), d([length]), d(range(per)).view(1, per), NH, NKV, D, D ** -0.5, 0, parts=p)
    got, want = run(parts), run((1, 0))
    assert torch.equal(got.isnan(), want.isnan()) and not want.isinf().any() and not got.isinf().any()
    assert want.isnan().any()
    torch.testing.assert_close(got, want, equal_nan=True, **tol(torch.bfloat16))
    assert ops.gemm_status() == 0


def test_attention_tc_parts():
    """One block where the SMs have enough of them, more where they have not, never more than key tiles."""
    from acvram_b200.kernels.ops import attention_tc_parts
    assert attention_tc_parts(16, (136, 16, 1), 32, 8, 0, 148) == (1, 0)
    assert attention_tc_parts(8, (355, 47, 41), 40, 8, 0, 148) == (1, 2)
    assert attention_tc_parts(8, (355, 47, 41), 16, 8, 0, 148)[0] > 1
    assert attention_tc_parts(8, (355, 47, 41), 16, 8, 2, 148) == (1, 0)
    assert attention_tc_parts(1, (3, 3, 3), 2, 2, 0, 148)[0] <= 3


@pytest.mark.parametrize("NH,NKV,D,T,K", [(32, 8, 128, 8, 4096), (6, 2, 64, 5, 264), (5, 1, 64, 17, 128), (4, 4, 128, 1, 512),
                                          (3, 1, 128, 32, 136),
                                          # many tokens: tokens on the tensor-memory lanes, whole heads inside a thread's row
                                          (8, 2, 128, 300, 512), (6, 2, 64, 129, 264), (5, 1, 64, 700, 128), (3, 1, 128, 257, 136)])
@pytest.mark.parametrize("normed,rotated,pair", [(True, True, False), (False, True, False), (True, False, False), (True, True, True)])
def test_gemm_tc_qkv_epilogue(ops, NH, NKV, D, T, K, normed, rotated, pair):
    """The stacked projection with norm, rotation and append in its own kernel against the projection followed by the
    rotation kernel: the same queries, and the same keys and values in the same pages (the sums of squares are added
    in another order, so a rounding may move here and there)."""
    page, n_pages = 16, 12
    N = (NH + 2 * NKV) * D
    x = rnd(T, K, dtype=torch.bfloat16, seed=150)
    w = rnd(N, K, dtype=torch.bfloat16, scale=0.05, seed=151)
    qw = (1.0 + 0.1 * rnd(D, dtype=torch.float32, seed=152)) if normed else None
    kw = (1.0 + 0.1 * rnd(D, dtype=torch.float32, seed=153)) if normed else None
    table_rows = max(200, T)
    ang = torch.rand(table_rows, D // 2, device="cuda") * 6.28
    cos_sin = torch.cat([ang.cos(), ang.sin()], dim=1).contiguous() if rotated else None
    # tokens of three requests at scattered positions; one token's page is missing (-1)
    seq = torch.tensor([i % 3 for i in range(T)], dtype=torch.int32, device="cuda")
    pos = torch.tensor([(7 * i + 3) % 150 if T <= 32 else i // 3 for i in range(T)], dtype=torch.int32, device="cuda")
    per_request = int(pos.max()) // page + 1
    n_pages = 3 * per_request + 2
    table = torch.randperm(n_pages, device="cuda").to(torch.int32)[:3 * per_request].view(3, per_request).contiguous()
    if T > 2:
        table[int(seq[2]), int(pos[2]) // page] = -1
    if not ops.gemm_tc_qkv_takes(x, w, D, cos_sin, torch.empty(n_pages, NKV, page, D, device="cuda", dtype=torch.bfloat16)):
        pytest.skip("no fused form for this plan")
    if pair and T <= 128:
        pytest.skip("pairs of CTAs serve the tokens-on-rows form")
    plan = (0, 256, 1, 6, ops.GEMM_PAIR) if pair else None
    kp1 = torch.zeros(n_pages, NKV, page, D, device="cuda", dtype=torch.bfloat16)
    vp1, kp2, vp2 = torch.zeros_like(kp1), torch.zeros_like(kp1), torch.zeros_like(kp1)
    want = ops.gemm_tc(x, w, torch.zeros(T, N, device="cuda", dtype=torch.bfloat16))
    ops.qk_norm_rope_append(want, NH, NKV, D, qw, kw, 1e-6, cos_sin, pos, seq, table, kp1, vp1)
    got = torch.zeros(T, N, device="cuda", dtype=torch.bfloat16)
    ops.gemm_tc_qkv(x, w, got, NH, NKV, D, qw, kw, 1e-6, cos_sin, pos, seq, table, kp2, vp2, plan=plan)
    assert ops.gemm_status() == 0
    q1, q2 = want[:, :NH * D], got[:, :NH * D]
    torch.testing.assert_close(q2, q1, **tol(torch.bfloat16))
    torch.testing.assert_close(kp2, kp1, **tol(torch.bfloat16))
    assert torch.equal(vp2, vp1)
    assert (q2 != q1).float().mean() < 0.02 and (kp2 != kp1).float().mean() < 0.02


@pytest.mark.parametrize("tile", [8, 16])
@pytest.mark.parametrize("form", ["gated", "pairs", "plain", "down"])
@pytest.mark.parametrize("T,E,top,N,K", [(1, 4, 2, 64, 64), (13, 6, 3, 96, 640), (40, 3, 2, 32, 2112)])
def test_moe_rows(ops, tile, form, T, E, top, N, K):
    """The experts' products in tiles of 8 and 16 rows against the tiled form, row by row: experts without a row, with a part of a
    tile and with several tiles; K that leaves warps without a chunk and K that their rings go round in."""
    rows = T * top
    g = torch.Generator(device="cuda").manual_seed(280)
    ids = torch.randint(0, max(1, E - 1), (rows,), device="cuda", generator=g, dtype=torch.int32)      # (the last expert has none)
    weight = torch.rand(rows, device="cuda", generator=g) + 0.5
    glu, plain = form in ("gated", "pairs"), "silu" if form == "plain" else None
    w = rnd(E, 2 * N if glu else N, K, dtype=torch.bfloat16, scale=0.05, seed=281)
    outs = []
    for t in (ops.MOE_TILE, tile):
        tiles = ops.moe_max_tiles(rows, E, t)
        grouped, te, place = (torch.empty(n, device="cuda", dtype=torch.int32) for n in (tiles * t, tiles, rows))
        used = torch.empty(1, device="cuda", dtype=torch.int32)
        ops.moe_group(ids, E, grouped, place, te, t, used)
        x = rnd(T, K, dtype=torch.bfloat16, seed=282)
        if form == "down":
            by_row = rnd(rows, K, dtype=torch.bfloat16, seed=283)
            x = torch.zeros(tiles * t, K, device="cuda", dtype=torch.bfloat16)
            x[place.long()] = by_row
        out = torch.zeros(tiles * t, N, device="cuda", dtype=torch.float32 if form == "down" else torch.bfloat16)
        more = dict(limit=7.0, alpha=1.702, pairs=form == "pairs", plain_act=plain)
        if t == ops.MOE_TILE:
            ops.moe_gemm_mma(x, w, out, grouped, te, weight, top, glu, **more)
        else:
            ops.moe_rows(x, w, out, grouped, te, used, t, weight, top, glu, **more)
        outs.append(out[place.long()])
    torch.testing.assert_close(outs[1], outs[0], **(dict(rtol=1e-4, atol=1e-4) if form == "down" else tol(torch.bfloat16)))
    assert outs[0].abs().max() > 0
