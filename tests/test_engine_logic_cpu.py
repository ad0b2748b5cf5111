"""The step function, the batch builder and the cache on the CPU, with each kernel replaced by its
plain PyTorch reference (tests/kernel_refs.py): only the logic is under test here; the kernels
themselves are tested on the GPU."""

from __future__ import annotations

import dataclasses

import pytest
import torch

import kernel_refs
import plain_qwen3
from acvram_b200.engine.batch import StepEntry
from acvram_b200.engine.runner import ModelRunner
from acvram_b200.models import DecoderModel, plan_of_folder
from acvram_b200.parts import Runtime, ScheduleEntry
from acvram_b200.weights import load_tensors
from conftest import TINY_PAGE, random_ids


@pytest.fixture(autouse=True)
def references_in_place_of_kernels(monkeypatch):
    kernel_refs.patch_ops(monkeypatch)


def build(folder, change_plan=None):
    _, plan = plan_of_folder(folder)
    if change_plan:
        plan = change_plan(plan)
    model = DecoderModel(plan)
    model.load(load_tensors(folder, model.tensor_needs()), Runtime(torch.device("cpu"), torch.float32))
    return model


@pytest.mark.parametrize("name", ["A", "B"])
def test_portions_and_mixing_equal_whole(name, tiny_folders, plain_models):
    cfg, t = plain_models[name]
    model = build(tiny_folders[name])
    ids_a = random_ids(cfg["vocab_size"], 45, 1)
    ids_b = random_ids(cfg["vocab_size"], 23, 2)
    ref_a = plain_qwen3.forward_logits(cfg, t, ids_a)
    ref_b = plain_qwen3.forward_logits(cfg, t, ids_b)
    r = ModelRunner(model, TINY_PAGE[name], 10, 4)
    got_a, got_b = [], []
    got_a.append(r.step([StepEntry("a", ids_a[:19], range(19))]))
    lg = r.step([StepEntry("a", ids_a[19:21], range(2)), StepEntry("b", ids_b[:20], range(20))])
    got_a.append(lg[:2]); got_b.append(lg[2:])
    pa, pb = 21, 20
    while pa < 45 or pb < 23:
        entries = []
        if pb < 23:
            entries.append(StepEntry("b", ids_b[pb:pb + 1], [0]))
        if pa < 45:
            n = min(5, 45 - pa)
            entries.append(StepEntry("a", ids_a[pa:pa + n], range(n)))
        lg = r.step(entries)
        if pb < 23:
            got_b.append(lg[:1]); lg = lg[1:]; pb += 1
        if pa < 45:
            got_a.append(lg); pa += n
    assert (torch.cat(got_a) - ref_a).abs().max() < 2e-6
    assert (torch.cat(got_b) - ref_b).abs().max() < 2e-6
    r.release("a"); r.release("b")
    r.manager.check()
    assert r.manager.free_pages() == [10]


def test_wanted_rows_only(tiny_folders, plain_models):
    cfg, t = plain_models["A"]
    model = build(tiny_folders["A"])
    ids = random_ids(cfg["vocab_size"], 12, 3)
    ref = plain_qwen3.forward_logits(cfg, t, ids)
    r = ModelRunner(model, 16, 4, 2)
    assert r.step([StepEntry("a", ids[:5], ())]).shape == (0, cfg["vocab_size"])
    lg = r.step([StepEntry("a", ids[5:], (6, 0))])
    assert (lg[0] - ref[11]).abs().max() < 2e-6 and (lg[1] - ref[5]).abs().max() < 2e-6


def test_a_layer_twice_and_a_shared_cache(tiny_folders, plain_models):
    """The order of layers is data: layer 1 runs twice (each run with a cache slot of its own)."""
    cfg, t = plain_models["B"]
    sched = (ScheduleEntry(0, 0), ScheduleEntry(1, 1), ScheduleEntry(1, 2), ScheduleEntry(2, 3))
    model = build(tiny_folders["B"], lambda p: dataclasses.replace(p, schedule=sched))
    ids = random_ids(cfg["vocab_size"], 30, 4)
    ref = plain_qwen3.forward_logits(cfg, t, ids, schedule=[0, 1, 1, 2])
    r = ModelRunner(model, 8, 8, 2)
    got = torch.cat([r.step([StepEntry("a", ids[:17], range(17))]), r.step([StepEntry("a", ids[17:], range(13))])])
    assert (got - ref).abs().max() < 2e-6
    assert model.cache_plan().slots_per_group == [4]


def test_reading_another_layers_cache(tiny_folders, plain_models):
    """Layer 2 reads the keys and values that layer 1 wrote (it appends nothing of its own)."""
    cfg, t = plain_models["B"]
    sched = (ScheduleEntry(0, 0), ScheduleEntry(1, 1), ScheduleEntry(2, 1, writes=False))
    model = build(tiny_folders["B"], lambda p: dataclasses.replace(p, schedule=sched))
    assert model.cache_plan().slots_per_group == [2]
    ids = random_ids(cfg["vocab_size"], 21, 5)
    r = ModelRunner(model, 8, 8, 2)
    whole = r.step([StepEntry("w", ids, range(21))])
    r.release("w")
    parts = torch.cat([r.step([StepEntry("p", ids[:9], range(9))]), r.step([StepEntry("p", ids[9:], range(12))])])
    assert (whole - parts).abs().max() < 2e-6, "portions equal whole for a layer that shares a cache"
    base = plain_qwen3.forward_logits(cfg, t, ids)
    assert (whole - base).abs().max() > 1e-4, "and sharing the cache does change the model"


def test_window_layers_get_their_own_group_and_free_pages(tiny_folders, plain_models):
    """A window on some layers: another cache group, pages returned as the window passes."""
    cfg, t = plain_models["A"]

    def windowed(plan):
        layers = list(plan.layers)
        layers[1] = dataclasses.replace(layers[1], mixer=layers[1].mixer.with_params(window=16))
        return dataclasses.replace(plan, layers=tuple(layers))

    model = build(tiny_folders["A"], windowed)
    assert len(model.cache_plan().groups) == 2
    ids = random_ids(cfg["vocab_size"], 80, 6)
    r = ModelRunner(model, 8, 12, 2)
    got = []
    pos = 0
    for n in (30, 2, 17, 1, 1, 1, 28):
        got.append(r.step([StepEntry("a", ids[pos:pos + n], range(n))]))
        pos += n
    got = torch.cat(got)
    full_pages, window_pages = r.manager.free_pages()
    assert full_pages == 12 - 10 and window_pages == 12 - 2, "the windowed group holds only the window's pages"
    # plain: layer 0 full, layer 1 windowed
    s = plain_qwen3.sizes(cfg)
    x = plain_qwen3.embed(t["model.embed_tokens.weight"], torch.tensor(ids), torch.float32)
    positions = torch.arange(80)
    x = plain_qwen3.decoder_layer(x, t, 0, s, positions, 0)
    x = plain_qwen3.decoder_layer(x, t, 1, s, positions, 16)
    ref = plain_qwen3.output_logits(x, t, s)
    assert (got - ref).abs().max() < 2e-6


def test_bad_inputs_are_refused(tiny_folders):
    model = build(tiny_folders["A"])
    r = ModelRunner(model, 16, 4, 2)
    with pytest.raises(ValueError):
        r.step([StepEntry("a", [1, 2, 999], ())])
    with pytest.raises(ValueError):
        r.step([StepEntry("b", [1, 2], (5,))])
    with pytest.raises(ValueError):
        r.step([StepEntry("c", [], ())])


def test_requests_that_take_pages_over_get_the_plain_logits(tiny_folders, plain_models):
    """Scheduler and step function together, with prefix reuse and a pool small enough to preempt: requests whose
    prompts begin alike run behind the pages of earlier ones, and the logits that choose each of their tokens are
    the plain implementation's for the tokens they hold (greedy, so the tokens are the plain ones too)."""
    from acvram_b200.engine.scheduler import Request, Scheduler
    from acvram_b200.sampling import SamplingParams
    cfg, t = plain_models["A"]
    model = build(tiny_folders["A"])
    page = 8
    r = ModelRunner(model, page, 14, 3, enable_prefix_cache=True)
    s = Scheduler(r.manager, 3, 24, 128)
    stem = random_ids(cfg["vocab_size"], 40, 31)
    prompts = [stem[:33], stem[:40], stem[:21] + random_ids(cfg["vocab_size"], 9, 32), stem[:33], stem[:9]]
    reqs = [Request(f"r{i}", list(p), SamplingParams(temperature=0.0, max_tokens=7, ignore_eos=True)) for i, p in enumerate(prompts)]
    pending = list(reqs)
    step = 0
    while pending or not s.idle:
        if pending and step % 3 == 0:
            s.add(pending.pop(0))
        plan = s.schedule()
        if plan.entries:
            entries = [StepEntry(e.request.request_id, e.request.token_slice(e.start, e.count),
                                 (e.count - 1,) if e.samples else ()) for e in plan.entries]
            logits = r.step(entries)
            rows = [e.request for e in plan.entries if e.samples]
            for req, row in zip(rows, logits):
                want = plain_qwen3.forward_logits(cfg, t, req.tokens)[-1]
                assert (row - want).abs().max() < 5e-6, f"{req.request_id} at {len(req.tokens)} tokens (took over {req.reused})"
            s.commit(plan, [int(row.argmax()) for row in logits])
        r.manager.check()
        step += 1
        assert step < 400
    for req, p in zip(reqs, prompts):
        assert req.output == plain_qwen3.greedy_generate(cfg, t, p, 7)
    assert s.counters["reused_tokens"] >= 32 + 16 + 32 and r.manager.free_pages() == [14]


def test_step_cost_follows_the_plan(tiny_folders, plain_models):
    """What a step reads and computes, as the parts report it, against the sums written out for this architecture."""
    cfg, _ = plain_models["B"]
    model = build(tiny_folders["B"])
    L, H, I, V = cfg["num_hidden_layers"], cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"]
    NH, NKV, D = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
    matrices = L * (H * (NH + 2 * NKV) * D + NH * D * H + 3 * H * I) + V * H
    norms = L * (2 * H + 2 * D) + H
    q_lens, kv_lens = [1, 1, 5], [30, 7, 12]
    cost = model.step_cost(q_lens, kv_lens, logit_rows=3)
    assert cost["weight_bytes"] == 4 * (matrices + norms)              # a float32 model; norm weights are float32 too
    assert cost["cache_bytes"] == L * 2 * sum(kv_lens) * NKV * D * 4
    seen = 30 + 7 + sum(range(8, 13))                                   # keys that each query sees
    want = 2.0 * 7 * (matrices - V * H) + 2.0 * 3 * V * H + L * 4.0 * NH * D * seen
    assert abs(cost["flops"] - want) < 1e-6 * want
    # a layer that runs twice is read twice
    twice = build(tiny_folders["B"], lambda p: dataclasses.replace(
        p, schedule=p.schedule + (ScheduleEntry(0, p.num_cache_slots, True),)))
    assert twice.step_cost([1], [5], 1)["weight_bytes"] > model.step_cost([1], [5], 1)["weight_bytes"]


def test_the_plan_of_a_product_follows_its_shape():
    """Which tile form a tensor-core product takes, for a device of 148 multiprocessors: weights on the tile's rows up to
    128 tokens (split along K where the tiles alone do not fill the device), tokens on the rows above; pairs of CTAs on
    256 x 256 where their rounds cost less than any width of one CTA's tile, whole heads in a tile where the epilogue
    wants them."""
    from acvram_b200.kernels import ops
    plan = lambda *a, **k: ops.gemm_tc_plan(*a, sms=148, **k)
    for M in (1, 8, 16):
        swap, bn, splits, stages = plan(M, 4096, 4096)[:4]
        assert (swap, bn) == (1, 16) and splits > 1, "32 tiles of weights on 148 SMs: the K range is shared out"
    assert plan(100, 6144, 4096)[:2] == (1, 128)
    for shape in ((2048, 6144, 4096), (2048, 4096, 4096), (2048, 24576, 4096), (2048, 4096, 12288), (8192, 24576, 4096)):
        p = plan(*shape)
        assert p[:3] == (0, 256, 1) and p[4] == ops.GEMM_PAIR, shape
    assert len(plan(1056, 34816, 5120)) == 4 and plan(1056, 34816, 5120)[:2] == (0, 256)      # 1280 rows of pair tiles for 1056 tokens
    assert plan(1056, 5120, 5120)[:2] == (0, 160), "a narrower tile where it saves a round"
    assert plan(1056, 5120, 5120, bn_multiple=128)[1] % 128 == 0
    assert plan(300, 200, 512)[:2] == (0, 128) and plan(300, 40, 512)[:2] == (0, 64)
    # a device with one multiprocessor has no pairs
    assert len(ops.gemm_tc_plan(2048, 4096, 4096, sms=1)) == 4


@pytest.mark.parametrize("M,refused", [(1, True), (65, True), (128, True), (129, False)])
def test_the_clamped_unit_refuses_what_its_documentation_refuses(monkeypatch, M, refused):
    """128 tokens and fewer, also where the plan of a plain product puts them on the rows (a weight of more tiles than SMs)."""
    from acvram_b200.kernels import ops
    launched = []

    class Library:
        def acv_gemm_tc_glu(self, *args):
            launched.append(args)
            return 0

    monkeypatch.setattr(ops, "library", Library)
    monkeypatch.setattr(ops, "_need_cuda", lambda *a: None)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "sm_count", lambda *a: 148)
    monkeypatch.setattr(ops, "_gemm_buffers", lambda *a: (None, None, None))
    N, K = 128 * 160, 64
    x, w, out = (torch.empty(*s, dtype=torch.bfloat16) for s in ((M, K), (N, K), (M, N // 2)))
    if refused:
        with pytest.raises(ops.KernelError, match="more than 128"):
            ops.linear_bf16_glu(x, w, out, 7.0, 1.7)
    else:
        ops.linear_bf16_glu(x, w, out, 7.0, 1.7)
    assert len(launched) == (0 if refused else 1)


@pytest.mark.parametrize("sms", [1, 74, 132, 148, 256])
def test_split_products_share_nothing_between_streams(sms):
    """Splits of K that ``gemm_tc_plan`` asks for are summed inside a cluster (8 CTAs and 100 KB of partial tiles at most),
    through no workspace at all."""
    from acvram_b200.kernels import ops
    for M in (1, 16, 17, 32, 33, 64, 65, 128, 129, 256, 300, 512, 513, 1056):
        for N in list(range(128, 128 * 600, 128 * 7)) + [200, 5120, 4096, 19000]:
            for K in (64, 1024, 2048, 3072, 4096, 8192, 17408):
                swap, bn, splits = ops.gemm_tc_plan(M, N, K, sms=sms)[:3]
                if splits > 1:
                    assert swap and splits <= 8 and (splits - 1) * bn * 128 * 4 <= 100 * 1024, (M, N, K)


def test_products_that_split_through_a_workspace_have_one_each(monkeypatch):
    """The plan by which the experts' router and the wkv decay split a long product has no cluster: each call brings a
    workspace and counters of its own, of the size that the kernel asks for, inside a capture too, whatever ran before."""
    from acvram_b200.kernels import ops
    calls = []

    class Library:
        def acv_gemm_tc(self, *args):
            calls.append(args)
            return 0

    kept = []
    for name in ("empty", "zeros"):         # (kept, so that no address comes twice)
        monkeypatch.setattr(torch, name, lambda *a, make=getattr(torch, name), **k: kept.append(make(*a, **k)) or kept[-1])
    monkeypatch.setattr(ops, "library", Library)
    monkeypatch.setattr(ops, "_need_cuda", lambda *a: None)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "sm_count", lambda *a: 148)
    monkeypatch.setattr(ops, "_gemm_scratch", {})
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    ops.gemm_tc(torch.zeros(4, 64).bfloat16(), torch.zeros(128, 64).bfloat16(), torch.zeros(4, 128))       # (a product ran before)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    w = torch.zeros(64, 2048).bfloat16()
    seen = set()
    for T in (512, 4096, 8192, 8192):
        ops.gemm_tc(torch.zeros(T, 2048).bfloat16(), w, torch.zeros(T, 64), plan=(0, 128, 8, 4, 0))
        workspace, floats, counters, n_counters = calls[-1][14:18]
        tiles = T // 128
        assert floats >= tiles * 8 * 128 * 128 and n_counters >= tiles
        for address, size in ((workspace, 4 * floats), (counters, 4 * n_counters)):
            address = getattr(address, "value", address)
            assert address and not any(a < address + size and address < b for a, b in seen)
            seen.add((address, address + size))
    ops.gemm_tc(torch.zeros(8, 2048).bfloat16(), w, torch.zeros(8, 64), plan=(1, 16, 8, 8))
    assert calls[-1][15] == 0 and calls[-1][17] == 0, "a cluster needs neither"


def test_the_splits_of_decode_attention_follow_what_fits_the_device(monkeypatch):
    """How the split-KV kernel cuts the context, for a device that holds 296 of its CTAs at once (stubbed: the real
    figure is asked of the runtime): a few long requests are split so far that a CTA's own streaming is short, many
    requests not at all; more than 8 splits, through scratch memory, only where 8 leave a CTA thousands of keys; and
    where the clusters of some size fit the device badly, that size is passed over."""
    from acvram_b200.kernels import ops
    fits = {}

    def resident(num_heads, num_kv_heads, head_dim, page_size, n_splits, pages_of_split, cluster_merge, alone=False):
        if alone:       # one CTA to an SM, 148 SMs: whole clusters only
            return {1: 148, 2: 148, 4: 132, 6: 132, 8: 120}[n_splits if cluster_merge else 1]
        return fits.get((n_splits, cluster_merge), 296)
    monkeypatch.setattr(ops, "decode_resident", resident)
    plan = lambda n_dec, max_kv: ops.decode_plan.__wrapped__(n_dec, 32, 8, 128, 64, max_kv)
    assert plan(64, 2048) == (1, False) and plan(64, 16384) == (1, False)
    n, in_clusters = plan(8, 2048)
    assert 2 <= n <= 4 and in_clusters
    n, in_clusters = plan(1, 8192)
    assert n == 8 and in_clusters
    n, in_clusters = plan(1, 65536)
    assert n > 8 and not in_clusters
    assert plan(1, 300) == (1, False), "no split shorter than 256 keys"
    # 24 clusters of 8 for 3 requests: all at once on this device, not on one that holds 15 of them
    assert plan(3, 16384) == (8, True)
    fits[(8, True)] = 120
    assert plan(3, 16384)[0] != 8 or not plan(3, 16384)[1]
    # the cost itself: a second round costs, and so does every split's share of the merge
    one = ops.decode_splits_cost(2, 8, 8192, 8, True, 296, 512)
    assert ops.decode_splits_cost(2, 8, 8192, 8, True, 64, 512) > 1.3 * one
    assert ops.decode_splits_cost(2, 8, 8192, 8, False, 296, 512) > one


def test_the_exponentials_polynomial_is_as_exact_as_the_unit_beside_it():
    """The constants of csrc/attention_tc.cu's 2^f, evaluated in float as the kernel does: over [-1/2, 1/2] the relative
    error stays under 1.3e-7, the least that the special-function unit's largest comes to on any part of the range
    (1.31e-7 to 1.46e-7 over all floats in [-126, 8]), and 2^0 is 1."""
    import os
    import re
    import numpy as np
    import acvram_b200.kernels.build as kbuild
    with open(os.path.join(kbuild.CSRC, "attention_tc.cu")) as f:
        body = f.read().split("at_f2 at_exp2_poly(at_f2 y) {")[1].split("at_split(z, a, b);")[0].split("at_f2 q = ")[1]
    coefficients = [np.float32(c) for c in re.findall(r"at_both\(([-+.0-9e]+)f\)", body)]
    assert len(coefficients) > 4 and coefficients[-1] == 1.0
    f = np.linspace(-0.5, 0.5, 400001).astype(np.float32)
    q = np.full_like(f, coefficients[0])
    for c in coefficients[1:]:          # a fused multiply-add: exact in 64 bits, rounded once
        q = (q.astype(np.float64) * f + np.float64(c)).astype(np.float32)
    exact = 2.0 ** f.astype(np.float64)
    assert (np.abs(q - exact) / exact).max() < 1.3e-7
    assert q[200000] == 1.0 and f[200000] == 0.0


@pytest.mark.parametrize("q_lens,held", [([1], [700]), ([1, 1, 1], [0, 5, 127]), ([128, 1, 129, 2], [0, 40, 255, 126]), ([300, 300, 3], [0, 0, 600]), ([], [])])
def test_attention_work_lists(q_lens, held):
    """The requests of one token, the others' tiles with most keys first (equal ones in the batch's order), and the counts."""
    import numpy as np
    from acvram_b200.kernels.ops import QUERY_TILE, attention_work
    kv_lens, cu = [h + q for h, q in zip(held, q_lens)], np.concatenate([[0], np.cumsum(q_lens)]).astype(np.int32)
    tiles = [(i, a, held[i] + min(a + QUERY_TILE, q)) for i, q in enumerate(q_lens) if q > 1 for a in range(0, q, QUERY_TILE)]
    tiles.sort(key=lambda t: -t[2])
    blocks = [-(-t[2] // QUERY_TILE) for t in tiles]
    dec = [i for i, q in enumerate(q_lens) if q == 1]
    arrays, values = attention_work(q_lens, kv_lens, cu)
    assert all(a.dtype == np.int32 for a in arrays.values())
    assert {k: a.tolist() for k, a in arrays.items()} == {"dec_tokens": [int(cu[i]) for i in dec], "dec_seqs": dec,
                                                          "tile_seq": [t[0] for t in tiles], "tile_q0": [t[1] for t in tiles]}
    assert values == {"n_dec": len(dec), "n_tiles": len(tiles), "max_dec_kv": max((kv_lens[i] for i in dec), default=0),
                      "max_tile_kv": max((k for k, q in zip(kv_lens, q_lens) if q > 1), default=0),
                      **({"tile_blocks": (sum(blocks), max(blocks), min(blocks))} if tiles else {})}


@pytest.mark.parametrize("head_dim", [64, 128])
def test_blocks_that_share_keys_have_an_sm_each(head_dim):
    """Blocks of a cluster that waits for all of its blocks while each holds all of an SM's tensor memory: two of them on one SM
    could wait for each other's columns without an end.  Their shared memory alone (228 KB an SM, 1 KB of it to each block's
    system) keeps them apart, whatever registers the compiler gives them."""
    from acvram_b200.kernels import ops
    assert 2 * (ops.library().acv_attention_tc_shared_bytes(head_dim, 2) + 1024) > 228 * 1024


def _device_functions(path):
    """(name, is it a kernel, body) of the functions of a CUDA source, which begin and end at a line's start."""
    import re
    with open(path) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for head, body in re.findall(r"^((?:template|__global__|__device__|static __device__)[^;{]*?)\{\n(.*?)^\}", text, re.M | re.S):
        name = re.search(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\([^)]*\)", "", head))
        if name:            # (not a struct)
            yield name.group(1), "__global__" in head, body


@pytest.mark.parametrize("source", ["sampling.cu", "gemm_rows.cu", "gemm_split_tc.cu", "gemm_simt.cu", "attention_tc.cu", "attention_decode.cu",
                                    "attention_generic.cu", "gemm_tc.cu"])
def test_kernels_know_that_their_cluster_has_started_before_they_touch_a_peer(source):
    """A block's shared memory may be touched by a peer only once the block is known to run: in each kernel a wait of the
    cluster's barrier stands before the first peer address, also where a function that it calls makes that address."""
    import os
    import re
    import acvram_b200.kernels.build as kbuild
    functions = list(_device_functions(os.path.join(kbuild.CSRC, source)))
    touches, kernels = {"cluster_map"}, 0
    for _ in functions:         # (functions that touch a peer before they have waited for the cluster themselves)
        for name, kernel, body in functions:
            peer = re.search(r"\b(" + "|".join(touches) + r")\s*\(", body)
            waited = re.search(r"\bcluster_(wait|sync_all)\s*\(", body)
            if peer and not (waited and waited.start() < peer.start()):
                assert not kernel, f"{source}: {name} touches a peer through {peer.group(1)} before it has waited for its cluster"
                touches.add(name)
            kernels += bool(kernel and peer)
    assert kernels


def test_read_only_loads_are_of_what_no_kernel_in_front_writes():
    """Kernels begin while the one in front still runs, and ``__ldg`` is for what stays as it is for a kernel's whole life: norm
    weights and biases, never a row of activations."""
    import os
    import re
    import acvram_b200.kernels.build as kbuild
    constants = ("w + i0 + c", "w + half + i0 + c", "reinterpret_cast<const float4*>(p.bias + col0")
    for path in kbuild.sources() + kbuild._headers():
        with open(path) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        assert "ld.global.nc" not in text, path
        for found in re.finditer(r"__ldg\(", text):
            assert text[found.end():].startswith(constants), f"{os.path.basename(path)}: {text[found.start():found.end() + 40]!r}"


@pytest.mark.parametrize("wrong", ["positions", "seq_of_token", "block_table", "k_pages", "v_pages", "k_pages + 8", "v_pages + 4", "cos_sin + 4", "out + 2",
                                   "ldo", "page_size", "N", "D", "NKV"])
def test_the_projection_of_few_tokens_refuses_what_the_others_refuse(wrong):
    """A missing array, pages, angles or a result off their 16 bytes, sizes that do not fit: refused on the host by both entry points of
    the projection with its norm, rotation and append, so that a call does not depend on its number of tokens."""
    import ctypes
    from acvram_b200.kernels import ops
    lib = ops.library()
    at = 1 << 20            # (an address that nobody reads: the call ends at its checks)
    a = dict(x=at, ldx=1024, w=at, ldw=1024, out=at, ldo=4096, M=8, N=4096, K=1024, NH=16, NKV=8, D=128, q_w=None, k_w=None, eps=1e-6, cos_sin=at,
             table_rows=100, positions=at, seq_of_token=at, block_table=at, bt_stride=16, bt_rows=None, k_pages=at, v_pages=at, page_size=16, num_pages=8)
    name, _, add = wrong.partition(" + ")
    a[name] = a[name] + int(add) if add else {"ldo": 4100, "page_size": 0, "N": 4224, "D": 96, "NKV": 0}.get(name)
    tail = [a[k] for k in ("NH", "NKV", "D", "q_w", "k_w")] + [ctypes.c_float(a["eps"])] + [
        a[k] for k in ("cos_sin", "table_rows", "positions", "seq_of_token", "block_table", "bt_stride", "bt_rows", "k_pages", "v_pages", "page_size", "num_pages")] + [None]
    head = [a[k] for k in ("x", "ldx", "w", "ldw", "out", "ldo", "M", "N", "K")]
    size = -3
    assert lib.acv_gemm_rows_qkv(*head, 1, 148, *tail) == size
    if name not in ("out", "ldo"):          # (those the other finds out behind its tensor maps, which need a device)
        assert lib.acv_gemm_tc_qkv(*head, 1, 16, 1, None, 0, None, 0, at, 148, 4, 2, *tail) == size


def test_attention_work_over_many_batches():
    """The native lists against a sort in plain Python, over batches of all kinds: one-token requests, portions behind contexts,
    tiles that see equally many keys, many of each."""
    import random
    import numpy as np
    from acvram_b200.kernels.ops import QUERY_TILE, attention_work
    r = random.Random(3)
    for _ in range(300):
        q_lens = [r.choice([1, 1, 2, 127, 128, 129, 300, r.randrange(1, 3000)]) for _ in range(r.choice([1, 2, 3, 20, 150]))]
        kv_lens = [q + r.choice([0, 0, 128, r.randrange(5000)]) for q in q_lens]
        cu = np.concatenate([[0], np.cumsum(q_lens)]).astype(np.int32)
        tiles = [(i, a, kv - q + min(a + QUERY_TILE, q)) for i, (q, kv) in enumerate(zip(q_lens, kv_lens)) if q > 1 for a in range(0, q, QUERY_TILE)]
        tiles.sort(key=lambda t: -t[2])
        blocks = [-(-t[2] // QUERY_TILE) for t in tiles]
        dec = [i for i, q in enumerate(q_lens) if q == 1]
        arrays, values = attention_work(q_lens, kv_lens, cu)
        assert {k: (a.dtype, a.tolist()) for k, a in arrays.items()} == {
            k: (np.int32, v) for k, v in {"dec_tokens": [int(cu[i]) for i in dec], "dec_seqs": dec, "tile_seq": [t[0] for t in tiles],
                                          "tile_q0": [t[1] for t in tiles]}.items()}
        assert values == {"n_dec": len(dec), "n_tiles": len(tiles), "max_dec_kv": max((kv_lens[i] for i in dec), default=0),
                          "max_tile_kv": max((k for k, q in zip(kv_lens, q_lens) if q > 1), default=0),
                          **({"tile_blocks": (sum(blocks), max(blocks), min(blocks))} if tiles else {})}


def test_shares_of_a_tile_are_the_cheapest_by_the_model():
    """The native choice of blocks to a tile's keys against the model in plain Python, over groups of one to nine heads, windows, and
    few and many tiles."""
    import random
    from acvram_b200.kernels.ops import attention_tc_parts
    at_once_of = (0, 148, 74, 45, 33, 26, 22, 15, 15)

    def cheapest(units, work, longest, shortest, most, sms):
        best = None
        for parts in range(1, max(1, min(8, most)) + 1):
            at_once = max(1, at_once_of[parts] * sms // 148)
            span = longest if parts == 1 else longest / most * -(-most // parts)
            if units > at_once:
                span = max(span, work / (parts * at_once) + shortest / parts)
            cost = -(-units // at_once) * (4.0 if parts == 1 else 12.0) + span * 2.1
            if best is None or cost < (0.95 * best[0] if best[1] == 1 else best[0]):
                best = (cost, parts)
        return best

    r, seen = random.Random(4), set()
    for _ in range(2000):
        blocks = [r.randrange(1, r.choice([2, 9, 70, 300])) for _ in range(r.choice([1, 2, 8, 40]))]
        if r.random() < 0.5:        # (a portion behind a context)
            blocks = [blocks[0] + i for i in range(r.choice([1, 4, 8, 16]))]
        n, total, longest, shortest = len(blocks), sum(blocks), max(blocks), min(blocks)
        kv, rep, limit, sms = r.choice([1, 2, 4, 8]), r.randrange(1, 10), r.choice([0, 0, 1, 5, 40]), r.choice([148, 132])
        got = attention_tc_parts(n, (total, longest, shortest), kv * rep, kv, limit, sms)
        if limit and limit < longest:
            total, longest, shortest = min(total, n * limit), limit, min(shortest, limit)
        pairs, odd = rep // 2, rep % 2
        lone = lambda: cheapest(n * kv, total * kv * 0.6, longest * 0.6, shortest * 0.6, longest, sms)
        if rep == 1:
            want = lone()[1], 0
        else:
            cost, parts = cheapest(n * kv * (pairs + odd), total * kv * (pairs + 0.6 * odd), longest, shortest * (0.6 if odd else 1.0), longest, sms)
            a, b = cheapest(n * kv * pairs, total * kv * pairs, longest, shortest, longest, sms), lone()
            want = (a[1], b[1]) if odd and a[0] + b[0] + 3.0 < 0.95 * cost else (parts, 0)
        assert got == want, (blocks, kv, rep, limit, sms)
        seen.add(want)
    assert {w[0] for w in seen} >= set(range(1, 9)) and any(w[1] for w in seen)


@pytest.mark.parametrize("which", ["neither", "up", "down"])
@pytest.mark.parametrize("how", ["off its 16 bytes", "every other matrix", "float"])
def test_experts_of_few_rows_want_both_products_weights_dense_and_aligned(which, how):
    """Weights that the tiled products on the tensor cores leave to the CUDA cores are not sent to the kernel for few rows, which
    would refuse them: the first product's and the second's alike."""
    import torch
    from acvram_b200.kernels import ops
    E, H, F = 4, 128, 64

    def weights(rows, cols, odd):
        if not odd:
            return torch.zeros(E, rows, cols, dtype=torch.bfloat16)
        if how == "float":
            return torch.zeros(E, rows, cols)
        if how == "every other matrix":
            return torch.zeros(2 * E, rows, cols, dtype=torch.bfloat16)[::2]
        return torch.zeros(E * rows * cols + 4, dtype=torch.bfloat16)[4:].view(E, rows, cols)

    h = torch.zeros(3, H, dtype=torch.bfloat16)
    tile = ops.moe_rows_tile(6, E, h, weights(2 * F, H, which == "up"), weights(H, F, which == "down"))
    assert (tile == 8) == (which == "neither")


@pytest.mark.parametrize("M,N,K,pays", [
    (1, 6144, 1024, True), (8, 4096, 4096, True), (16, 4096, 1024, True), (32, 6144, 512, True), (8, 32768, 512, True), (1, 151936, 1024, True),
    (8, 151936, 4096, True), (2, 65536, 1024, True), (5, 16400, 1024, True),
    # measured slower than with tiles of 128 weight rows: short K behind many blocks, sixteen rows to a block, even last rounds there
    (32, 32768, 128, False), (16, 49168, 64, False), (8, 49152, 512, False), (8, 49168, 640, False), (4, 32784, 256, False), (8, 32768, 128, False),
    (8, 24576, 64, False), (16, 24576, 512, False), (16, 16400, 512, False), (32, 12288, 640, False), (2, 131072, 1024, False), (8, 66000, 1024, False),
    # sizes that the kernel does not take
    (33, 4096, 1024, False), (8, 4104, 1024, False), (8, 4096, 1000, False)])
def test_products_of_few_tokens_go_where_they_are_faster(M, N, K, pays):
    from acvram_b200.kernels import ops
    assert ops.gemm_rows_pays(M, N, K, 148) == pays


@pytest.mark.parametrize("T,E,top,W,F,tile", [
    (1, 64, 6, 4096, 1024, 8), (40, 64, 6, 4096, 1024, 8), (41, 64, 6, 4096, 1024, 16), (64, 64, 6, 4096, 1024, 16), (106, 64, 6, 4096, 1024, 16),
    (107, 64, 6, 4096, 1024, 0), (64, 128, 8, 2048, 768, 8), (56, 32, 4, 2048, 768, 16), (113, 32, 2, 2048, 768, 0), (64, 64, 8, 768, 384, 0),
    (32, 64, 8, 768, 384, 8), (64, 32, 4, 1024, 256, 16), (4, 8, 2, 96, 64, 0), (4, 8, 2, 128, 96, 0)])
def test_tiles_of_experts_of_few_rows(T, E, top, W, F, tile):
    """Eight or sixteen rows by the rows to an expert and the tokens, which bound how often an expert's weights are read, however
    unevenly they choose; none for short rows behind many blocks and for sizes that the kernel does not take."""
    import torch
    from acvram_b200.kernels import ops
    weights = lambda rows, cols: torch.empty(E, rows, cols, dtype=torch.bfloat16)
    assert ops.moe_rows_tile(T * top, E, torch.zeros(T, W, dtype=torch.bfloat16), weights(2 * F, W), weights(W, F)) == tile
