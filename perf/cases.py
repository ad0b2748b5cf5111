"""The work that users of acvram_b200 have it do, as cases that can be timed and compared.

The kinds, each through an entry point that a program calls:

    step       a whole model, ``ModelRunner.step``: decoding requests (replayed from a captured graph) or prompts; logits
    attention  one attention layer's mixer: decoding requests, portions of prompts behind a context, or both in a step
    mlp        the gated feed-forwards of a model's layers, one after the other
    moe        one mixture of experts
    delta      one gated delta mixer: prompts, or requests that bring one token
    sample     the sampler over a vocabulary's logits

Steps in which every request brings one token are replayed from CUDA graphs by the engine; the parts' cases do the same
for up to 64 such rows.  All weights are random, N(0, 0.02) with norm weights around one and embedding rows of unit
size (as a trained model's stream has), in bfloat16 (a float32 run holds the same values); layer sizes are those that
the benchmark and its notes name.
"""

from __future__ import annotations

import math
import random

import torch

DEVICE = "cuda:0"
EPS = 1e-6
THETA = 1e6
POSITIONS = 16384

# hidden, intermediate, query heads, kv heads, head size
SIZES = {
    "0.6b": (1024, 3072, 16, 8, 128),
    "1.7b": (2048, 6144, 16, 8, 128),
    "4b": (2560, 9728, 32, 8, 128),
    "8b": (4096, 12288, 32, 8, 128),
    "14b": (5120, 17408, 40, 8, 128),
}
# width, experts, choices, an expert's size; value heads, query/key heads, key size, value size, taps of the delta mixer
ZOGAPEL = {
    "s": (2048, 32, 4, 768, 16, 8, 128, 128, 4),
    "m": (4096, 64, 6, 1024, 32, 16, 128, 128, 4),
}
VOCAB = 151936
GRAPH_ROWS = 64         # decode steps of up to so many rows are captured here


def listed() -> list[dict]:
    return [
        # one user chatting with a small model: the smallest step there is
        {"name": "step_0.6b_decode_1", "kind": "step", "size": "0.6b", "dtype": "bf16", "layers": 6, "batch": 1, "context": 700, "new": 1},
        # the headline: eight users at 2048-token contexts, some of the layers of the 8B sizes and the whole head
        {"name": "step_8b_decode_8", "kind": "step", "size": "8b", "dtype": "bf16", "layers": 4, "batch": 8, "context": 2048, "new": 1},
        # a check of the model in 32-bit: a few prompts of odd lengths, whole
        {"name": "step_0.6b_f32_prompts", "kind": "step", "size": "0.6b", "dtype": "f32", "layers": 4, "batch": 3, "context": 0, "new": 301},
        # the same model's tokens one by one
        {"name": "step_0.6b_f32_decode_3", "kind": "step", "size": "0.6b", "dtype": "f32", "layers": 4, "batch": 3, "context": 500, "new": 1},
        # a full house: 64 users, contexts of all lengths
        {"name": "attention_8b_decode_64", "kind": "attention", "size": "8b", "batch": 64, "context": 4096, "portion": 0, "prefix": 0},
        # a prompt in one step, what a first answer waits for
        {"name": "attention_8b_prompt_2048", "kind": "attention", "size": "8b", "batch": 0, "context": 0, "portion": 2048, "prefix": 0},
        # serving under load: decoding requests beside a portion of somebody's long prompt
        {"name": "attention_14b_mixed", "kind": "attention", "size": "14b", "batch": 32, "context": 1500, "portion": 1000, "prefix": 5000},
        # the feed-forwards of a decode step of a batch of an odd size
        {"name": "mlp_4b_decode_5", "kind": "mlp", "size": "4b", "layers": 3, "tokens": 5},
        # the feed-forward of a prompt
        {"name": "mlp_8b_prompt_2048", "kind": "mlp", "size": "8b", "layers": 1, "tokens": 2048},
        # experts for a decode step of a middling batch: most of them are chosen by a row or two
        {"name": "moe_m_decode_16", "kind": "moe", "size": "m", "tokens": 16},
        # a recurrent layer over a prompt of ragged requests
        {"name": "delta_s_prompts_1500", "kind": "delta", "size": "s", "batch": 3, "context": 0, "new": 500},
        # sampled decoding, nucleus and the other rules, for a batch
        {"name": "sample_16", "kind": "sample", "batch": 16, "vocab": VOCAB, "logprobs": False},
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["step", "step", "step32", "attention", "attention", "mlp", "mlp", "moe", "delta", "sample"])
    if kind == "step":
        if rng.random() < 0.7:
            size = rng.choice(["0.6b", "1.7b", "4b", "8b"])
            return {"kind": "step", "size": size, "dtype": "bf16", "layers": 3, "batch": _log(rng, 1, 64), "context": _log(rng, 16, 4096), "new": 1}
        return {"kind": "step", "size": rng.choice(["0.6b", "1.7b", "4b"]), "dtype": "bf16", "layers": 2, "batch": rng.randint(1, 3),
                "context": 0, "new": _log(rng, 16, 600)}
    if kind == "step32":
        if rng.random() < 0.5:
            return {"kind": "step", "size": rng.choice(["0.6b", "1.7b"]), "dtype": "f32", "layers": 2, "batch": _log(rng, 1, 16),
                    "context": _log(rng, 16, 1500), "new": 1}
        return {"kind": "step", "size": "0.6b", "dtype": "f32", "layers": 2, "batch": rng.randint(1, 3), "context": 0, "new": _log(rng, 16, 400)}
    if kind == "attention":
        size = rng.choice(["0.6b", "1.7b", "8b", "14b"])
        shape = rng.randrange(3)
        if shape == 0:
            return {"kind": "attention", "size": size, "batch": _log(rng, 1, 64), "context": _log(rng, 64, 4096), "portion": 0, "prefix": 0}
        prefix = rng.choice([0, _log(rng, 16, 5000)])
        return {"kind": "attention", "size": size, "batch": 0 if shape == 1 else rng.randint(1, 32), "context": 0 if shape == 1 else _log(rng, 64, 2000),
                "portion": _log(rng, 64, 2048), "prefix": prefix}
    if kind == "mlp":
        size = rng.choice(list(SIZES))
        tokens = _log(rng, 1, 1100)
        return {"kind": "mlp", "size": size, "layers": {"0.6b": 16, "1.7b": 6, "4b": 3}.get(size, 1) if tokens <= 64 else 1, "tokens": tokens}
    if kind == "moe":
        return {"kind": "moe", "size": rng.choice(list(ZOGAPEL)), "tokens": _log(rng, 1, 1500)}
    if kind == "delta":
        size = rng.choice(list(ZOGAPEL))
        if rng.random() < 0.5:
            return {"kind": "delta", "size": size, "batch": rng.randint(1, 4), "context": 0, "new": _log(rng, 16, 600)}
        return {"kind": "delta", "size": size, "batch": _log(rng, 1, 64), "context": rng.randint(1, 40), "new": 1}
    return {"kind": "sample", "batch": _log(rng, 1, 64), "vocab": rng.choice([VOCAB, 32768, _log(rng, 20000, 200000)]),
            "logprobs": rng.random() < 0.3}


# ----------------------------------------------------------------------------- inputs, the same for every reader
def _gen(seed: int, salt: int) -> torch.Generator:
    return torch.Generator(device=DEVICE).manual_seed((seed * 1000003 + salt) & 0x7FFFFFFF)


def _normal(g: torch.Generator, *shape: int, std: float = 1.0, mean: float = 0.0) -> torch.Tensor:
    return torch.empty(shape, device=DEVICE, dtype=torch.bfloat16).normal_(mean, std, generator=g)


def _lengths(batch: int, longest: int) -> list[int]:
    """Ragged lengths, the first the longest, none under half of it (a property of the case, not of its seed)."""
    return [max(1, longest - (i * 7919) % max(1, longest // 2)) for i in range(batch)]


def _qwen3_shapes(case: dict, vocab: int) -> dict:
    H, I, NH, NKV, D = SIZES[case["size"]]
    shapes = {"model.embed_tokens.weight": (vocab, H), "model.norm.weight": (H,), "lm_head.weight": (vocab, H)}
    for i in range(case.get("layers", 1)):
        p = f"model.layers.{i}."
        shapes.update({
            p + "input_layernorm.weight": (H,), p + "post_attention_layernorm.weight": (H,),
            p + "self_attn.q_proj.weight": (NH * D, H), p + "self_attn.k_proj.weight": (NKV * D, H),
            p + "self_attn.v_proj.weight": (NKV * D, H), p + "self_attn.o_proj.weight": (H, NH * D),
            p + "self_attn.q_norm.weight": (D,), p + "self_attn.k_norm.weight": (D,),
            p + "mlp.gate_proj.weight": (I, H), p + "mlp.up_proj.weight": (I, H), p + "mlp.down_proj.weight": (H, I)})
    return shapes


def _zogapel_shapes(case: dict) -> dict:
    W, E, _, F, NV, NK, D, DV, K = ZOGAPEL[case["size"]]
    p = "l0."
    shapes = {"embed": (256, W), "final.norm": (W,), p + "norm1": (W,), p + "norm1b": (W,)}
    m = p + "mix."
    for role, n in (("q", NK * D), ("k", NK * D), ("v", NV * DV)):
        shapes.update({m + role: (n, W), m + role + ".conv": (n, K)})
    shapes.update({m + "g": (NV * DV, W), m + "b": (NV, W), m + "a": (NV, W), m + "A_log": (NV,), m + "dt_bias": (NV,),
                   m + "norm": (DV,), m + "o": (W, NV * DV)})
    if case["kind"] == "moe":
        shapes.update({p + "norm2": (W,), p + "norm2b": (W,), p + "mlp.router": (E, W), p + "mlp.router.b": (E,)})
        for e in range(E):
            shapes.update({f"{p}mlp.e{e}.gate": (F, W), f"{p}mlp.e{e}.up": (F, W), f"{p}mlp.e{e}.down": (W, F)})
    return shapes


def _tensors(shapes: dict, seed: int) -> dict:
    g = _gen(seed, 1)
    out = {}
    for name, shape in shapes.items():
        if name.endswith(".conv"):
            out[name] = _normal(g, *shape, std=0.5)
        elif name.endswith(("A_log", "dt_bias", "router.b")):
            out[name] = _normal(g, *shape, std=0.1)
        elif len(shape) == 1:
            out[name] = _normal(g, *shape, std=0.1, mean=0.0 if name.startswith(("l0.norm", "final")) else 1.0)
        else:
            out[name] = _normal(g, *shape, std=1.0 if name == "model.embed_tokens.weight" else 0.02)
    return out


def _context(case: dict, seed: int, layer: int, request: int, length: int):
    """Keys and values of a request's context as the cache holds them: keys of unit size after norm and rotation."""
    NKV, D = SIZES[case["size"]][3:]
    g = _gen(seed, 1000 + layer * 4096 + request)
    return _normal(g, length, NKV, D), _normal(g, length, NKV, D)


def _ids(case: dict, seed: int) -> list[list[int]]:
    r = random.Random(seed * 31 + 7)
    new = [1] * case["batch"] if case["new"] == 1 else _lengths(case["batch"], case["new"])
    return [[r.randrange(VOCAB) for _ in range(n)] for n in new]


def _attention_work(case: dict) -> list[tuple[int, int]]:
    """(keys before the step, new tokens) of each request of an attention case."""
    rows = [(n - 1, 1) for n in _lengths(case["batch"], max(case["context"], 2))]
    return rows + ([(case["prefix"], case["portion"])] if case["portion"] else [])


def _tokens(case: dict, seed: int, T: int, width: int) -> torch.Tensor:
    """A layer's input: what a norm leaves."""
    return _normal(_gen(seed, 2), T, width)


# ----------------------------------------------------------------------------- what a user's program holds
def _qwen3(case: dict, seed: int, dtype: torch.dtype, vocab: int):
    from acvram_b200.config import Qwen3Config
    from acvram_b200.models import DecoderModel
    from acvram_b200.models.qwen3 import qwen3_plan
    from acvram_b200.parts import Runtime

    H, I, NH, NKV, D = SIZES[case["size"]]
    cfg = Qwen3Config(vocab_size=vocab, hidden_size=H, intermediate_size=I, num_hidden_layers=case.get("layers", 1),
                      num_attention_heads=NH, num_key_value_heads=NKV, head_dim=D, rms_norm_eps=EPS, rope_theta=THETA,
                      max_position_embeddings=POSITIONS, tie_word_embeddings=False)
    model = DecoderModel(qwen3_plan(cfg))
    model.load(_tensors(_qwen3_shapes(case, vocab), seed), Runtime(torch.device(DEVICE), dtype))
    return model


def _zogapel(case: dict, seed: int):
    from acvram_b200.config import ZogapelConfig
    from acvram_b200.models import DecoderModel
    from acvram_b200.models.zogapel import zogapel_plan
    from acvram_b200.parts import Runtime

    W, E, top, F, NV, NK, D, DV, K = ZOGAPEL[case["size"]]
    moe = {"kind": "moe", "router": {"experts": E, "top": top}, "expert": {"ff": F}} if case["kind"] == "moe" else None
    cfg = ZogapelConfig.from_dict({
        "architecture": "Zogapel", "vocab": 256, "width": W, "embedding": {"scale": 1.0}, "norm": {"eps": EPS},
        "layers": [{"type": "delta", "mixer": {"heads": NV, "kv_heads": NK, "dim": D, "vdim": DV, "conv": K}, "mlp": moe}]})
    model = DecoderModel(zogapel_plan(cfg))
    model.load(_tensors(_zogapel_shapes(case), seed), Runtime(torch.device(DEVICE), torch.bfloat16))
    return model


def _seat(runner, names, lengths) -> None:
    """The requests hold so many tokens each."""
    for name, n in zip(names, lengths):
        if name in runner.manager.lengths:
            runner.release(name)
    for name, n in zip(names, lengths):
        runner.admit(name)
        if n:
            runner.manager.grow(name, n)
            runner.manager.advance(name, n)


def _fill(runner, case: dict, seed: int, names, lengths) -> None:
    """Random pages, and each request's context where its block table says."""
    for slot in range(runner.model.plan.num_cache_slots):
        for pages in runner.storage.pages(slot):
            pages.normal_(generator=_gen(seed, 3 + slot))
        page = runner.manager.page_size
        for r, (name, n) in enumerate(zip(names, lengths)):
            if n == 0:
                continue
            table = torch.tensor(runner.manager.block_table(name, 0), device=DEVICE)
            at = torch.arange(n, device=DEVICE)
            for pages, rows in zip(runner.storage.pages(slot), _context(case, seed, slot, r, n)):
                pages[table[at // page], :, at % page] = rows.to(pages.dtype)


def _captured(fn):
    """``fn`` as a replayed graph, as the engine runs decode steps: (graph, what it returns)."""
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fn()
    return graph, out


GROWTH = 1000       # tokens a decoding request of a step case may grow by before it makes room for another


@torch.no_grad()
def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "step":
        from acvram_b200.engine.batch import StepEntry
        from acvram_b200.engine.runner import ModelRunner

        dtype = torch.float32 if case["dtype"] == "f32" else torch.bfloat16
        model = _qwen3(case, seed, dtype, VOCAB)
        ids = _ids(case, seed)
        names = [f"r{i}" for i in range(case["batch"])]
        page = 16
        decode = case["new"] == 1
        lengths = _lengths(case["batch"], case["context"]) if decode else [0] * case["batch"]
        room = sum(n + GROWTH + 2 * page for n in lengths) if decode else sum(len(i) + page for i in ids)
        runner = ModelRunner(model, page, room // page + 8, case["batch"], max_len=POSITIONS)
        if decode and dtype == torch.bfloat16:
            runner.enable_graphs()
        entries = [StepEntry(n, i, (len(i) - 1,)) for n, i in zip(names, ids)]
        if decode:
            _seat(runner, names, lengths)
            _fill(runner, case, seed, names, lengths)
        return {"kind": kind, "runner": runner, "entries": entries, "names": names, "lengths": lengths, "decode": decode}
    if kind == "attention":
        from acvram_b200.engine.batch import StepEntry
        from acvram_b200.engine.runner import ModelRunner

        work = _attention_work(case)
        model = _qwen3(case, seed, torch.bfloat16, 256)
        page = 64
        T = sum(q for _, q in work)
        names = [f"r{i}" for i in range(len(work))]
        runner = ModelRunner(model, page, sum((n + q) // page + 1 for n, q in work) + 4, len(work), max_len=POSITIONS)
        lengths = [n for n, _ in work]
        _seat(runner, names, lengths)
        _fill(runner, case, seed, names, lengths)
        ctx = runner.prepare([StepEntry(n, [1] * q, ()) for n, (_, q) in zip(names, work)])
        # (the runner has reserved the pages; the context of the step is read by every pass)
        from acvram_b200.parts import CacheView
        k_pages, v_pages = runner.storage.pages(0)
        view = CacheView(0, True, k_pages=k_pages, v_pages=v_pages)
        h = _tokens(case, seed, T, SIZES[case["size"]][0])
        mixer = model.blocks[0].mixer
        state = {"kind": kind, "keep": runner, "call": lambda: mixer.forward(h, ctx, view), "pages": (k_pages, v_pages)}
        if case["portion"] == 0 and T <= GRAPH_ROWS:
            state["graph"], state["out"] = _captured(state["call"])
        return state
    if kind in ("mlp", "moe"):
        if kind == "mlp":
            model, width = _qwen3(case, seed, torch.bfloat16, 256), SIZES[case["size"]][0]
        else:
            model, width = _zogapel(case, seed), ZOGAPEL[case["size"]][0]
        h = _tokens(case, seed, case["tokens"], width)
        units = [b.feed_forward for b in model.blocks]
        state = {"kind": kind, "keep": model, "call": lambda: [u.forward(h, None) for u in units]}
        if case["tokens"] <= GRAPH_ROWS:
            state["graph"], state["out"] = _captured(state["call"])
        return state
    if kind == "delta":
        from acvram_b200.engine.batch import StepEntry
        from acvram_b200.engine.runner import ModelRunner
        from acvram_b200.parts import CacheView

        model = _zogapel(case, seed)
        B = case["batch"]
        news = [1] * B if case["new"] == 1 else _lengths(B, case["new"])
        olds = _lengths(B, case["context"]) if case["context"] else [0] * B
        runner = ModelRunner(model, 16, 8, B, max_len=POSITIONS)
        names = [f"r{i}" for i in range(B)]
        rows = _tokens(case, seed, sum(olds) + sum(news), ZOGAPEL[case["size"]][0])
        leaves = dict(((path, runner.storage.state(slot)) for path, slot in model.slot_leaves[0]))
        groups = dict(((path, runner.manager.plan.group_of_slot[slot]) for path, slot in model.slot_leaves[0]))
        view = CacheView(-1, True, parts={p[-1]: CacheView(groups[p], True, state=t) for p, t in leaves.items()})
        mixer = model.blocks[0].mixer
        if sum(olds):       # the requests' earlier tokens, which leave their states
            ctx = runner.prepare([StepEntry(n, [1] * k, ()) for n, k in zip(names, olds)])
            mixer.forward(rows[:sum(olds)], ctx, view)
            for n, k in zip(names, olds):
                runner.manager.advance(n, k)
        ctx = runner.prepare([StepEntry(n, [1] * k, ()) for n, k in zip(names, news)])
        h = rows[sum(olds):]
        state = {"kind": kind, "keep": runner, "call": lambda: mixer.forward(h, ctx, view), "states": list(leaves.values())}
        if case["new"] == 1:
            saved = [t.clone() for t in leaves.values()]
            state["graph"], state["out"] = _captured(state["call"])
            for t, s in zip(leaves.values(), saved):
                t.copy_(s)
        return state
    from acvram_b200.sampling import SamplingParams
    from acvram_b200.sampling.sampler import Sampler

    B = case["batch"]
    logits = torch.empty((B, case["vocab"]), device=DEVICE).normal_(0.0, 2.5, generator=_gen(seed, 2))
    kinds = [dict(temperature=0.7, top_p=0.9), dict(temperature=1.0, top_p=0.95, top_k=50), dict(temperature=0.7, top_p=0.9),
             dict(temperature=1.2, min_p=0.05), dict(temperature=0.0), dict(temperature=0.8, top_k=20)]
    params = [SamplingParams(**kinds[i % len(kinds)]) for i in range(B)]
    return {"kind": kind, "sampler": Sampler(DEVICE), "logits": logits, "params": params, "seeds": [seed * 64 + i for i in range(B)],
            "counters": list(range(B)), "none": [()] * B, "logprobs": case["logprobs"]}


@torch.no_grad()
def run(state: dict):
    kind = state["kind"]
    if kind == "step":
        runner = state["runner"]
        if state["decode"]:
            if runner.length(state["names"][0]) >= state["lengths"][0] + GROWTH:
                _seat(runner, state["names"], state["lengths"])
            return runner.step(state["entries"])
        logits = runner.step(state["entries"])
        for n in state["names"]:
            runner.release(n)
        return logits
    if kind == "sample":
        tokens, logprobs = state["sampler"](state["logits"], state["params"], state["none"], state["seeds"], state["counters"],
                                            state["logprobs"])
        return [tokens] if logprobs is None else [tokens, logprobs]
    if "graph" in state:
        state["graph"].replay()
        out = state["out"]
    else:
        out = state["call"]()
    if kind == "attention":
        return [out, *state["pages"]]
    if kind == "delta":
        return [out, *state["states"]]
    return out


# ----------------------------------------------------------------------------- what a pass cannot do without
def _seen(old: int, new: int) -> float:
    return new * old + new * (new + 1) / 2


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("step", "attention", "mlp"):
        H, I, NH, NKV, D = SIZES[case["size"]]
        att = (2 * NH + 2 * NKV) * D * H
        if kind == "mlp":
            T, n = case["tokens"], case["layers"]
            return {"bytes": n * (3 * H * I * 2 + T * H * 2) + T * H * 2, "flops": n * 6.0 * T * H * I}
        if kind == "attention":
            rows = _attention_work(case)
            T = sum(q for _, q in rows)
            kv = sum(n + 2 * q if n else q for n, q in rows) * 2 * NKV * D * 2
            return {"bytes": att * 2 + kv + 2 * T * H * 2, "flops": 2.0 * T * att + 4.0 * NH * D * sum(_seen(n, q) for n, q in rows)}
        size = 4 if case["dtype"] == "f32" else 2
        news = [1] * case["batch"] if case["new"] == 1 else _lengths(case["batch"], case["new"])
        olds = _lengths(case["batch"], case["context"]) if case["new"] == 1 else [0] * case["batch"]
        T, R, n = sum(news), case["batch"], case["layers"]
        per_layer = att + 3 * H * I
        kv = sum(o + q for o, q in zip(olds, news)) * 2 * NKV * D
        return {"bytes": n * (per_layer + kv) * size + VOCAB * H * size + T * H * size + R * VOCAB * 4,
                "flops": n * (2.0 * T * per_layer + 4.0 * NH * D * sum(_seen(o, q) for o, q in zip(olds, news))) + 2.0 * R * VOCAB * H}
    if kind == "moe":
        W, E, top, F = ZOGAPEL[case["size"]][:4]
        T = case["tokens"]
        active = E * (1.0 - (1.0 - top / E) ** T)
        return {"bytes": (active * 3 * F * W + E * W + 2 * T * W) * 2, "flops": T * (top * 6.0 * F * W + 2.0 * E * W)}
    if kind == "delta":
        W, _, _, _, NV, NK, D, DV, K = ZOGAPEL[case["size"]]
        B = case["batch"]
        T = B if case["new"] == 1 else sum(_lengths(B, case["new"]))
        weights = W * (2 * NK * D + 3 * NV * DV + 2 * NV)
        states = B * (NV * D * DV + K * (2 * NK * D + NV * DV)) * 4
        return {"bytes": weights * 2 + states * (2 if case["context"] else 1) + 2 * T * W * 2,
                "flops": 2.0 * T * weights + T * NV * D * DV * 7.0}
    return {"bytes": case["batch"] * (case["vocab"] * 4 + 40), "flops": case["batch"] * case["vocab"] * 4.0}


def tolerance(case: dict):
    kind = case["kind"]
    if kind == "sample":
        return {"rel": 1e-5, "max": 1e-3, "differ": 0.0}       # tokens are the same tokens; log probabilities are 32-bit sums
    if kind == "step":
        return {"rel": 2e-5, "max": 1e-3} if case["dtype"] == "f32" else {"rel": 2.5e-2}
    return {"rel": 1e-2}


# ----------------------------------------------------------------------------- the same in 64 bits
def _rms(x, w, offset=0.0):
    return x / (x * x).mean(-1, keepdim=True).add(EPS).sqrt() * (w.double() + offset)


def _rotate(x, positions):
    D = x.shape[-1]
    inv = THETA ** (-torch.arange(0, D, 2, device=DEVICE, dtype=torch.float64) / D)
    ang = positions.double()[:, None, None] * inv
    a, b = x[..., :D // 2], x[..., D // 2:]
    return torch.cat((a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()), -1)


def _attend(h, w, p, sizes, rows, kept):
    """The attention layer over requests that hold ``rows`` = (old, new) tokens; ``kept(r, n)``: the cache's rows."""
    H, _, NH, NKV, D = sizes
    q = _rms((h @ w[p + "q_proj.weight"].double().T).view(-1, NH, D), w[p + "q_norm.weight"])
    k = _rms((h @ w[p + "k_proj.weight"].double().T).view(-1, NKV, D), w[p + "k_norm.weight"])
    v = (h @ w[p + "v_proj.weight"].double().T).view(-1, NKV, D)
    out, at = torch.empty((h.shape[0], NH, D), device=DEVICE, dtype=torch.float64), 0
    for r, (old, new) in enumerate(rows):
        pos = torch.arange(old, old + new, device=DEVICE)
        qr, kr, vr = _rotate(q[at:at + new], pos), _rotate(k[at:at + new], pos), v[at:at + new]
        if old:
            k0, v0 = kept(r, old)
            kr, vr = torch.cat((k0.double(), kr)), torch.cat((v0.double(), vr))
        hidden = torch.arange(old + new, device=DEVICE)[None, :] > pos[:, None]
        for n in range(NKV):
            g = slice(n * (NH // NKV), (n + 1) * (NH // NKV))
            s = torch.einsum("qhd,kd->hqk", qr[:, g], kr[:, n]) * D ** -0.5
            out[at:at + new, g] = torch.einsum("hqk,kd->qhd", s.masked_fill(hidden, -math.inf).softmax(-1), vr[:, n])
        at += new
    return out.reshape(h.shape[0], NH * D) @ w[p + "o_proj.weight"].double().T


def _gated(h, w, p, gate="gate_proj.weight", up="up_proj.weight", down="down_proj.weight"):
    g = h @ w[p + gate].double().T
    return (g * torch.sigmoid(g) * (h @ w[p + up].double().T)) @ w[p + down].double().T


@torch.no_grad()
def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "step":
        w = _tensors(_qwen3_shapes(case, VOCAB), seed)
        ids = _ids(case, seed)
        olds = _lengths(case["batch"], case["context"]) if case["new"] == 1 else [0] * case["batch"]
        rows = [(o, len(i)) for o, i in zip(olds, ids)]
        x = w["model.embed_tokens.weight"][torch.tensor([t for i in ids for t in i], device=DEVICE)].double()
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            x = x + _attend(_rms(x, w[p + "input_layernorm.weight"]), w, p + "self_attn.", SIZES[case["size"]], rows,
                            lambda r, n: _context(case, seed, i, r, n))
            x = x + _gated(_rms(x, w[p + "post_attention_layernorm.weight"]), w, p + "mlp.")
        last = torch.tensor([len(i) for i in ids], device=DEVICE).cumsum(0) - 1
        return _rms(x[last], w["model.norm.weight"]) @ w["lm_head.weight"].double().T
    if kind == "attention":
        w = _tensors(_qwen3_shapes(case, 256), seed)
        rows = _attention_work(case)
        h = _tokens(case, seed, sum(q for _, q in rows), SIZES[case["size"]][0]).double()
        out = _attend(h, w, "model.layers.0.self_attn.", SIZES[case["size"]], rows, lambda r, n: _context(case, seed, 0, r, n))
        return [out, None, None]
    if kind == "mlp":
        w = _tensors(_qwen3_shapes(case, 256), seed)
        h = _tokens(case, seed, case["tokens"], SIZES[case["size"]][0]).double()
        return [_gated(h, w, f"model.layers.{i}.mlp.") for i in range(case["layers"])]
    if kind == "moe":
        W, E, top = ZOGAPEL[case["size"]][:3]
        w = _tensors(_zogapel_shapes(case), seed)
        h = _tokens(case, seed, case["tokens"], W).double()
        z, chosen = (h @ w["l0.mlp.router"].double().T + w["l0.mlp.router.b"].double()).topk(top, -1)
        share = z.softmax(-1)
        out = torch.zeros_like(h)
        for e in range(E):
            t, j = (chosen == e).nonzero(as_tuple=True)
            if len(t):
                out[t] += share[t, j, None] * _gated(h[t], w, f"l0.mlp.e{e}.", "gate", "up", "down")
        return [out]
    if kind == "delta":
        W, _, _, _, NV, NK, D, DV, K = ZOGAPEL[case["size"]]
        B = case["batch"]
        w = _tensors(_zogapel_shapes(case), seed)
        news = [1] * B if case["new"] == 1 else _lengths(B, case["new"])
        olds = _lengths(B, case["context"]) if case["context"] else [0] * B
        all_rows = _tokens(case, seed, sum(olds) + sum(news), W).double()
        old_rows, new_rows = all_rows[:sum(olds)].split(olds), all_rows[sum(olds):].split(news)
        m = "l0.mix."
        f = lambda name: w[m + name].double()
        longest = max(o + n for o, n in zip(olds, news))
        h = torch.zeros((B, longest, W), device=DEVICE, dtype=torch.float64)    # (a request's rows end it: zeros behind)
        for b in range(B):
            h[b, :olds[b] + news[b]] = torch.cat((old_rows[b], new_rows[b]))

        def conv(role):
            x = torch.nn.functional.pad(h @ f(role).T, (0, 0, K - 1, 0))
            y = sum(f(role + ".conv")[:, j] * x[:, j:j + longest] for j in range(K))
            return y * torch.sigmoid(y)

        unit = lambda x: x / ((x * x).sum(-1, keepdim=True) + 1e-6).sqrt()
        q = unit(conv("q").view(B, longest, NK, D)).repeat_interleave(NV // NK, 2) * D ** -0.5
        k = unit(conv("k").view(B, longest, NK, D)).repeat_interleave(NV // NK, 2)
        v = conv("v").view(B, longest, NV, DV)
        beta = torch.sigmoid(h @ f("b").T)
        decay = torch.exp(-f("A_log").exp() * torch.nn.functional.softplus(h @ f("a").T + f("dt_bias")))
        S = torch.zeros((B, NV, D, DV), device=DEVICE, dtype=torch.float64)
        o = torch.empty((B, longest, NV, DV), device=DEVICE, dtype=torch.float64)
        for t in range(longest):
            S = S * decay[:, t, :, None, None]
            u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None] @ S)[:, :, 0])
            S = S + k[:, t, :, :, None] * u[:, :, None]
            o[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
        gate = h @ f("g").T
        y = (_rms(o, w[m + "norm"]).reshape(B, longest, NV * DV) * gate * torch.sigmoid(gate)) @ f("o").T
        out = torch.cat([y[b, olds[b]:olds[b] + news[b]] for b in range(B)])
        return [out, None, None]
    return None
