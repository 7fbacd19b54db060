"""The calls that programs built on this library spend their time in, as cases that can be timed and compared.

step       one forward over a ragged batch through the C ABI (b2_model_step), as every serving and generation loop issues it: single
           tokens of running sequences, portions of prompts, or both packed together.  The model is a flat decoder with random
           group-quantized weights; the sequences' earlier tokens are in the page pool before the call, and are what is left
           in it after the call (the new positions are cut off again, as a verification step does).
generate   a model described layer by layer: prompts, then single tokens, each step with the logits of all sequences.
attention  the decode attention on its own, on pages that lie in any order.

Token ids come from the seed; feeding given ids keeps the work of a pass independent of which of two nearly equal logits is larger."""
import ctypes
import functools
import math

import numpy as np
import torch

from mlx_llm_b200 import _lib, engine, kernels, workloads

PAGE = 16
SHAPES = {"llama3_8b_q4": (workloads.LLAMA3_8B, 4), "qwen3_32b_q8": (workloads.QWEN3_32B, 8)}
DESIGNS = {"zukitar": lambda size, n: workloads.layered_config(size, n // 2), "tirezen": workloads.tirezen_config,
           "zokuzen": workloads.zokuzen_config, "pokadra": workloads.pokadra_config}


def listed():
    return [
        # one user and a chat model: nothing but the latency of a token
        _step("token_8b_q4_1", "llama3_8b_q4", 32, decode=1, lo=512, hi=768),
        # a handful of users, no prompt arriving
        _step("tokens_8b_q4_16", "llama3_8b_q4", 32, decode=16, lo=64, hi=1500),
        # a busy server between two prompts: contexts of very different lengths
        _step("tokens_8b_q4_64", "llama3_8b_q4", 32, decode=64, lo=32, hi=2048),
        # a loaded server's ordinary iteration: a 512-token portion of one prompt packed with everybody's next token
        _step("serve_8b_q4", "llama3_8b_q4", 32, decode=96, lo=32, hi=1300, portions=1, portion=512, cached=512),
        # prompts that arrive together and are taken whole, of a size that divides nothing
        _step("prompts_8b_q4", "llama3_8b_q4", 32, portions=3, portion=1049),
        # a portion far inside a long document; the large model, as many of its equal layers as keep the preparation short
        _step("document_32b_q8", "qwen3_32b_q8", 8, portions=1, portion=512, cached=11800),
        # a few long conversations with the large model
        _step("tokens_32b_q8_6", "qwen3_32b_q8", 8, decode=6, lo=2000, hi=9000),
        # the four layered designs, dense bf16: a long prompt alone, a few of middling length, many short ones
        _generate("zukitar_w4096", "zukitar", "w4096", seqs=4, prompt=520, tokens=8),
        _generate("tirezen_w2048", "tirezen", "w2048", seqs=16, prompt=150, tokens=16),
        _generate("zokuzen_w2048", "zokuzen", "w2048", seqs=8, prompt=260, tokens=12),
        _generate("pokadra_w4096", "pokadra", "w4096", seqs=1, prompt=1777, tokens=8),
        # the attention of a server that brings its own model code: the library's microbenchmark batch
        dict(name="attention_64", kind="attention", seqs=64, lo=128, hi=4096, hq=32, hkv=8, dim=128),
    ]


def _step(name, model, layers, decode=0, lo=0, hi=0, portions=0, portion=0, cached=0):
    return dict(name=name, kind="step", model=model, layers=layers, decode=decode, lo=lo, hi=hi, portions=portions, portion=portion, cached=cached)


def _generate(name, design, size, seqs, prompt, tokens):
    return dict(name=name, kind="generate", design=design, size=size, layers=8, seqs=seqs, prompt=prompt, tokens=tokens)


def _between(rng, lo, hi):
    """A whole number whose logarithm is spread evenly."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.99)))))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "generate", "generate", "attention"])
    if kind == "attention":
        hkv, group = rng.choice([1, 2, 4, 8]), rng.choice([1, 2, 4, 8])
        hi = _between(rng, 64, 4096)
        return dict(kind=kind, seqs=_between(rng, 1, 64), lo=_between(rng, 1, hi), hi=hi, hq=hkv * group, hkv=hkv, dim=rng.choice([64, 128]))
    if kind == "generate":
        seqs = _between(rng, 1, 16)
        case = _generate("", rng.choice(sorted(DESIGNS)), rng.choice(["w2048", "w4096"]), seqs, _between(rng, 2, 2400 // seqs), rng.randint(1, 16))
    else:
        small = rng.random() < 0.6
        model, layers = ("llama3_8b_q4", 32) if small else ("qwen3_32b_q8", 8)
        decode, portions = rng.choice([(1, 0), (0, 1), (1, 1)])
        decode *= _between(rng, 1, 96 if small else 12)
        hi = _between(rng, 64, min(2048 if small else 9000, 90000 // max(decode, 1)))
        portion = _between(rng, 2, 1500) * portions
        portions *= rng.randint(1, 2)
        case = _step("", model, layers, decode, min(hi, 16) if decode else 0, hi if decode else 0, portions, portion,
                     rng.choice([0, _between(rng, 16, 2048 if small else 11000)]) if portions else 0)
    del case["name"]
    return case


# ---- inputs ------------------------------------------------------------------------------------------------------------
@functools.lru_cache(None)
def _context():
    return _lib.Context(0)  # one per GPU and thread, as the library asks


class Served:
    """A model, its page pool and its caches, released together."""

    def __init__(self, model, tokens_per_seq):
        self.model = model
        blocks = [(t + PAGE - 1) // PAGE + 1 for t in tokens_per_seq]
        self.pool = engine.BlockPool(_context(), model, PAGE, sum(blocks), len(blocks), max(blocks))
        self.caches = [engine.PagedKvCache(self.pool) for _ in blocks]

    def __del__(self):
        for c in getattr(self, "caches", []):
            c.free()
        if hasattr(self, "pool"):
            self.pool.free()
        self.model.free()


class Call:
    """One b2_model_step call, with the buffers that a program keeps for it."""

    def __init__(self, model, ids, caches):
        rows, vocab = len(ids), model.config().vocab_size
        self.model, self.caches = model, caches
        self.ids = np.concatenate(ids).astype(np.int32)
        self.n = np.array([len(i) for i in ids], np.int32)
        self.handles = (ctypes.c_void_p * rows)(*[c.h for c in caches])
        self.logits = torch.empty((rows, vocab), dtype=torch.float32 if model.logits_f32() else torch.bfloat16, pin_memory=True)
        self.tokens = np.empty(rows, np.int32)
        self.args = (model.h, _lib.ptr(self.ids), _lib.ptr(self.n), rows, self.handles, _lib.ptr(self.logits.data_ptr()), _lib.ptr(self.tokens))

    def __call__(self):
        _lib.check(_lib.load().b2_model_step(*self.args))
        # the logits, and the logit of the token that the step picked
        return [self.logits, self.logits[torch.arange(len(self.tokens)), torch.from_numpy(self.tokens).long()]]


def _sequences(case, seed):
    """Token ids of every sequence: those in the cache already, and those of the step."""
    rng = np.random.default_rng(seed)
    vocab = SHAPES[case["model"]][0]["vocab_size"]
    have = list(rng.integers(case["lo"], case["hi"] + 1, case["decode"])) + [case["cached"]] * case["portions"]
    new = [1] * case["decode"] + [case["portion"]] * case["portions"]
    return [rng.integers(0, vocab, int(h)) for h in have], [rng.integers(0, vocab, n) for n in new]


def _prompts(case, seed):
    """Prompts from half to one and a half times the middling length, and the ids of every single-token step."""
    rng = np.random.default_rng(seed)
    n = case["seqs"]
    lengths = [max(2, case["prompt"] * (n + 2 * i + 1) // (2 * n)) for i in range(n)] if n > 1 else [case["prompt"]]
    vocab = _design(case)["vocab"]
    return [rng.integers(0, vocab, t) for t in lengths], rng.integers(0, vocab, (case["tokens"], n))


def _design(case):
    return DESIGNS[case["design"]](case["size"], case["layers"])


def prepare(case, seed):
    if case["kind"] == "attention":
        return _prepare_attention(case, seed)
    if case["kind"] == "generate":
        prompts, tokens = _prompts(case, seed)
        served = Served(engine.CausalLm.synthetic_json(_context(), _design(case), seed), [len(p) + len(tokens) for p in prompts])
        calls = [Call(served.model, prompts, served.caches)] + [Call(served.model, [t[i:i + 1] for i in range(len(t))], served.caches) for t in tokens]
        return dict(kind="generate", served=served, calls=calls)
    shape, bits = SHAPES[case["model"]]
    have, new = _sequences(case, seed)
    config = engine.model_config(**dict(shape, num_layers=case["layers"]), quant_bits=bits, quant_group=64)
    served = Served(engine.CausalLm.synthetic(_context(), config, seed), [len(h) + len(n) for h, n in zip(have, new)])
    todo = [[served.caches[i], h] for i, h in enumerate(have)]
    while any(len(h) for _, h in todo):  # the earlier tokens, a few thousand per forward
        room, seqs = 6144, []
        for t in todo:
            n = min(room, len(t[1]))
            if n:
                seqs.append((t[1][:n], t[0]))
                t[1] = t[1][n:]
                room -= n
        served.model.step_at(seqs, [[] for _ in seqs])
    return dict(kind="step", served=served, call=Call(served.model, new, served.caches), have=[len(h) for h in have])


def _prepare_attention(case, seed):
    rng = np.random.default_rng(seed)
    gen = torch.Generator("cuda").manual_seed(seed)
    ctx = rng.integers(case["lo"], case["hi"] + 1, case["seqs"])
    blocks = (ctx + PAGE - 1) // PAGE
    pages = 2 * int(blocks.sum())
    tables, order, at = np.zeros((len(ctx), int(blocks.max())), np.int32), rng.permutation(pages), 0
    for i, b in enumerate(blocks):
        tables[i, :b] = order[at:at + b]
        at += b
    normal = lambda *s: torch.randn(*s, generator=gen, device="cuda", dtype=torch.bfloat16)
    k, v = (normal(pages, case["hkv"], PAGE, case["dim"]) for _ in range(2))
    q = normal(len(ctx), case["hq"], case["dim"])
    return dict(kind="attention", case=case, k=k, v=v, q=q, out=torch.empty_like(q), lengths=ctx, tables=torch.from_numpy(tables).cuda(),
                ctx=torch.from_numpy(ctx.astype(np.int32)).cuda())


def run(state):
    if state["kind"] == "attention":
        c, p = state["case"], {n: state[n].data_ptr() for n in ("q", "k", "v", "tables", "ctx", "out")}
        kernels.paged_attn_decode(_context(), p["q"], p["k"], p["v"], p["tables"], p["ctx"], c["seqs"], c["hq"], c["hkv"], c["dim"], PAGE,
                                  c["dim"] ** -0.5, p["out"], state["tables"].shape[1])
        return state["out"]
    if state["kind"] == "generate":
        for c in state["served"].caches:
            c.reset()
        return [call() for call in state["calls"]]
    out = state["call"]()
    for cache, n in zip(state["served"].caches, state["have"]):
        cache.truncate(n)
    return out


# ---- work and tolerance ------------------------------------------------------------------------------------------------
def _pairs(have, new):
    """(query, visible key) pairs of `new` tokens behind `have` ones."""
    return new * have + new * (new + 1) / 2


def work(case):
    if case["kind"] == "attention":
        keys = case["seqs"] * (case["lo"] + case["hi"]) / 2
        return {"bytes": 2 * (2 * keys * case["hkv"] + 2 * case["seqs"] * case["hq"]) * case["dim"], "flops": 4 * keys * case["hq"] * case["dim"]}
    if case["kind"] == "generate":
        return _work_generate(case)
    shape, bits = SHAPES[case["model"]]
    shape = dict(shape, num_layers=case["layers"])
    rows, tokens = case["decode"] + case["portions"], case["decode"] + case["portions"] * case["portion"]
    cached = case["decode"] * (case["lo"] + case["hi"]) / 2 + case["portions"] * case["cached"]
    pairs = case["decode"] * _pairs((case["lo"] + case["hi"]) / 2, 1) + case["portions"] * _pairs(case["cached"], case["portion"])
    head = shape["vocab_size"] * shape["hidden_size"]
    return {"bytes": workloads.step_weight_bytes(shape, bits) + workloads.kv_bytes_per_token(shape) * (cached + tokens)
            + 2 * shape["hidden_size"] * tokens + 2 * rows * shape["vocab_size"],
            "flops": 2.0 * workloads.projection_params(shape) * tokens + 2.0 * head * rows
            + 4.0 * pairs * shape["num_layers"] * shape["num_heads"] * shape["head_dim"]}


def _work_generate(case):
    """Weights: everything a token passes through, of the experts those that a step's tokens can reach; caches and states once per step."""
    cfg, (prompts, steps) = _design(case), _prompts(case, 0)
    w = cfg["width"]
    lengths = [len(p) for p in prompts]
    work = {"bytes": 0.0, "flops": 0.0}
    for at in range(len(steps) + 1):
        tokens = sum(lengths) if at == 0 else len(lengths)
        weights = flops = 0.0
        moved = 4.0 * len(lengths) * cfg["vocab"] + 2.0 * tokens * w
        for layer in cfg["layers"]:
            for kind, m in _mixers(layer):
                params, pair, row, state = _mixer_sizes(kind, m, w)
                weights += params
                flops += 2.0 * params * tokens + 6.0 * state * tokens
                moved += 8.0 * state * len(lengths)
                for t in lengths:
                    flops += pair * (_pairs(0, t) if at == 0 else t + at)
                    moved += 2.0 * row * (t + at)
            mlp = layer["mlp"]
            if mlp["kind"] == "dense":
                dense, one, experts, top = (2 if "limit" not in mlp and cfg["architecture"] == "Tirezen" else 3) * w * mlp["ff"], 0, 0, 0
            else:
                dense, one = w * mlp["router"]["experts"] + 3 * w * mlp.get("shared", {}).get("ff", 0), 3 * w * mlp["expert"]["ff"]
                experts, top = mlp["router"]["experts"], mlp["router"]["top"]
            weights += dense + one * min(experts, top * tokens)
            flops += 2.0 * (dense + top * one) * tokens
        head = cfg["vocab"] * w
        work["bytes"] += 2.0 * (weights + head) + moved
        work["flops"] += flops + 2.0 * head * len(lengths)
    return work


def _mixers(layer):
    m = layer["mixer"]
    return [("attention", m["left"]), ("memory", m["right"])] if layer["type"] == "parallel" else [(layer["type"], m)]


def _mixer_sizes(kind, m, w):
    """Weights, flops per (query, key) pair, cached values per token, values of the recurrent state."""
    if kind == "latent_attention":
        dim, rot = m["dim"], m.get("rot_dim", 0)
        params = w * (m["heads"] * (dim + rot) + m["kv_rank"] + rot) + m["heads"] * (dim + m["vdim"]) * m["kv_rank"] + w * m["heads"] * m["vdim"]
        return params, 2 * m["heads"] * (dim + rot + m["vdim"]), m["kv_rank"] + rot, 0
    if kind == "attention":
        maps = 2 if "diff" in m else 1
        own = 0 if "kv_from" in m else m["kv_heads"] * (maps * m["dim"] + m["vdim"])
        return (w * (m["heads"] * (maps * m["dim"] + m["vdim"]) + own), 2 * maps * m["heads"] * (m["dim"] + m["vdim"]),
                m["kv_heads"] * (maps * m["dim"] + m["vdim"]), 0)
    if kind == "mamba2":
        inner, bc = m["heads"] * m["vdim"], 2 * m["groups"] * m["state"]
        return w * (3 * inner + bc + m["heads"]), 0, 0, inner * m["state"]
    if kind == "mingru":
        return 4 * w * m["width"], 0, 0, m["width"]
    keys, values = m.get("kv_heads", m["heads"]) * m["dim"], m["heads"] * m.get("vdim", m["dim"])
    return w * (2 * keys + 3 * values), 0, 0, values * m["dim"]


def tolerance(case):
    # About four times what was measured.  Against `exact`: 0.0017 for the attention, 0.0077 and 0.021 for the flat models (bf16
    # activations through all layers), 0.0083 for the layered designs with dense feed-forwards.  With routed experts rounding decides
    # which of two nearly equal experts a token gets: two orders of summation differ by 0.02 to 0.27 from step to step.
    if case["kind"] == "attention":
        return {"rel": 7e-3}
    if case["kind"] == "generate":
        return {"rel": 0.7 if case["design"] in ("zukitar", "zokuzen") else 0.033}
    return {"rel": 0.03 if case["model"] == "llama3_8b_q4" else 0.08}


# ---- what 64-bit arithmetic gives ----------------------------------------------------------------------------------------
MASK = (1 << 64) - 1
GOLD = 0x9E3779B97F4A7C15


def _signed(v):
    v &= MASK
    return v - (1 << 64) if v >> 63 else v


def _shift(z, n):
    return (z >> n) & ((1 << (64 - n)) - 1)


def _mix(z):
    """The finaliser of SplitMix64 on a tensor of 64-bit words."""
    z = (z ^ _shift(z, 30)) * _signed(0xBF58476D1CE4E5B9)
    z = (z ^ _shift(z, 27)) * _signed(0x94D049BB133111EB)
    return z ^ _shift(z, 31)


def _word(seed, index):
    return _mix(index * _signed(GOLD) + _signed(seed + GOLD))


def _mix_int(z):
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9 & MASK
    z = (z ^ (z >> 27)) * 0x94D049BB133111EB & MASK
    return z ^ (z >> 31)


def _fields(words):
    return sum(_shift(words, 16 * i) & 0xffff for i in range(4))


def _bf16(x):
    return x.to(torch.bfloat16)


class Drawn:
    """The random weights of a flat model, drawn as the library documents them: twelve 16-bit uniforms per normal value."""

    def __init__(self, shape, bits, seed):
        self.shape, self.bits, self.seed = shape, bits, seed

    def _seed(self, layer, which):
        return _mix_int(self.seed ^ (0x5EED0000 + {7: 1, 8: 2}.get(which, 16 * (layer + 1) + which)))

    def _normal(self, seed, index):
        return (sum(_fields(_word(seed, 3 * index + i)) for i in range(3)).float() - 393210.0) * (1.0 / 65536.0)

    def rows(self, which, index):
        """Rows of the embedding (7) or the head (8)."""
        cols = torch.arange(self.shape["hidden_size"], device="cuda")
        return _bf16(self._normal(self._seed(0, which), index[:, None] * len(cols) + cols) * 0.02).double()

    def projection(self, layer, which, n, k):
        seed, dev = self._seed(layer, which), dict(device="cuda")
        group = torch.arange(n * k // 64, **dev)
        mul, mid = (0.02 / 7.5, 8.0) if self.bits == 4 else (0.02 / 127.5, 128.0)
        scale = _bf16(self._normal(seed + 1, group).abs() * np.float32(mul).item())
        bias = _bf16((self._normal(seed + 2, group).double() * np.float32(1e-3).item() - mid * scale.double()).float())
        words = _shift(_word(seed, torch.arange(n * k * self.bits // 32, **dev)), 16)
        code = (words[:, None] >> torch.arange(0, 32, self.bits, **dev)) & ((1 << self.bits) - 1)
        w = code.view(-1, 64).float() * scale.float()[:, None] + bias.float()[:, None]
        return _bf16(w).double().view(n, k)


def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _turn_halves(x, pos, freq):
    """x [..., tokens, dims]: coordinates i and i + dims / 2 turned by pos * freq[i]."""
    a = pos.double()[:, None] * freq
    x1, x2 = x.chunk(2, -1)
    return torch.cat([x1 * a.cos() - x2 * a.sin(), x2 * a.cos() + x1 * a.sin()], -1)


def _frequencies(shape):
    f = shape["rope_theta"] ** (-torch.arange(0, shape["head_dim"], 2, dtype=torch.float64, device="cuda") / shape["head_dim"])
    if shape["rope_kind"] == 1:
        wave, original = 2 * math.pi / f, shape["rope_original_context"]
        low, high = shape["rope_low_freq_factor"], shape["rope_high_freq_factor"]
        smooth = ((original / wave - low) / (high - low)).clamp(0, 1)
        f = torch.where(wave > original / low, f / shape["rope_factor"], torch.where(wave < original / high, f, (1 - smooth) * f / shape["rope_factor"] + smooth * f))
    return f


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "attention":
            return _exact_attention(case, seed)
        if case["kind"] == "generate":
            # with routed experts the result jumps where rounding decides who is routed where: 64 bits are no yardstick there
            return {"tirezen": _exact_tirezen, "pokadra": _exact_pokadra}[case["design"]](case, seed) if case["design"] in ("tirezen", "pokadra") else None
        return _exact_step(case, seed)


def _exact_attention(case, seed):
    s = _prepare_attention(case, seed)
    out, group = torch.zeros_like(s["q"], dtype=torch.float64), case["hq"] // case["hkv"]
    for i, n in enumerate(s["lengths"]):
        at = torch.arange(int(n), device="cuda")
        page = s["tables"][i].long()[at // PAGE]
        k, v = (s[x][page, :, at % PAGE].double().repeat_interleave(group, 1) for x in "kv")
        p = torch.softmax(torch.einsum("hd,thd->ht", s["q"][i].double(), k) * case["dim"] ** -0.5, -1)
        out[i] = torch.einsum("ht,thd->hd", p, v)
    return out


def _exact_step(case, seed):
    shape, bits = SHAPES[case["model"]]
    shape = dict(shape, num_layers=case["layers"])
    have, new = _sequences(case, seed)
    ids = [torch.from_numpy(np.concatenate(p)).cuda() for p in zip(have, new)]
    if 2.0 * workloads.projection_params(shape) * sum(len(i) for i in ids) > 2.5e14:
        return None  # more than about twenty seconds
    w, eps = Drawn(shape, bits, seed), shape["rms_norm_eps"]
    H, hq, hkv, d, ff = (shape[n] for n in ("hidden_size", "num_heads", "num_kv_heads", "head_dim", "intermediate_size"))
    freq, split = _frequencies(shape), [len(i) for i in ids]
    x = w.rows(7, torch.cat(ids))
    for l in range(case["layers"]):
        h = _rms(x, eps)
        q, k, v = (h @ w.projection(l, i, n * d, H).T for i, n in enumerate((hq, hkv, hkv)))
        a = torch.empty_like(q)
        at = 0
        for n in split:
            rows, pos = slice(at, at + n), torch.arange(n, device="cuda")
            at += n
            part = lambda t, heads: t[rows].view(n, heads, d).transpose(0, 1)
            normed = (lambda t: _rms(t, eps)) if shape["qk_norm"] else (lambda t: t)
            qs, ks, vs = _turn_halves(normed(part(q, hq)), pos, freq), _turn_halves(normed(part(k, hkv)), pos, freq), part(v, hkv)
            for i in range(hq):
                for r in range(0, n, 4096):  # (scores of a few thousand queries at a time)
                    top = min(n, r + 4096)
                    s = (qs[i, r:top] @ ks[i * hkv // hq, :top].T) * d ** -0.5
                    s.masked_fill_(pos[None, :top] > pos[r:top, None], -math.inf)
                    a[at - n + r:at - n + top, i * d:(i + 1) * d] = torch.softmax(s, -1) @ vs[i * hkv // hq, :top]
        x = x + a @ w.projection(l, 3, H, hq * d).T
        h = _rms(x, eps)
        act = torch.nn.functional.silu(h @ w.projection(l, 4, ff, H).T) * (h @ w.projection(l, 5, ff, H).T)
        x = x + act @ w.projection(l, 6, H, ff).T
    last = _rms(x[torch.tensor(split, device="cuda").cumsum(0) - 1], eps)
    step = 16384
    logits = torch.cat([last @ w.rows(8, torch.arange(r, min(r + step, shape["vocab_size"]), device="cuda")).T for r in range(0, shape["vocab_size"], step)], 1)
    return [logits, logits.max(-1).values]


class Filled:
    """The random weights of a layered model: every tensor in turn takes the next seed; four 16-bit uniforms per value."""

    def __init__(self, seed):
        self.seed = seed

    def vector(self, *shape, mean=1.0, sd=0.0):
        self.seed += 1
        words = _word(self.seed * GOLD, torch.arange(math.prod(shape), device="cuda"))
        return (mean + np.float32(sd).item() * (_fields(words).float() - 131070.0) * np.float32(1 / 37837.2).item()).view(shape).double()

    def matrix(self, rows, cols):
        return _bf16(self.vector(rows, cols, mean=0.0, sd=1.0 / math.sqrt(cols)).float()).double()


def _batch(case, seed):
    """All sequences side by side, padded at the end: ids [sequences, tokens], and the places whose logits a pass returns, step by step."""
    prompts, steps = _prompts(case, seed)
    lengths = [len(p) for p in prompts]
    ids = torch.zeros(len(prompts), max(lengths) + len(steps), dtype=torch.int64)
    for i, p in enumerate(prompts):
        ids[i, :lengths[i] + len(steps)] = torch.from_numpy(np.concatenate([p, steps[:, i]]))
    return ids.cuda(), [torch.tensor([n - 1 + t for n in lengths], device="cuda") for t in range(len(steps) + 1)]


def _logits(x, head, places):
    out = []
    for at in places:
        z = x[torch.arange(len(x), device="cuda"), at] @ head.T
        out.append([z, z.max(-1).values])
    return out


def _heads(x, n):
    """[sequences, tokens, n * d] -> [sequences, n, tokens, d]"""
    return x.view(x.shape[0], x.shape[1], n, -1).transpose(1, 2)


def _flat(x):
    return x.transpose(1, 2).flatten(2)


def _attend(q, k, v, scale, cap=0.0, sink=False):
    """q [S, H, T, D], k and v [S, G, T, .]: softmax attention over earlier and equal places; a sink is one more term exp(0)."""
    T, out = q.shape[2], torch.empty(*q.shape[:3], v.shape[3], dtype=q.dtype, device=q.device)
    later = torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1)
    for h in range(q.shape[1]):
        g = h * k.shape[1] // q.shape[1]
        s = q[:, h] @ k[:, g].transpose(1, 2) * scale
        s = (cap * torch.tanh(s / cap) if cap else s).masked_fill_(later, -math.inf)
        top = s.amax(-1, keepdim=True).clamp(min=0.0 if sink else -math.inf)
        e = torch.exp(s - top)
        out[:, h] = e @ v[:, g] / (e.sum(-1, keepdim=True) + (torch.exp(-top) if sink else 0.0))
    return out


def _remember(q, k, v, decay, beta=None):
    """q, k, decay [S, H, T, D], v [S, H, T, V]: a matrix per head that fades and takes up k v^T, or with beta the delta rule."""
    S, out = torch.zeros(*k.shape[:2], k.shape[3], v.shape[3], dtype=q.dtype, device=q.device), torch.empty_like(v)
    for t in range(k.shape[2]):
        S = decay[:, :, t, :, None] * S
        u = v[:, :, t] if beta is None else beta[:, :, t, None] * (v[:, :, t] - torch.einsum("shd,shdv->shv", k[:, :, t], S))
        S = S + k[:, :, t, :, None] * u[:, :, None]
        out[:, :, t] = torch.einsum("shd,shdv->shv", q[:, :, t], S)
    return out


def _exact_tirezen(case, seed):
    cfg, f = _design(case), Filled(seed)
    ids, places = _batch(case, seed)
    W, eps, silu, sig = cfg["width"], cfg["norm"]["eps"], torch.nn.functional.silu, torch.sigmoid
    pos = torch.arange(ids.shape[1], device="cuda")
    base = lambda m: m["rot"]["base"] ** (-torch.arange(0, m["rot"]["dims"], 2, dtype=torch.float64, device="cuda") / m["rot"]["dims"])
    embed, head = f.matrix(cfg["vocab"], W), f.matrix(cfg["vocab"], W)
    x = embed[ids]
    for layer in cfg["layers"]:
        f.vector(W)
        h, m, ff = _rms(x, eps), layer["mixer"], layer["mlp"]["ff"]
        if layer["type"] == "parallel":
            a = m["left"]
            sizes = (a["heads"], a["dim"]), (a["kv_heads"], a["dim"]), (a["kv_heads"], a["vdim"])
            qkv = [h @ f.matrix(n * d, W).T for n, d in sizes]
            q, k, v = (_heads(t + f.vector(n * d, mean=0.0, sd=0.1), n) for t, (n, d) in zip(qkv, sizes))
            f.vector(a["dim"]), f.vector(a["dim"])
            q, k = (_turn_halves(_rms(t, eps), pos, base(a)) for t in (q, k))
            left = _flat(_attend(q, k, v, a["scale"], a["softcap"], True))
            m = m["right"]
        H, G, D, V = m["heads"], m.get("kv_heads", m["heads"]), m["dim"], m["vdim"]
        q, k, v = (h @ f.matrix(n, W).T for n in (G * D, G * D, H * V))
        if layer["type"] == "retention":
            q, k = (_turn_halves(_heads(t, H), pos, base(m)) for t in (q, k))
            o = _remember(q, k * D ** -0.5, _heads(v, H), torch.tensor(m["decay"], dtype=torch.float64, device="cuda")[None, :, None, None].expand(len(ids), H, len(pos), D))
            o = _flat(_rms(o, eps)) * silu(h @ f.matrix(H * V, W).T)
        else:
            conv, qkv = f.vector(m["conv"], 2 * G * D + H * V, mean=0.0, sd=0.5), torch.cat([q, k, v], -1)
            qkv = silu(sum(torch.nn.functional.pad(qkv, (0, 0, m["conv"] - 1 - j, 0))[:, :len(pos)] * conv[j] for j in range(m["conv"])))
            unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)
            q, k, v = qkv.split([G * D, G * D, H * V], -1)
            q, k, v = unit(_heads(q, G)).repeat_interleave(H // G, 1) * D ** -0.5, unit(_heads(k, G)).repeat_interleave(H // G, 1), _heads(v, H)
            if layer["type"] == "parallel":
                r = max(8, min(D, V))
                a1, g1, a2, g2, b = f.matrix(r, W), f.matrix(r, W), f.matrix(H * D, r), f.matrix(V * H, r), f.matrix(H, W)
                step, gate = h @ a1.T @ a2.T, sig(h @ g1.T @ g2.T)
            else:
                g, a, b = f.matrix(H * V, W), f.matrix(H, W), f.matrix(H, W)
                step, gate = h @ a.T, silu(h @ g.T)
            step = _heads(torch.nn.functional.softplus(step + f.vector(step.shape[-1], mean=-3.0, sd=1.0)), H)
            decay = torch.exp(-torch.exp(f.vector(H, sd=0.7))[None, :, None, None] * step).expand(-1, -1, -1, D)
            o = _remember(q, k, v, decay, _heads(sig(h @ b.T), H)[..., 0])
            f.vector(V)
            o = _flat(_rms(o, eps)) * gate
        if layer["type"] == "parallel":
            y = layer["mixer"]["left_scale"] * left @ f.matrix(W, left.shape[-1]).T + layer["mixer"]["right_scale"] * o @ f.matrix(W, H * V).T
        else:
            y = o @ f.matrix(W, H * V).T
        up, down = f.matrix(ff, W), f.matrix(W, ff)
        x = x + y + torch.nn.functional.gelu(h @ up.T) @ down.T
    return _logits(_rms(x, eps), head, places)


def _turn_pairs(x, pos, rot):
    """x [..., tokens, dims]: neighbours turned by frequencies that are interpolated for the slow pairs, everything grown a little."""
    n, s = rot["dims"], rot["scaling"]
    f = rot["base"] ** (-torch.arange(0, n, 2, dtype=torch.float64, device="cuda") / n)
    place = lambda turns: n * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(rot["base"]))
    lo, hi = max(math.floor(place(s["fast"])), 0), min(math.ceil(place(s["slow"])), n - 1)
    ramp = ((torch.arange(n // 2, device="cuda").double() - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    a, grow = pos.double()[:, None] * (f / s["factor"] * ramp + f * (1 - ramp)), 0.1 * math.log(s["factor"]) + 1.0
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1).flatten(-2) * grow


def _exact_pokadra(case, seed):
    cfg, f = _design(case), Filled(seed)
    ids, places = _batch(case, seed)
    W, V, n = cfg["width"], cfg["vocab"], cfg["token_side"]["dim"]
    eps, groups, mult, pairs = cfg["norm"]["eps"], cfg["norm"]["groups"], cfg["residual_mult"], cfg["embedding"]["bigram"]
    silu, sig, pos = torch.nn.functional.silu, torch.sigmoid, torch.arange(ids.shape[1], device="cuda")
    group_norm = lambda t: _rms(t.unflatten(-1, (groups, -1)), eps).flatten(-2)
    embed, head, table, side = f.matrix(V, W), f.matrix(V, W), f.matrix(pairs["buckets"] + 1, W), f.matrix(V, n * len(cfg["layers"]))
    at = torch.cat([torch.full_like(ids[:, :1], pairs["buckets"]), (ids[:, :-1] * pairs["mul_prev"] + ids[:, 1:] * pairs["mul_cur"]) % pairs["buckets"]], 1)
    x = embed[ids] * cfg["embedding"]["scale"] + table[at]
    before, stored = [x], {}
    assert ids.shape[1] <= cfg["layers"][0]["mixer"]["mask"]["size"]  # everything earlier is visible
    for i, layer in enumerate(cfg["layers"]):
        f.vector(W)
        side_gate, side_proj = f.matrix(n, W), f.matrix(W, n)
        f.vector(W)
        weights = f.vector(i + 2, mean=np.float32(1.0 / (i + 2)).item())
        m = layer["mixer"]
        if layer["type"] == "mingru":
            z, u, g = (x @ f.matrix(m["width"], W).T for _ in range(3))
            z = sig(z - 1.0 - 5.0 * torch.arange(m["width"], device="cuda") / m["width"])
            c, S, a = torch.where(u >= 0, u + 0.5, sig(u)), torch.zeros_like(u[:, 0]), torch.empty_like(u)
            for t in range(len(pos)):
                S = (1.0 - z[:, t]) * S + z[:, t] * c[:, t]
                a[:, t] = S
            y = a * silu(g)
        else:
            H, G, D, own = m["heads"], m["kv_heads"], m["dim"], "kv_from" not in m
            maps = lambda t, heads: _turn_pairs(_rms(_heads(t, 2 * heads), eps), pos, m["rot"]).unflatten(1, (heads, 2))
            q = maps(x @ f.matrix(2 * H * D, W).T, H)
            if own:
                k = x @ f.matrix(2 * G * D, W).T
                stored[i] = maps(k, G), _heads(x @ f.matrix(G * m["vdim"], W).T, G)
            k, v = stored[i if own else m["kv_from"]]
            gate = sig(x @ f.matrix(H, W).T)
            for _ in range(2 if own else 1):
                f.vector(D)
            o = _attend(q[:, :, 0], k[:, :, 0], v, m["scale"]) - m["diff"] * _attend(q[:, :, 1], k[:, :, 1], v, m["scale"])
            y = _flat(_rms(o, eps) * (1.0 - m["diff"]) * gate.transpose(1, 2)[..., None])
        x = x + mult * group_norm(y @ f.matrix(W, y.shape[-1]).T)
        f.vector(W)
        ff, limit = layer["mlp"]["ff"], layer["mlp"]["limit"]
        a, u = (x @ f.matrix(ff, W).T).clamp(max=limit), (x @ f.matrix(ff, W).T).clamp(-limit, limit)
        x = x + mult * group_norm((a * sig(1.702 * a) * (u + 1.0)) @ f.matrix(W, ff).T)
        e = side[ids][..., i * n:(i + 1) * n]
        x = x + mult * _rms((torch.nn.functional.gelu(x @ side_gate.T, approximate="tanh") * e) @ side_proj.T, eps)
        before.append(x)
        x = sum(c * t for c, t in zip(weights, before))
    return _logits(group_norm(x), head, places)
