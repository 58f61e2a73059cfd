"""What users of the library have it do, as cases that can be timed and compared.

Three kinds of work, all through the public entry points:

``serve``   requests from their first token on: ``Engine.open``, one ``Engine.step`` with all prompts, then ``steps`` tokens a
            sequence through ``Engine.decode_session`` (none: a prompt alone), ``Engine.close``.  Every step's logits come back.
``decode``  sequences that already stand in the cache go on for ``steps`` tokens; afterwards ``Engine.truncate`` rewinds them.
``sample``  one token per row of given logits by ``sampling.sample_rows``.

The tokens that are fed back are given and not picked from the logits (``DecodeSession.feed``, as sampling on the device feeds
them), so that two implementations that round differently run the same tokens.  Weights are random, of the sizes in
``config.presets`` for the Llama-family decoder and of the benchmark's 2,048-wide sizes for the Nikodra and Soporax decoders.
Decoders whose experts are picked by computed scores are left out: a near tie that rounds the other way sends a token through
other experts, and two correct implementations are then further apart than any useful bound.  Soporax picks by a table.

``exact`` restates the decoders in float64 on whole sequences, without a cache and without the library's code.
"""
from __future__ import annotations

import math
import zlib

import numpy as np
import torch

F64 = torch.float64
DESIGNS = ("nikodra-w2048", "soporax-w2048")


def listed():
    return [
        # a short chat turn on the smallest model: every launch counts
        dict(name="chat-05b", kind="serve", model="minicpm4-0.5b", dtype="bfloat16", rows=1, low=37, high=37, steps=16),
        # one user's decoding at a short context: weights streamed once a token
        dict(name="decode-2b-b1", kind="decode", model="minicpm-2b", dtype="bfloat16", rows=1, low=128, high=128, steps=8),
        # the benchmark's headline: weights and a long cache
        dict(name="decode-2b-b8", kind="decode", model="minicpm-2b", dtype="bfloat16", rows=8, low=4096, high=4096, steps=4),
        # a busy server: a full batch of unequal contexts, sixteen query heads on a key/value head
        dict(name="decode-8b-b64", kind="decode", model="minicpm4-8b", dtype="bfloat16", rows=64, low=200, high=520, steps=4),
        # the benchmark's prompt
        dict(name="prompt-2b-2048", kind="serve", model="minicpm-2b", dtype="bfloat16", rows=1, low=2048, high=2048, steps=0),
        # a full batch of unequal prompts in one step
        dict(name="prompts-05b-64", kind="serve", model="minicpm4-0.5b", dtype="bfloat16", rows=64, low=16, high=2048, steps=0),
        # a question of a few lines on a large model, and the first tokens of its answer
        dict(name="chat-8b", kind="serve", model="llama-8b-like", dtype="bfloat16", rows=1, low=181, high=181, steps=4),
        # a long document
        dict(name="prompt-8b-6145", kind="serve", model="llama-8b-like", dtype="bfloat16", rows=1, low=6145, high=6145, steps=0),
        # the true 32-bit path, as replays and comparisons use it
        dict(name="float32-05b", kind="serve", model="minicpm4-0.5b", dtype="float32", rows=3, low=90, high=300, steps=4),
        # a batch's sampling with everything a chat front end sets
        dict(name="sample-32", kind="sample", rows=32, vocab=122753, top_k=50, top_p=0.95, min_p=0.02, penalties=True),
        # recurrences and attention side by side: prompts and decoding of a batch
        dict(name="nikodra-b8", kind="serve", model="nikodra-w2048", dtype="bfloat16", rows=8, low=120, high=520, steps=8),
        # latent attention, windows, gates and experts: one longer prompt and decoding
        dict(name="soporax-b2", kind="serve", model="soporax-w2048", dtype="bfloat16", rows=2, low=700, high=1300, steps=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.random()
    if what < 0.15:
        return dict(kind="sample", rows=_log_int(rng, 1, 64), vocab=rng.choice([32000, 73448, 122753, 128256]),
                    top_k=rng.choice([0, 20, 50, 200]), top_p=rng.choice([1.0, 0.9, 0.95]), min_p=rng.choice([0.0, 0.05]),
                    penalties=rng.random() < 0.5)
    if what < 0.45:
        model = rng.choice(["minicpm-2b", "minicpm4-0.5b", "minicpm4-8b", "llama-8b-like"])
        rows = _log_int(rng, 1, 64)
        # at most some 24,000 tokens of context in all: they are put there by real steps
        high = _log_int(rng, 40, max(41, min(4096, 24000 // rows)))
        return dict(kind="decode", model=model, dtype="bfloat16", rows=rows, low=max(1, int(high * rng.uniform(0.3, 1.0))), high=high,
                    steps=rng.randint(2, 8))
    if what < 0.7:
        model, dtype = rng.choice([("minicpm-2b", "bfloat16"), ("minicpm4-0.5b", "bfloat16"), ("minicpm4-8b", "bfloat16"),
                                   ("llama-8b-like", "bfloat16"), ("minicpm4-0.5b", "float32")])
        most = 900 if dtype == "float32" else 5000              # tokens of all prompts together
    else:
        model, dtype, most = rng.choice(["minicpm4-0.5b", *DESIGNS]), "bfloat16", 5000
    rows = _log_int(rng, 1, 32)
    high = _log_int(rng, 16, max(17, min(4096, most // rows)))
    return dict(kind="serve", model=model, dtype=dtype, rows=rows, low=max(1, int(high * rng.uniform(0.1, 1.0))), high=high,
                steps=rng.choice([0, 1, 3, 8]))


# -- configurations -----------------------------------------------------------

def _nikodra():
    width, heads, hd = 2048, 16, 128
    att = {"heads": heads, "kv_heads": heads, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "v_mix": True,
           "rot": {"base": 500000.0, "dims": hd, "scaling": {"factor": 8.0, "original": 4096, "fast": 16.0, "slow": 2.0}}}
    left = {"heads": heads, "kv_heads": heads, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "mask": {"size": 1024}}
    right = {"heads": heads, "dim": 64, "vdim": hd, "decay": [1.0 - 2.0 ** (-4.0 - 6.0 * i / heads) for i in range(heads)],
             "rot": {"base": 10000.0, "dims": 64}}
    kinds = [("attention", att), ("attention", att), ("parallel", {"left": left, "right": right}),
             ("wkv", {"heads": width // 64, "dim": 64, "decay_rank": 64})]
    return dict(vocab=32000, width=width, norm_eps=1e-6, residual_mult=0.5, bigram={"buckets": 65521, "mul_prev": 1000003, "mul_cur": 31},
                layers=[(kinds[i % 4][0], kinds[i % 4][1], {"kind": "dense", "ff": 5632}) for i in range(8)])


def _soporax():
    heads, hd = 16, 128
    plain = {"heads": heads, "kv_heads": heads, "dim": hd, "vdim": hd, "scale": hd ** -0.5}
    latent = dict(heads=heads, dim=128, rot_dim=64, vdim=128, q_rank=768, kv_rank=512, scale=192 ** -0.5,
                  rot={"base": 10000.0, "dims": 64, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}})
    rot = {"base": 500000.0, "dims": hd, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}
    moe = {"kind": "moe", "expert": {"ff": 1408}, "router": {"experts": 16, "top": 2}}
    kinds = [("latent_attention", latent, {"kind": "dense", "ff": 5632, "limit": 7.0}),
             ("attention", dict(plain, mask={"size": 1024}), moe), ("attention_2", dict(plain, rot=rot), moe)]
    return dict(vocab=32000, width=2048, norm_eps=1e-6, logit_scale=0.5, loop={"start": 1, "stop": 3, "times": 2},
                layers=[kinds[i % 3] for i in range(6)])


def _plan(model):
    import exl3_server_b200 as E
    from exl3_server_b200.config import presets
    from exl3_server_b200.config.nikodra import NikodraLayer
    from exl3_server_b200.config.soporax import SoporaxLayer
    if model == "nikodra-w2048":
        c = _nikodra()
        cfg = E.NikodraConfig(**{**c, "layers": [NikodraLayer(k, dict(m), dict(f)) for k, m, f in c["layers"]]})
    elif model == "soporax-w2048":
        c = _soporax()
        cfg = E.SoporaxConfig(**{**c, "layers": [SoporaxLayer(k, dict(m), dict(f)) for k, m, f in c["layers"]]})
    else:
        cfg = E.LlamaConfig(**presets.sizes(model))
    return E.resolve_architecture(cfg.to_dict()).build_plan(cfg)


class _Weights:
    """Random tensors by name: matrices N(0, 0.02), norm weights near what norms are trained to.  As in trained models no
    sublayer outweighs the residual that it joins: the Llama-family's projections into it are N(0, 0.0025), and embeddings
    without a factor of their own have the size of the sublayers' outputs.  (With N(0, 0.02) everywhere the wider models
    amplify rounding from layer to layer, to 5 % of the logits after 32.)"""

    def __init__(self, model, dtype, seed):
        self.model, self.seed = model, seed
        self.dtype = torch.float32 if dtype == "float32" else torch.bfloat16

    def __call__(self, name, shape, high=0):
        g = torch.Generator(device="cuda").manual_seed((self.seed << 32) + zlib.crc32(name.encode()))
        if high:                                                # a table: each row's entries differ
            return torch.rand((*shape[:-1], high), generator=g, device="cuda").topk(shape[-1], dim=-1).indices.to(torch.int32)
        last = name.rsplit(".", 1)[-1]
        if last == "w0" or ".mu." in name:                      # decays near one; blends of a token with the one before
            x = torch.rand(shape, generator=g, device="cuda")
            return (x if ".mu." in name else 5.0 * x - 6.0).to(self.dtype)
        x = torch.randn(shape, generator=g, device="cuda") * 0.02
        if last == "vmix":
            x = x + 0.5
        elif name.endswith(("o_proj.weight", "down_proj.weight")):
            x = 0.125 * x
        elif self.model in ("llama-8b-like", "nikodra-w2048") and name in ("model.embed_tokens.weight", "embed", "bigram"):
            x = 50.0 * x
        elif name.endswith(("norm.weight", "layernorm.weight")) or (last.startswith("norm") or last == "out" or name == "final.norm"):
            around_zero = self.model == "nikodra-w2048" and (last in ("norm1", "norm1b", "norm2", "norm2b") or name == "final.norm")
            x = x if around_zero else 1.0 + x
        return x.to(self.dtype)

    def f64(self, name, *shape):
        return self(name, shape).to(F64)


# -- inputs -------------------------------------------------------------------

def _lengths(case):
    """Lengths of the sequences: spread over [low, high], both ends among them where there are several."""
    n, lo, hi = case["rows"], case["low"], case["high"]
    if n == 1 or lo == hi:
        return [hi] * n
    r = np.random.default_rng(7)                                # the same lengths for every seed: the same work
    return [lo, hi] + [int(x) for x in r.integers(lo, hi + 1, n - 2)]


def _tokens(case, seed):
    """Per sequence its prompt (or context), and the tokens fed in every later step [steps, rows]."""
    vocab = _vocab(case["model"])
    r = np.random.default_rng(seed)
    prompts = [r.integers(0, vocab, n).tolist() for n in _lengths(case)]
    return prompts, r.integers(0, vocab, (case["steps"], case["rows"]), dtype=np.int32)


def _vocab(model):
    if model in DESIGNS:
        return 32000
    from exl3_server_b200.config import presets
    return presets.SIZES[model]["vocab_size"]


def prepare(case, seed):
    if case["kind"] == "sample":
        from exl3_server_b200.sampling import RowSampler, SampleOptions
        g = torch.Generator(device="cuda").manual_seed(seed)
        rows, vocab = case["rows"], case["vocab"]
        # a language model's logits: a broad bulk and some tens of likely tokens
        logits = torch.randn(rows, vocab, generator=g, device="cuda") * 2.0
        likely = torch.randint(0, vocab, (rows, 40), generator=g, device="cuda")
        logits.scatter_add_(1, likely, 8.0 + 3.0 * torch.randn(rows, 40, generator=g, device="cuda"))
        extra = dict(repetition_penalty=1.1, presence_penalty=0.2, frequency_penalty=0.1) if case["penalties"] else {}
        opt = SampleOptions(temperature=0.8, top_k=case["top_k"], top_p=case["top_p"], min_p=case["min_p"], seed=seed + 1, **extra)
        r = np.random.default_rng(seed)
        return dict(kind="sample", logits=logits, rows=[RowSampler(opt, i, r.integers(0, vocab, 200).tolist()) for i in range(rows)])

    import exl3_server_b200 as E
    from exl3_server_b200.engine.model import plan_manifest
    plan = _plan(case["model"])
    w = _Weights(case["model"], case["dtype"], seed)
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    tensors = {s.name: w(s.name, s.shape, s.high) for s in plan_manifest(plan) if not s.optional}
    model = E.Model(plan, tensors, dtype, "cuda:0")
    prompts, fed = _tokens(case, seed)
    room = sum((len(p) + case["steps"] + 65) // 64 * 64 + 64 for p in prompts)
    engine = E.Engine(model, max_tokens=room, max_slots=case["rows"])
    state = dict(kind=case["kind"], engine=engine, prompts=prompts, fed=torch.from_numpy(fed).cuda(), steps=case["steps"])
    if case["kind"] == "decode":
        slots = [engine.open() for _ in prompts]
        at, per = 0, max(1, 8192 // len(slots))
        while at < max(len(p) for p in prompts):                # the contexts come from real steps
            engine.step([E.StepEntry(s, p[at:at + per], None) for s, p in zip(slots, prompts) if at < len(p)])
            at += per
        state["slots"] = slots
        _decode(state, slots)                                   # a server that has been decoding
        for s, p in zip(slots, prompts):
            engine.truncate(s, len(p))
    return state


def _decode(state, slots):
    session = state["engine"].decode_session(slots, max_new=state["steps"] + 1)
    out = []
    for k in range(state["steps"]):
        session.feed(state["fed"][k])
        out.append(session.step(None).clone())                  # the session's own buffer lives until its next step
    session.close()
    return out


def run(state):
    if state["kind"] == "sample":
        from exl3_server_b200.sampling import sample_rows
        return np.array(sample_rows(state["logits"], state["rows"]))
    import exl3_server_b200 as E
    engine, prompts = state["engine"], state["prompts"]
    if state["kind"] == "decode":
        out = _decode(state, state["slots"])
        for s, p in zip(state["slots"], prompts):
            engine.truncate(s, len(p))
        return out
    slots = [engine.open() for _ in prompts]
    out = [engine.step([E.StepEntry(s, p, "last") for s, p in zip(slots, prompts)])]
    if state["steps"]:
        out += _decode(state, slots)
    for s in slots:
        engine.close(s)
    return out


# -- what a pass cannot do without --------------------------------------------

def work(case):
    if case["kind"] == "sample":
        # the logits once, the ids; the counts of the penalties are per row and as long as the logits
        n = case["rows"] * case["vocab"] * 4.0
        return {"bytes": n * (2 if case["penalties"] else 1) + case["rows"] * 4.0, "flops": 0.0}
    from exl3_server_b200.engine.model import plan_manifest
    plan = _plan(case["model"])
    item = 4 if case["dtype"] == "float32" else 2
    size = {s.name: math.prod(s.shape) for s in plan_manifest(plan) if not s.optional}
    vocab, width = _vocab(case["model"]), plan.embedding.width
    tables = [n for n in size if "embed" in n or n == "bigram" or n.endswith(".table")]
    head = vocab * width
    body = sum(v for n, v in size.items() if n not in tables and n not in ("head", "lm_head.weight"))
    experts, picked = 0, 0.0
    if case["model"] == "soporax-w2048":
        twice = sum(v for n, v in size.items() if n.startswith(("l1.", "l2.")) and n not in tables)
        experts = sum(v * (2 if n.startswith(("l1.", "l2.")) else 1) for n, v in size.items() if ".mlp.e" in n)
        body += twice
        picked = 2.0 / 16.0
    # keys a token sees are read, and its own written, per layer (features of a key and a value together)
    if case["model"] == "nikodra-w2048":
        attn = [(2 * 16 * 128, 4096 * 2, 0)] * 4 + [(2 * 16 * 128, 4096 * 2, 1024)] * 2
        fixed = 2 * 2 * 4 * (16 * 64 * 128 + 32 * 64 * 64)           # float32 states of a step, read and written
    elif case["model"] == "soporax-w2048":
        attn = [(576, 2 * 16 * (576 + 512), 0)] * 2 + [(2 * 16 * 128, 4096 * 2, 1024)] * 3 + [(2 * 16 * 128, 4096 * 2, 0)] * 3
        fixed = 0
    else:
        from exl3_server_b200.config import presets
        z = presets.SIZES[case["model"]]
        attn = [(2 * z["num_key_value_heads"] * z["head_dim"], 4 * z["num_attention_heads"] * z["head_dim"], 0)] * z["num_hidden_layers"]
        fixed = 0
    out = {"bytes": 0.0, "flops": 0.0}

    def step(starts, counts):
        tokens, rows = sum(counts), len(counts)
        seen = body - experts * (1.0 - picked) if picked else body
        read = body - experts * (1.0 - picked) ** tokens if picked else body      # experts that some token of the step lists
        out["bytes"] += item * (read + head + tokens * width) + 4.0 * rows * vocab + rows * fixed
        out["flops"] += 2.0 * seen * tokens + 2.0 * head * rows
        for feats, per_key, window in attn:
            for s, n in zip(starts, counts):
                past = min(s, window) if window else s
                out["bytes"] += item * feats * (past + n)
                full = n * s + n * (n + 1) / 2.0
                out["flops"] += per_key * (min(full, n * float(window)) if window else full)

    lens = _lengths(case)
    if case["kind"] == "serve":
        step([0] * len(lens), lens)
    for k in range(case["steps"]):
        step([n + k for n in lens], [1] * len(lens))
    return out


def tolerance(case):
    if case["kind"] == "sample":
        return {"rel": 0.0, "differ": 0.01}      # a draw within float32 rounding of a boundary between two tokens
    if case["dtype"] == "float32":
        return {"rel": 5e-6}                     # 0.8e-6 away from 64 bits
    # bfloat16 between kernels is 0.002 to 0.007 away from 64 bits; two roundings of it can be apart by both
    return {"rel": 0.025, "max": 0.25}


# -- the same in 64 bits ------------------------------------------------------

def _unit(x, eps):
    return x * torch.rsqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _turn(x, freqs, mult=1.0, neighbours=False):
    """x [T, heads, d] at positions 0 .. T-1, the first 2 len(freqs) features rotated in pairs."""
    n = len(freqs)
    a = torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * torch.tensor(freqs, dtype=F64, device=x.device)
    c, s = (a.cos() * mult)[:, None], (a.sin() * mult)[:, None]
    y = x.clone()
    first, second = (slice(0, 2 * n, 2), slice(1, 2 * n, 2)) if neighbours else (slice(0, n), slice(n, 2 * n))
    u, v = x[..., first], x[..., second]
    y[..., first], y[..., second] = u * c - v * s, v * c + u * s
    return y


def _attend(q, k, v, scale, sink=None, window=0, block=0):
    """q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H * dv], causal.  ``sink``: [H] scores of a key without a value."""
    T, H = q.shape[:2]
    G = k.shape[1]
    at = torch.arange(T, device=q.device)
    out = torch.empty(T, H, v.shape[2], dtype=F64, device=q.device)
    for g in range(G):
        mine = slice(g * (H // G), (g + 1) * (H // G))
        for a in range(0, T, 1024):
            b = min(T, a + 1024)
            i, j = at[a:b, None], at[None, :b]
            hidden = j > i
            if window:
                hidden = hidden | (i - j >= window)
            if block:
                hidden = hidden | (i // block != j // block)
            s = torch.einsum("thd,sd->hts", q[a:b, mine], k[:b, g]).mul_(scale).masked_fill_(hidden, -math.inf)
            if sink is None:
                p = torch.softmax(s, dim=-1)
            else:
                extra = sink[mine].view(-1, 1, 1).expand(-1, b - a, 1)
                p = torch.softmax(torch.cat([s, extra], dim=-1), dim=-1)[..., :-1]
            out[a:b, mine] = torch.einsum("hts,sd->thd", p, v[:b, g])
    return out.reshape(T, -1)


def _each(seqs, f):
    """f on every sequence's rows of the packed tensors."""
    return lambda *xs: torch.cat([f(*(x[a:b] for x in xs)) for a, b in seqs])


def _exact_llama(case, w, ids, seqs):
    from exl3_server_b200.config import presets
    z = presets.SIZES[case["model"]]
    W, H, G, d, ff = (z[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim", "intermediate_size"))
    eps, n = z["rms_norm_eps"], z["num_hidden_layers"]
    rho = z["scale_depth"] / math.sqrt(n) if "scale_depth" in z else 1.0
    freqs = [z["rope_theta"] ** (-2.0 * i / d) for i in range(d // 2)]
    attend = _each(seqs, lambda q, k, v: _attend(_turn(q, freqs), _turn(k, freqs), v, d ** -0.5))
    table = w("model.embed_tokens.weight", (z["vocab_size"], W))
    x = table[ids].to(F64) * z.get("scale_emb", 1.0)
    for i in range(n):
        p = f"model.layers.{i}."
        h = _unit(x, eps) * w.f64(p + "input_layernorm.weight", W)
        q, k, v = ((h @ w.f64(f"{p}self_attn.{t}_proj.weight", m * d, W).T).view(-1, m, d) for t, m in (("q", H), ("k", G), ("v", G)))
        x = x + rho * (attend(q, k, v) @ w.f64(p + "self_attn.o_proj.weight", W, H * d).T)
        h = _unit(x, eps) * w.f64(p + "post_attention_layernorm.weight", W)
        h = _silu(h @ w.f64(p + "mlp.gate_proj.weight", ff, W).T) * (h @ w.f64(p + "mlp.up_proj.weight", ff, W).T)
        x = x + rho * (h @ w.f64(p + "mlp.down_proj.weight", W, ff).T)
    head = table if z["tie_word_embeddings"] else w("lm_head.weight", (z["vocab_size"], W))
    scale = z.get("dim_model_base", W) / W

    def logits(rows):
        return (_unit(x[rows], eps) * w.f64("model.norm.weight", W) * scale) @ head.to(F64).T
    return logits


def _ramped(rot):
    """Frequencies and the factor on sines and cosines, scaled along a ramp over the pairs."""
    dims, base, s = rot["dims"], rot["base"], rot.get("scaling")
    freqs = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    if not s:
        return freqs, 1.0
    pair_of = lambda turns: dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(pair_of(s["fast"])), 0), min(math.ceil(pair_of(s["slow"])), dims - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
    return [f / s["factor"] * r + f * (1.0 - r) for f, r in zip(freqs, ramp)], 0.1 * math.log(s["factor"]) + 1.0


def _padded(x, seqs):
    """Packed rows as [sequences, longest, ...], zeros behind the shorter ones."""
    y = x.new_zeros(len(seqs), max(b - a for a, b in seqs), *x.shape[1:])
    for i, (a, b) in enumerate(seqs):
        y[i, :b - a] = x[a:b]
    return y


def _packed(y, seqs):
    return torch.cat([y[i, :b - a] for i, (a, b) in enumerate(seqs)])


def _exact_nikodra(case, w, ids, seqs):
    c = _nikodra()
    W, eps, mult = c["width"], c["norm_eps"], c["residual_mult"]
    norm = lambda x, name: _unit(x, eps) * (1.0 + w.f64(name, W))  # noqa: E731
    bg = c["bigram"]
    rows = torch.cat([torch.cat([ids.new_full((1,), bg["buckets"]), (ids[a:b - 1] * bg["mul_prev"] + ids[a + 1:b] * bg["mul_cur"]) % bg["buckets"]])
                      for a, b in seqs])
    x = w("embed", (c["vocab"], W))[ids].to(F64) + w("bigram", (bg["buckets"] + 1, W))[rows].to(F64)
    zero, first_values = None, None
    for i, (kind, m, mlp) in enumerate(c["layers"]):
        p = f"l{i}.mix."
        h = norm(x, f"l{i}.norm1")
        lin = lambda name, n, src=None: (h if src is None else src) @ w.f64(p + name, n, (h if src is None else src).shape[1]).T  # noqa: E731
        if kind == "attention":
            H, d = m["heads"], m["dim"]
            freqs, factor = _ramped(m["rot"])
            zero = torch.zeros(H, dtype=F64, device=x.device)
            q, k, v = ((lin(t, H * d) + w.f64(f"{p}{t}.b", H * d)).view(-1, H, d) for t in "qkv")
            q, k = (_unit(t, eps) * w.f64(f"{p}{n}.norm", d) for t, n in ((q, "q"), (k, "k")))
            if first_values is None:
                first_values = v
            else:
                lam = w.f64(p + "vmix")
                v = (1.0 - lam) * v + lam * first_values
            o = _each(seqs, lambda q, k, v: _attend(_turn(q, freqs, factor, True), _turn(k, freqs, factor, True), v, m["scale"], zero))(q, k, v)
            y = o @ w.f64(p + "o", W, H * d).T + w.f64(p + "o.b", W)
        elif kind == "parallel":
            a, b = m["left"], m["right"]
            H, d = a["heads"], a["dim"]
            q, k, v = (lin(f"left.{t}", H * d).view(-1, H, d) for t in "qkv")
            left = _each(seqs, lambda q, k, v: _attend(_unit(q, eps), _unit(k, eps), v, a["scale"], zero, block=a["mask"]["size"]))(q, k, v)
            left = left @ w.f64(p + "left.o", W, H * d).T
            H, d, dv = b["heads"], b["dim"], b["vdim"]
            freqs, _ = _ramped(b["rot"])
            q, k, v = (lin(f"right.{t}", H * n).view(-1, H, n) for t, n in (("q", d), ("k", d), ("v", dv)))
            q, k = _each(seqs, lambda t: _turn(t, freqs))(q), _each(seqs, lambda t: _turn(t, freqs))(k) * d ** -0.5
            # o_t = sum over s <= t of decay^(t - s) (q_t k_s) v_s
            decay = torch.tensor(b["decay"], dtype=F64, device=x.device)

            def retained(q, k, v):
                T = q.shape[0]
                at = torch.arange(T, device=q.device)
                gap = (at[:, None] - at[None, :]).clamp(min=0).to(F64)
                return torch.stack([((q[:, n] @ k[:, n].T) * (decay[n] ** gap).tril_()) @ v[:, n] for n in range(H)], dim=1)
            o = _unit(_each(seqs, retained)(q, k, v), eps).reshape(-1, H * dv)
            right = (o * _silu(lin("right.g", H * dv))) @ w.f64(p + "right.o", W, H * dv).T
            y = 0.5 * (_unit(left, eps) * w.f64(p + "left.out", W) + _unit(right, eps) * w.f64(p + "right.out", W))
        else:
            H, d = m["heads"], m["dim"]
            before = _each(seqs, lambda t: torch.cat([torch.zeros_like(t[:1]), t[:-1]]))(h)
            mixed = {s: h + (before - h) * w.f64(f"{p}mu.{s}", W) for s in "rkvgw"}
            r, k, v = (_padded(lin(s, H * d, mixed[s]).view(-1, H, d), seqs) for s in "rkv")
            rank = lin("w1", m["decay_rank"], mixed["w"]).tanh()
            decay = torch.exp(-torch.exp(rank @ w.f64(p + "w2", H * d, m["decay_rank"]).T + w.f64(p + "w0", H * d)))
            decay, u = _padded(decay.view(-1, H, d), seqs), w.f64(p + "u", H, d)
            S = x.new_zeros(len(seqs), H, d, d)
            o = torch.empty_like(v)
            for t in range(v.shape[1]):
                kv = k[:, t, :, :, None] * v[:, t, :, None, :]
                o[:, t] = torch.einsum("bhij,bhi->bhj", S + u[:, :, None] * kv, r[:, t])
                S = decay[:, t, :, :, None] * S + kv
            o = _unit(_packed(o, seqs), eps).reshape(-1, H * d)
            y = (o * w.f64(p + "norm", H * d) * _silu(lin("g", H * d, mixed["g"]))) @ w.f64(p + "o", W, H * d).T
        x = x + mult * norm(y, f"l{i}.norm1b")
        h = norm(x, f"l{i}.norm2") @ w.f64(f"l{i}.mlp.up", mlp["ff"], W).T
        h = 0.5 * h * (1.0 + torch.erf(h / math.sqrt(2.0)))
        x = x + mult * norm(h @ w.f64(f"l{i}.mlp.down", W, mlp["ff"]).T, f"l{i}.norm2b")
    return lambda at: norm(x[at], "final.norm") @ w.f64("head", c["vocab"], W).T


def _banded(rot):
    """Frequencies with a short wavelength kept, with a long one divided, a straight line between."""
    s, out = rot["scaling"], []
    for f in (rot["base"] ** (-2.0 * i / rot["dims"]) for i in range(rot["dims"] // 2)):
        wave = 2.0 * math.pi / f
        part = min(1.0, max(0.0, (s["original"] / wave - s["low"]) / (s["high"] - s["low"])))
        out.append((1.0 - part) * f / s["factor"] + part * f)
    return out


def _exact_soporax(case, w, ids, seqs):
    c = _soporax()
    W, eps, loop = c["width"], c["norm_eps"], c["loop"]
    norm = lambda x, name: _unit(x, eps) * w.f64(name, x.shape[1])  # noqa: E731
    table = w("embed", (c["vocab"], W))
    start = table[ids].to(F64)
    x = start
    steps = w.f64("loop.step", loop["times"], W)
    order = [(i, None) for i in range(loop["start"])]
    for t in range(loop["times"]):
        order += [(i, t if i == loop["start"] else None) for i in range(loop["start"], loop["stop"])]
    order += [(i, None) for i in range(loop["stop"], len(c["layers"]))]
    for i, t in order:
        if t is not None:
            x = x + (start if t else 0.0) + steps[t]
        kind, m, mlp = c["layers"][i]
        p, f = f"l{i}.mix.", f"l{i}.mlp."
        h = norm(x, f"l{i}.norm1")
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        if kind == "latent_attention":
            rd, r = m["rot_dim"], m["kv_rank"]
            freqs, factor = _ramped(m["rot"])
            q = (norm(h @ w.f64(p + "dq", m["q_rank"], W).T, p + "dq.norm") @ w.f64(p + "uq", H * (d + rd), m["q_rank"]).T).view(-1, H, d + rd)
            down = h @ w.f64(p + "dkv", r + rd, W).T
            lat = norm(down[:, :r], p + "dkv.norm")
            k, v = (lat @ w.f64(p + "uk", H * d, r).T).view(-1, H, d), (lat @ w.f64(p + "uv", H * dv, r).T).view(-1, H, dv)
            turn = lambda t: _turn(t, freqs, factor, True)  # noqa: E731
            o = _each(seqs, lambda q, k, v, kr: _attend(
                torch.cat([q[..., :d], turn(q[..., d:])], dim=-1), torch.cat([k, turn(kr[:, None]).expand(-1, H, -1)], dim=-1), v,
                m["scale"]))(q, k, v, down[:, r:])
            o = o * torch.sigmoid(h @ w.f64(p + "g", H * dv, W).T)
        elif kind == "attention":
            q, k, v = ((h @ w.f64(p + s, H * d, W).T).view(-1, H, d) for s in "qkv")
            sink = w.f64(p + "sink", H)
            o = _each(seqs, lambda q, k, v: _attend(_unit(q, eps), _unit(k, eps), v, m["scale"], sink, window=m["mask"]["size"]))(q, k, v)
        else:
            freqs = _banded(m["rot"])
            q, k, v = ((h @ w.f64(p + s, H * d, W).T + w.f64(f"{p}{s}.b", H * d)).view(-1, H, d) for s in "qkv")
            zero = torch.zeros(H, dtype=F64, device=x.device)
            o = _each(seqs, lambda q, k, v: _attend(_turn(q, freqs, 1.0, True), _turn(k, freqs, 1.0, True), v, m["scale"], zero))(q, k, v)
            o = (o.view(-1, H, dv) * torch.sigmoid(h @ w.f64(p + "g", H, W).T)[:, :, None]).reshape(-1, H * dv)
        y = o @ w.f64(p + "o", W, H * dv).T
        if mlp["kind"] == "dense":
            g = torch.clamp(h @ w.f64(f + "gate", mlp["ff"], W).T, max=mlp["limit"])
            u = torch.clamp(h @ w.f64(f + "up", mlp["ff"], W).T, min=-mlp["limit"], max=mlp["limit"])
            y = y + (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w.f64(f + "down", W, mlp["ff"]).T
        else:
            n, top, ff = mlp["router"]["experts"], mlp["router"]["top"], mlp["expert"]["ff"]
            picks = w(f + "table", (c["vocab"], top), n)[ids]
            for e in range(n):
                at = (picks == e).any(dim=1).nonzero()[:, 0]
                z = _silu(h[at] @ w.f64(f"{f}e{e}.gate", ff, W).T) * (h[at] @ w.f64(f"{f}e{e}.up", ff, W).T)
                y = y.index_add(0, at, z @ w.f64(f"{f}e{e}.down", W, ff).T / top)
        x = x + y
    return lambda at: norm(x[at], "final.norm") @ table.to(F64).T * c["logit_scale"]


def exact(case, seed):
    if case["kind"] == "sample":
        return None                              # whole numbers, drawn
    if work({**case, "kind": "serve"})["flops"] > 4e14:
        return None                              # some 15 seconds in 64 bits
    prompts, fed = _tokens(case, seed)
    steps, first = case["steps"], 0 if case["kind"] == "serve" else 1
    whole = [p + fed[:, i].tolist() for i, p in enumerate(prompts)]
    ends = np.cumsum([len(t) for t in whole])
    seqs = [(int(e) - len(t), int(e)) for e, t in zip(ends, whole)]
    ids = torch.tensor([t for s in whole for t in s], dtype=torch.int64, device="cuda")
    w = _Weights(case["model"], case["dtype"], seed)
    restated = {"nikodra-w2048": _exact_nikodra, "soporax-w2048": _exact_soporax}.get(case["model"], _exact_llama)
    with torch.no_grad():
        logits = restated(case, w, ids, seqs)
        # the place of a sequence's k-th logits: after its last prompt token and the first k fed ones
        return [logits(torch.tensor([b - steps - 1 + k for _, b in seqs], device="cuda")) for k in range(first, steps + 1)]
