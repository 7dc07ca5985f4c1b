"""What generation with this framework is measured on: whole passes through its entry points.

Three kinds of pass, each on a loaded model with seeded random weights:

* ``prompt``: prompts of unequal length in one step (``LM.step``), float32 logits behind each prompt;
* ``generate``: the calls that ``LM.generate`` makes for a batch (open, prefill, a decode step per token, close), and
  behind the last token one ``LM.step``, so that logits come back beside the tokens;
* ``turn``: the same for a conversation whose earlier turns are kept in the cache (``retain``): only the turn's own
  tokens run before the answer.  Asked again, a turn starts from the same kept positions.

Shapes are the library's own (``cima_b200.config.shapes``); a design's shapes are cut to their first layers, as
``bench.py --design`` cuts them.  The weights are the library's random ones but for the embedding and the head: a
random head makes next tokens that rounding decides, where a trained one has margins.  So the embedding is as large
as what the layers add to it, and the head favours one follower for each token (the token itself where table and head
are one tensor).  What the layers compute is as with any other weights.
"""
from __future__ import annotations

import math
import re

import torch

import cima_b200
from cima_b200.config.shapes import SHAPES
from cima_b200.engine import StepEntry, build_plan

STEP, ADD = 7919, 12345             # the follower of token v is (v * STEP + ADD) mod vocab


# ---------------------------------------------------------------------------------------------- the cases
def _case(name, kind, shape, batch, prompt, kept=0, new=0, layers=0, dtype="bfloat16", sampling="greedy"):
    return dict(name=name, kind=kind, shape=shape, layers=layers, dtype=dtype, batch=batch, prompt=prompt, kept=kept, new=new,
                sampling=sampling)


def listed():
    return [
        # one user, a short question, a short answer on the smallest model: launches and latency
        _case("chat-0.5b", "generate", "qwen2.5-0.5b", 1, 37, new=24),
        # a request on the 32-bit path, sampled with the options that cut the tail
        _case("float32-0.5b", "generate", "qwen2.5-0.5b", 2, 201, new=12, dtype="float32", sampling="sampled"),
        # a few requests of odd lengths together, greedy
        _case("requests-1.5b", "generate", "qwen2.5-1.5b", 5, 333, new=20),
        # scoring or first tokens for a handful of prompts, short ones and long ones
        _case("prompts-1.5b", "prompt", "qwen2.5-1.5b", 9, 700),
        # a conversation with a long document behind it
        _case("document-1.5b", "turn", "qwen2.5-1.5b", 1, 61, kept=16001, new=24),
        # the benchmark's decode: the 7B shape, 8 sequences, 2,048 positions
        _case("turn-7b", "turn", "qwen2.5-7b", 8, 40, kept=2048, new=24),
        # the benchmark's prompt
        _case("prompt-7b", "prompt", "qwen2.5-7b", 1, 2048),
        # a full batch, sampled with the default options
        _case("batch-7b", "turn", "qwen2.5-7b", 64, 12, kept=260, new=12, sampling="default"),
        # delta rule by channel, decay recurrence, sigmoid-routed experts: prompts and answers
        _case("gisirax-1.5b", "generate", "gisirax-1.5b", 4, 900, new=16, layers=6),
        # differential attention and the gate recurrence: one long prompt
        _case("lipizen-3b", "prompt", "lipizen-3b", 1, 2048, layers=4),
        # delta rule by head, latent attention, ungated experts, token inputs: a batch of short requests
        _case("gudarax-1.5b", "generate", "gudarax-1.5b", 8, 150, new=32, layers=6),
    ]


_LARGEST = 5.0e11                   # bytes, or flops / 50, that a drawn case stays under


def draw(rng):
    while True:
        c = _draw(rng)
        w = work(c)
        if max(w["bytes"], w["flops"] / 50) <= _LARGEST and c["batch"] * (c["kept"] + c["prompt"]) <= 20000:
            return c


def _draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    shape, layers = rng.choice([("qwen2.5-0.5b", 0), ("qwen2.5-0.5b", 0), ("qwen2.5-1.5b", 0), ("qwen2.5-3b", 0), ("qwen2.5-7b", 0),
                                ("gisirax-1.5b", 6), ("gisirax-3b", 3), ("lipizen-1.5b", 4), ("lipizen-3b", 4), ("gudarax-1.5b", 6),
                                ("gudarax-3b", 3)])
    qwen2 = shape.startswith("qwen2")
    kind = rng.choice(["prompt", "generate", "turn"] if qwen2 else ["prompt", "generate"])
    dtype = "float32" if shape == "qwen2.5-0.5b" and rng.random() < 0.3 else "bfloat16"
    sampling = rng.choice(["greedy", "sampled"] if shape in ("qwen2.5-0.5b", "qwen2.5-1.5b", "qwen2.5-3b") else ["greedy", "default"])
    c = _case("", kind, shape, log(1, 64), log(8, 600 if dtype == "float32" else 2048), layers=layers, dtype=dtype)
    del c["name"]
    if kind != "prompt":
        c.update(new=log(4, 32), sampling=sampling)
    if kind == "turn":
        c.update(prompt=log(4, 256), kept=log(64, 8192))
    return c


# ---------------------------------------------------------------------------------------------- inputs
def _config(case):
    raw = dict(SHAPES[case["shape"]])
    if case["layers"]:
        raw["layers"] = raw["layers"][:case["layers"]]
    return raw


def _sizes(raw):
    """(width, vocabulary, layers, the feed-forward's values)."""
    if "layers" in raw:
        return raw["width"], raw["vocab"], len(raw["layers"]), 0
    return raw["hidden_size"], raw["vocab_size"], raw["num_hidden_layers"], raw["intermediate_size"]


def _lengths(n, batch):
    """``batch`` lengths around n: one of n, the others odd fractions of it."""
    return [n] + [max(1, n * (37 + 61 * i % 100) // 100 | 1) for i in range(1, batch)]


def _tokens(case, seed):
    """(kept, prompt) token ids of every sequence."""
    vocab = _sizes(_config(case))[1]
    g = torch.Generator().manual_seed(seed)
    make = lambda n: torch.randint(0, vocab, (n,), generator=g).tolist()                       # noqa: E731
    kept = [make(n) for n in _lengths(case["kept"], case["batch"])] if case["kept"] else [[] for _ in range(case["batch"])]
    return kept, [make(n) for n in _lengths(case["prompt"], case["batch"])]


def _model(case, seed):
    raw = _config(case)
    width, vocab, layers, ff = _sizes(raw)
    page = lambda n: -(-n // 64) * 64                                                           # noqa: E731
    most = [page(k + p + case["new"] + 2) for k, p in zip(_lengths(case["kept"], case["batch"]) if case["kept"] else [0] * case["batch"],
                                                           _lengths(case["prompt"], case["batch"]))]
    lm = cima_b200.load(config=raw, seed=seed, draw="device", dtype=case["dtype"], device="cuda:0", max_seqs=case["batch"],
                        max_tokens=max(sum(most), case["batch"] * 512), max_batch=case["batch"], verbose=False,
                        retain=case["batch"] if case["kind"] == "turn" else 0)
    w = lm.state_dict()
    embed = w["model.embed_tokens.weight" if ff else "embed"]
    # three times what the layers add in all: a dense feed-forward leaves about 0.01 sqrt(ff layers) min(1, 0.02^2 width);
    # six with the designs' experts, so that a choice between two of them that rounding decides stays a small difference;
    # where norms stand behind the sums it is the feed-forwards that are made smaller
    size = 3.0 * max(1.0, 0.01 * math.sqrt(ff * layers) * min(1.0, 0.0004 * width)) if ff else 1.0 if "postln_alpha" in raw else 6.0
    embed.mul_(size / 0.02)
    if "postln_alpha" in raw:
        for i in range(layers):
            w[f"l{i}.mlp.down"].mul_(0.25)
    scale = float(2.0 / math.sqrt(width))
    if raw.get("tie_word_embeddings"):
        w["model.norm.weight"].mul_(scale / float(embed.float().square().mean().sqrt()))
    else:
        at = torch.arange(vocab, device=embed.device)
        w["lm_head.weight" if ff else "head"][(at * STEP + ADD) % vocab] = embed * (scale / float(embed.float().square().mean().sqrt()))
    return lm


def _options(case):
    new = max(1, case["new"])
    if case["sampling"] == "default":
        return [cima_b200.GenOptions(max_tokens=new, ignore_eos=True, seed=11 + i) for i in range(case["batch"])]
    if case["sampling"] == "sampled":
        return [cima_b200.GenOptions(temperature=0.7, top_k=50, top_p=0.95, repeat_penalty=1.0, max_tokens=new, ignore_eos=True, seed=5 + i)
                for i in range(case["batch"])]
    return [cima_b200.GenOptions(temperature=0.0, repeat_penalty=1.0, max_tokens=new, ignore_eos=True)] * case["batch"]


def prepare(case, seed):
    """A loaded model that has served requests of these sizes before (its decode steps are recorded), kept turns in its
    cache where the case has them, and the next request's token ids."""
    lm = _model(case, seed)
    kept, prompts = _tokens(case, seed)
    st = {"lm": lm, "kind": case["kind"], "kept": kept, "prompts": prompts, "options": _options(case), "new": case["new"]}
    if case["kind"] == "turn":
        slots = lm.stepper.open(len(kept))
        lm.stepper.prefill(slots, kept, st["options"])
        lm.stepper.retain(slots, kept)
    warm = dict(st, prompts=_tokens(case, seed + 1000003)[1])
    for _ in range(2):                                   # a shape's second step is the one that is recorded
        run(warm)
    return st


# ---------------------------------------------------------------------------------------------- one pass
def run(state):
    lm = state["lm"]
    return _prompt(lm, state) if state["kind"] == "prompt" else _answer(lm, state)


def _prompt(lm, s):
    slots = lm.model.cache.open(len(s["prompts"]))
    try:
        return {"logits": lm.step([StepEntry(slot, p, [len(p) - 1]) for slot, p in zip(slots, s["prompts"])])}
    finally:
        lm.model.cache.close(slots)


def _answer(lm, s):
    st, options = lm.stepper, s["options"]
    prompts = [k + p for k, p in zip(s["kept"], s["prompts"])]
    if s["kind"] == "turn":
        taken = st.adopt(prompts)
        slots = [slot for slot, _ in taken]
        tokens = st.prefill(slots, prompts, options, reused=[n for _, n in taken])
    else:
        slots = st.open(len(prompts))
        tokens = st.prefill(slots, prompts, options)
    out = [tokens]
    for _ in range(s["new"] - 1):
        tokens = st.decode(slots, tokens, options)
        out.append(tokens)
    logits = lm.step([StepEntry(slot, [t], [0]) for slot, t in zip(slots, tokens)])
    if s["kind"] == "turn":
        st.retain(slots, s["kept"])
    else:
        st.close(slots)
    return {"tokens": torch.tensor(out), "logits": logits}


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    raw = _config(case)
    entry = cima_b200.lookup_architecture(raw)
    plan = build_plan(entry.spec(entry.parse(raw)))
    width, vocab, layers, _ = _sizes(raw)
    item = 4 if case["dtype"] == "float32" else 2
    dense = expert = 0
    for name, t in plan.items():
        n = math.prod(t.shape) if t.shape else 1
        if re.search(r"\.e\d+\.", name):
            expert += n
        elif not (name in ("embed", "pos", "bigram", "side.embed") or (name.startswith("model.embed") and not raw.get("tie_word_embeddings"))):
            dense += n
    moe = next((x["mlp"]["router"] for x in raw.get("layers", []) if x["mlp"]["kind"] == "moe"), {"experts": 1, "top": 1})
    body, head = dense - vocab * width, vocab * width
    # what attention reads and multiplies per position of context: the layers that keep keys and values
    if "layers" in raw:
        attn = [(x["mixer"].get("left") or x["mixer"], x["type"]) for x in raw["layers"]]
        attn = [(m, t) for m, t in attn if t in ("attention", "parallel", "latent_attention")]
        kv = sum(m["kv_rank"] if "kv_rank" in m else (0 if "kv_from" in m else m["kv_heads"] * (m["vdim"] + m["dim"] * (2 if "diff" in m else 1)))
                 for m, _ in attn)
        pairs = sum(2 * m["heads"] * (m["dim"] + m["vdim"]) * (2 if "diff" in m else 1) for m, _ in attn)
        window = min([(m.get("mask") or {}).get("size", 1 << 30) for m, _ in attn])
    else:
        kv = layers * 2 * raw["num_key_value_heads"] * raw["head_dim"]
        pairs = layers * 4 * raw["num_attention_heads"] * raw["head_dim"]
        window = 1 << 30
    kept, prompts = _lengths(case["kept"], case["batch"]) if case["kept"] else [0] * case["batch"], _lengths(case["prompt"], case["batch"])
    nbytes = flops = 0.0
    steps = [(kept, prompts)] + [([k + p + i for k, p in zip(kept, prompts)], [1] * case["batch"]) for i in range(case["new"])]
    for at, rows in steps:
        T = sum(rows)
        reach = min(1.0, T * moe["top"] / moe["experts"])
        nbytes += item * (body + head + expert * reach + kv * (sum(min(a, window) for a in at) + T)) + 4.0 * len(rows) * vocab
        flops += 2.0 * T * (body + expert * moe["top"] / moe["experts"]) + 2.0 * len(rows) * head
        flops += sum(pairs * min(a * n + n * (n + 1) / 2.0, float(n) * window) for a, n in zip(at, rows))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what the path is off its 64-bit result: 8e-7 in 32 bits, 0.002 to 0.007 in bfloat16; up to 0.02 where
    experts are chosen and rounding decides a choice."""
    if case["dtype"] == "float32":
        return {"rel": 5e-6, "differ": 0.0}
    if case["shape"].startswith(("gisirax", "gudarax")):
        return {"rel": 2.5e-2, "max": 0.4, "differ": 0.0}
    return {"rel": 1.5e-2, "max": 0.2, "differ": 0.0}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """Plain torch in 64 bits, layer by layer over whole sequences, no cache.  The tokens have no such value; the
    logits behind them follow from the token that the head favours after each."""
    raw = _config(case)
    lm = _model(case, seed)
    w = lm.state_dict()
    vocab = _sizes(raw)[1]
    kept, prompts = _tokens(case, seed)
    seqs = []
    for k, p in zip(kept, prompts):
        ids = k + p
        for _ in range(case["new"]):
            ids.append(ids[-1] if raw.get("tie_word_embeddings") else (ids[-1] * STEP + ADD) % vocab)
        seqs.append(torch.tensor(ids, device="cuda:0"))
    W = lambda name: w[name].double()                                                           # noqa: E731
    with torch.no_grad():
        logits = {"qwen2.5": _qwen2, "gisirax": _gisirax, "lipizen": _lipizen, "gudarax": _gudarax}[case["shape"].split("-")[0]](raw, w, W, seqs)
    return {"logits": logits} if case["kind"] == "prompt" else {"tokens": None, "logits": logits}


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _turned(x, freqs):
    """x [T, heads, dim]: value i of a head turns with value i + len(freqs) by position * freqs[i]; the rest passes."""
    half = freqs.numel()
    a = torch.arange(x.shape[0], device=x.device, dtype=x.dtype)[:, None] * freqs.to(x.device)[None]
    c, s = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * half:]], -1)


def _freqs(dims, base):
    return base ** (-torch.arange(0, dims, 2, dtype=torch.float64) / dims)


def _attend(q, k, v, scale, size=0, first=0, sink=False, slopes=None):
    """q [T, H, d], k [T, G, d], v [T, G, e]: causal softmax attention, [T, H, e]."""
    T, H = q.shape[:2]
    G = k.shape[1]
    kh, vh = k.permute(1, 2, 0), v.permute(1, 0, 2)
    out = []
    step = max(1, (1 << 27) // (H * T))
    for lo in range(0, T, step):
        hi = min(T, lo + step)
        i, j = torch.arange(lo, hi, device=q.device)[:, None], torch.arange(hi, device=q.device)[None]
        s = (q[lo:hi].view(hi - lo, G, H // G, -1).permute(1, 2, 0, 3).reshape(G, -1, q.shape[2]) @ kh[..., :hi]).view(H, hi - lo, hi) * scale
        if slopes is not None:
            s = s - slopes.to(q.device)[:, None, None] * (i - j)
        seen = j <= i
        if size:
            seen = seen & ((i - j < size) | (j < first))
        s = s.masked_fill(~seen, -math.inf)
        m = s.amax(-1, keepdim=True)
        if sink:
            m = m.clamp(min=0.0)
        e = (s - m).exp()
        e = e / (e.sum(-1, keepdim=True) + ((-m).exp() if sink else 0.0))
        out.append((e.view(G, -1, hi) @ vh[:, :hi]).view(H, hi - lo, -1).permute(1, 0, 2))
    return torch.cat(out)


def _taps(z, w):
    n = w.shape[1]
    z = torch.cat([z.new_zeros(n - 1, z.shape[1]), z])
    return sum(w[:, j] * z[j:z.shape[0] - n + 1 + j] for j in range(n))


def _walk(T, S, step):
    """o_t of a recurrence over T tokens: ``step(t, S)`` gives the state behind token t and what is read of it."""
    out = []
    for t in range(T):
        S, o = step(t, S)
        out.append(o)
    return torch.stack(out)


def _decay_rule(q, k, v, f):
    """S <- f S + k v^T by head (f [T, H, d] or [H, 1]), o = S^T q."""
    def step(t, S):
        S = (f[t] if f.dim() == 3 else f)[..., None] * S + k[t][..., None] * v[t][:, None]
        return S, (S * q[t][..., None]).sum(1)
    return _walk(q.shape[0], q.new_zeros(q.shape[1], q.shape[2], v.shape[2]), step)


def _delta(q, k, v, beta, g):
    """S <- g S; S <- S + k (beta (v - S^T k))^T; o = S^T q; g [T, H, d] or [T, H, 1]."""
    def step(t, S):
        S = g[t][..., None] * S
        u = beta[t][:, None] * (v[t] - (S * k[t][..., None]).sum(1))
        S = S + k[t][..., None] * u[:, None]
        return S, (S * q[t][..., None]).sum(1)
    return _walk(q.shape[0], q.new_zeros(q.shape[1], q.shape[2], v.shape[2]), step)


def _unit(z):
    return z * torch.rsqrt((z * z).sum(-1, keepdim=True) + 1e-6)


def _silu(z):
    return z * torch.sigmoid(z)


def _qwen2(raw, w, W, seqs):
    H, G, d, eps = raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"], raw["rms_norm_eps"]
    f = _freqs(d, raw["rope_theta"])
    xs = [w["model.embed_tokens.weight"][s].double() for s in seqs]
    for i in range(raw["num_hidden_layers"]):
        P = lambda n: W(f"model.layers.{i}.{n}")                                                # noqa: E731,B023
        a, b = P("input_layernorm.weight"), P("post_attention_layernorm.weight")
        wq, wk, wv = (P(f"self_attn.{n}_proj.weight") for n in "qkv")
        bq, bk, bv = (P(f"self_attn.{n}_proj.bias") for n in "qkv")
        wo, wg, wu, wd = P("self_attn.o_proj.weight"), P("mlp.gate_proj.weight"), P("mlp.up_proj.weight"), P("mlp.down_proj.weight")
        for n, x in enumerate(xs):
            h = _rms(x, eps) * a
            q, k = _turned((h @ wq.T + bq).view(-1, H, d), f), _turned((h @ wk.T + bk).view(-1, G, d), f)
            x = x + _attend(q, k, (h @ wv.T + bv).view(-1, G, d), d ** -0.5).reshape(-1, H * d) @ wo.T
            h = _rms(x, eps) * b
            xs[n] = x + (_silu(h @ wg.T) * (h @ wu.T)) @ wd.T
        del wq, wk, wv, wo, wg, wu, wd
    head = W("model.embed_tokens.weight" if raw["tie_word_embeddings"] else "lm_head.weight")
    return (_rms(torch.stack([x[-1] for x in xs]), eps) * W("model.norm.weight")) @ head.T


def _gisirax(raw, w, W, seqs):
    eps, big = raw["norm"]["eps"], raw["embedding"]["bigram"]
    xs = []
    for s in seqs:
        row = (torch.cat([s[:1] * 0, s[:-1]]) * big["mul_prev"] + s * big["mul_cur"]) % big["buckets"]
        row[0] = big["buckets"]
        xs.append(w["embed"][s].double() * raw["embedding"]["scale"] + w["bigram"][row].double())
    norm = lambda n, z: torch.tanh(W(n + ".alpha") * z) * W(n) + W(n + ".b")                    # noqa: E731
    for i, layer in enumerate(raw["layers"]):
        P = lambda n: W(f"l{i}.{n}")                                                            # noqa: E731,B023
        m, r = layer["mixer"], layer["mlp"]["router"]
        for n, x in enumerate(xs):
            h = norm(f"l{i}.norm1", x)
            T = h.shape[0]
            if layer["type"] == "channel_delta":
                H, d, e = m["heads"], m["dim"], m["vdim"]
                q, k, v = (_silu(_taps(h @ P(f"mix.{c}").T, P(f"mix.{c}.conv"))).view(T, H, -1) for c in "qkv")
                g = torch.nn.functional.softplus((h @ P("mix.a1").T) @ P("mix.a2").T + P("mix.dt_bias")).view(T, H, d)
                o = _delta(_unit(q) * d ** -0.5, _unit(k), v, torch.sigmoid(h @ P("mix.b").T), torch.exp(-P("mix.A_log").exp()[None, :, None] * g))
                gate = torch.sigmoid((h @ P("mix.g1").T) @ P("mix.g2").T).view(T, H, e)
                y = (_rms(o, eps) * P("mix.norm") * gate).reshape(T, H * e) @ P("mix.o").T
            else:
                L, R = m["left"], m["right"]
                rot, sc = L["rot"], L["rot"]["scaling"]
                f = _freqs(rot["dims"], rot["base"])
                wave = 2 * math.pi / f
                t = ((sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])).clamp(0.0, 1.0)
                f = (1 - t) * f / sc["factor"] + t * f
                q = _turned((h @ P("mix.left.q").T).view(T, L["heads"], -1), f)
                k = _turned((h @ P("mix.left.k").T).view(T, L["kv_heads"], -1), f)
                a = _attend(q, k, (h @ P("mix.left.v").T).view(T, L["kv_heads"], -1), L["scale"], sink=True).reshape(T, -1) @ P("mix.left.o").T
                q, k, v = (_silu(h @ P(f"mix.right.{c}").T).view(T, R["heads"], -1) for c in "qkv")
                o = _decay_rule(q, k, v, torch.tensor(R["decay"], device=h.device, dtype=h.dtype)[:, None]).reshape(T, -1)
                b = (_rms(o, eps) * P("mix.right.norm") * torch.sigmoid(h @ P("mix.right.g").T)) @ P("mix.right.o").T
                y = 0.5 * (_rms(a, eps) * P("mix.left.out") + _rms(b, eps) * P("mix.right.out"))
            xs[n] = x + raw["residual_mult"] * norm(f"l{i}.norm1b", y)
        # experts once for all sequences
        h = norm(f"l{i}.norm2", torch.cat(xs))
        s = torch.sigmoid(h @ P("mlp.router").T)
        grp = s.view(h.shape[0], r["groups"]["count"], -1)
        best = grp.topk(2, -1).values.sum(-1).topk(r["groups"]["keep"], -1).indices
        open_ = torch.zeros(grp.shape[:2], device=h.device, dtype=torch.bool).scatter_(1, best, True)
        top = s.masked_fill(~open_.repeat_interleave(grp.shape[2], 1), -1.0).topk(r["top"], -1)
        weight = torch.zeros_like(s).scatter_(1, top.indices, top.values / (top.values.sum(-1, keepdim=True) + 1e-20) * r["scale"])
        y = torch.zeros_like(h)
        for e in range(r["experts"]):
            at = weight[:, e].nonzero()[:, 0]
            z = _silu(h[at] @ P(f"mlp.e{e}.gate").T) * (h[at] @ P(f"mlp.e{e}.up").T)
            y[at] += weight[at, e:e + 1] * (z @ P(f"mlp.e{e}.down").T)
        y = raw["residual_mult"] * norm(f"l{i}.norm2b", y)
        xs = [x + part for x, part in zip(xs, y.split([x.shape[0] for x in xs]))]
    return norm("final.norm", torch.stack([x[-1] for x in xs])) @ W("head").T


def _lipizen(raw, w, W, seqs):
    eps, groups, cap = raw["norm"]["eps"], raw["norm"]["groups"], raw["logit_softcap"]
    norm = lambda n, z: _rms(z.view(z.shape[0], groups, -1), eps).reshape(z.shape) * W(n)       # noqa: E731
    xs, kept = [w["embed"][s].double() for s in seqs], {}
    for i, layer in enumerate(raw["layers"]):
        P = lambda n: W(f"l{i}.{n}")                                                            # noqa: E731,B023
        m, lim = layer["mixer"], layer["mlp"]["limit"]
        for n, x in enumerate(xs):
            T = x.shape[0]
            if layer["type"] == "hgrn2":
                low = P("mix.lower")
                f = (low + (1 - low) * torch.sigmoid(x @ P("mix.f").T + P("mix.f.b"))).view(T, m["heads"], -1)
                o = _decay_rule(_silu(x @ P("mix.q").T).view(f.shape), 1 - f, (x @ P("mix.v").T).view(T, m["heads"], -1), f)
                y = (_rms(o, eps) * P("mix.norm")).reshape(T, -1) @ P("mix.o").T
            else:
                H, G, d = m["heads"], m["kv_heads"], m["dim"]
                fr = _freqs(m["rot"]["dims"], m["rot"]["base"]) / m["rot"]["scaling"]["factor"]
                q = _turned(_rms(_taps(x @ P("mix.q").T, P("mix.q.conv")).view(T, H * 2, d), eps) * P("mix.q.norm"), fr).view(T, H, 2, d)
                if "kv_from" not in m:
                    k = _turned(_rms(_taps(x @ P("mix.k").T, P("mix.k.conv")).view(T, G * 2, d), eps) * P("mix.k.norm"), fr).view(T, G, 2, d)
                    kept[i, n] = k, _taps(x @ P("mix.v").T, P("mix.v.conv")).view(T, G, -1)
                k, v = kept[m.get("kv_from", i), n]
                lam = (P("mix.lq1") * P("mix.lk1")).sum().exp() - (P("mix.lq2") * P("mix.lk2")).sum().exp() + m["diff"]
                a, b = (_attend(q[:, :, c], k[:, :, c], v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"]) for c in (0, 1))
                o = _rms(a - lam * b, eps) * (1 - m["diff"]) * torch.sigmoid(x @ P("mix.g").T)[..., None]
                y = o.reshape(T, -1) @ P("mix.o").T
            x = norm(f"l{i}.norm1", raw["postln_alpha"] * x + y)
            g, u = (x @ P("mlp.gate").T).clamp(max=lim), (x @ P("mlp.up").T).clamp(-lim, lim)
            xs[n] = norm(f"l{i}.norm2", raw["postln_alpha"] * x + (g * torch.sigmoid(1.702 * g) * (u + 1)) @ P("mlp.down").T)
    return cap * torch.tanh(norm("final.norm", torch.stack([x[-1] for x in xs])) @ W("head").T / cap)


def _gudarax(raw, w, W, seqs):
    eps, side = raw["norm"]["eps"], raw["token_side"]["dim"]
    xs = [w["embed"][s].double() * raw["embedding"]["scale"] + w["pos"][:len(s)].double() for s in seqs]
    first = {}
    for i, layer in enumerate(raw["layers"]):
        P = lambda n: W(f"l{i}.{n}")                                                            # noqa: E731,B023
        m, mlp = layer["mixer"], layer["mlp"]
        for n, x in enumerate(xs):
            T = x.shape[0]
            h = _rms(x, eps) * P("norm1")
            if layer["type"] == "latent_attention":
                q = ((_rms(h @ P("mix.dq").T, eps) * P("mix.dq.norm")) @ P("mix.uq").T).view(T, m["heads"], -1)
                c = _rms(h @ P("mix.dkv").T, eps) * P("mix.dkv.norm")
                o = _attend(q, (c @ P("mix.uk").T).view(q.shape), (c @ P("mix.uv").T).view(T, m["heads"], -1), m["scale"]).reshape(T, -1)
                y = (o * torch.sigmoid(h @ P("mix.g").T)) @ P("mix.o").T
            elif layer["type"] == "delta":
                q, k, v = (_silu(_taps(h @ P(f"mix.{c}").T, P(f"mix.{c}.conv"))).view(T, m["heads"], -1) for c in "qkv")
                g = torch.exp(-P("mix.A_log").exp() * torch.nn.functional.softplus(h @ P("mix.a").T + P("mix.dt_bias")))
                o = _delta(_unit(q) * m["dim"] ** -0.5, _unit(k), v, torch.sigmoid(h @ P("mix.b").T), g[..., None])
                y = ((_rms(o, eps) * P("mix.norm")).reshape(T, -1) * _silu(h @ P("mix.g").T)) @ P("mix.o").T
            else:
                H, G = m["heads"], m["kv_heads"]
                q = (_rms(h @ P("mix.q").T + P("mix.q.b"), eps) * P("mix.q.norm")).view(T, H, -1)
                k = (_rms(h @ P("mix.k").T + P("mix.k.b"), eps) * P("mix.k.norm")).view(T, G, -1)
                v = h @ P("mix.v").T + P("mix.v.b")
                if n in first:
                    lam = P("mix.vmix")
                    v = (1 - lam) * v + lam * first[n]
                else:
                    first[n] = v
                slopes = 2.0 ** (-8.0 * torch.arange(1, H + 1, dtype=torch.float64) / H)
                y = _attend(q, k, v.view(T, G, -1), m["scale"], m["mask"]["size"], slopes=slopes).reshape(T, -1) @ P("mix.o").T
            xs[n] = x + y
        x = torch.cat(xs)
        h = _rms(x, eps) * P("norm2")
        if mlp["kind"] == "dense":
            y = (_silu(h @ P("mlp.gate").T) * (h @ P("mlp.up").T)) @ P("mlp.down").T
        else:
            s = torch.sigmoid(h @ P("mlp.router").T)
            chosen = torch.zeros_like(s, dtype=torch.bool).scatter_(1, s.topk(mlp["router"]["top"], -1).indices, True)
            y = torch.zeros_like(h)
            for e in range(mlp["router"]["experts"]):
                at = chosen[:, e].nonzero()[:, 0]
                y[at] += ((s[at, e:e + 1] * h[at]) @ P(f"mlp.e{e}.up").T).clamp(min=0.0).square() @ P(f"mlp.e{e}.down").T
        x = x + y
        e = w["side.embed"][torch.cat(seqs)][:, i * side:(i + 1) * side].double()
        z = torch.nn.functional.gelu(x @ P("side.gate").T, approximate="tanh") * e
        x = x + _rms(z @ P("side.proj").T, eps) * P("side.norm")
        xs = list(x.split([len(s) for s in seqs]))
    return (_rms(torch.stack([x[-1] for x in xs]), eps) * W("final.norm")) @ W("head").T
