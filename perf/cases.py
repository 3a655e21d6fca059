"""The work that janis_b200 is measured on: steps of whole models through `Engine.step`.

A case is a model at the 2B layer sizes with random weights and one kind of step:

* decode:  every sequence of a batch, brought to its length by prompt steps before, takes one token and gives its
  logits.  A pass is one step, so a sequence grows by a token a pass; where it has no room left, sequences of the
  first lengths take the place of the old ones, as they do in a server.
* prompt:  new sequences bring their whole prompts and get the logits behind them.
* pieces:  one new prompt comes in pieces, as a long document or a conversation does; logits behind the last one.

Gemma2 runs all of its 26 layers.  Sigalorn and Nosolix run four layers of the same width, which hold each of their
mixers twice (attention with mixed heads and gated linear attention; window attention beside a state-space-duality
mixer and a selective scan), with dense feed-forwards: a mixture's choice of experts may turn on the last bit of
a bfloat16, after which no two correct programs give comparable logits.

`exact` states the three models in 64-bit torch operations.  The weights are drawn by the published rule of
`janis_b200.from_config` (a hash of seed, tensor name and element), written out here once more.
"""
from __future__ import annotations

import hashlib
import math
import random

import torch

import janis_b200
from janis_b200 import StepEntry

WIDTH, VOCAB, FF, HEADS, KV_HEADS, HEAD = 2304, 256000, 9216, 8, 4, 256
GEMMA_LAYERS, OTHER_LAYERS, WINDOW, MOST_CONTEXT = 26, 4, 4096, 8192
ROOM = 1024                     # tokens that a sequence of a decode case can still take


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def _case(name, model, kind, batch, low, high, dtype="bfloat16", pieces=1):
    """`batch` sequences of lengths spread over [low, high]."""
    c = {"model": model, "kind": kind, "dtype": dtype, "batch": batch, "low": low, "high": high, "pieces": pieces}
    return dict(c, name=name) if name else c


def listed():
    return [
        _case("gemma2-decode-1", "gemma2", "decode", 1, 1024, 1024),              # one user waits for each token
        _case("gemma2-decode-8-long", "gemma2", "decode", 8, 7168, 7168),         # a small batch near the model's longest context
        _case("gemma2-decode-64", "gemma2", "decode", 64, 128, 2048),             # a server's batch of unequal conversations
        _case("gemma2-prompt-2048", "gemma2", "prompt", 1, 2048, 2048),           # the time to the first token of a usual prompt
        _case("gemma2-prompt-short", "gemma2", "prompt", 3, 19, 150),             # a few questions of a line or two together
        _case("gemma2-prompt-batch", "gemma2", "prompt", 8, 64, 4096),            # a batch of documents and questions mixed
        _case("gemma2-pieces", "gemma2", "pieces", 1, 4001, 4001, pieces=4),      # a long prompt that comes in pieces
        _case("gemma2-prompt-float32", "gemma2", "prompt", 3, 40, 300, dtype="float32"),   # reference logits in true 32-bit
        _case("sigalorn-prompt-2048", "sigalorn", "prompt", 1, 2048, 2048),
        _case("sigalorn-decode-8", "sigalorn", "decode", 8, 3000, 3000),
        _case("nosolix-prompt-2048", "nosolix", "prompt", 1, 2048, 2048),
        _case("nosolix-decode-8", "nosolix", "decode", 8, 3000, 3000),
    ]


def _spread(rng, lo, hi):
    """A whole number from [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    model = rng.choice(["gemma2", "gemma2", "sigalorn", "nosolix"])
    kind = rng.choice(["decode", "prompt", "prompt", "pieces"] if model == "gemma2" else ["decode", "prompt"])
    if kind == "decode":
        batch = _spread(rng, 1, 64)
        longest = min(7168 if model == "gemma2" else 3072, 65536 // batch)
        high = _spread(rng, 64, longest)
    elif kind == "prompt":
        batch = _spread(rng, 1, 8)
        high = _spread(rng, 17, min(4096, 16384 // batch) if model == "gemma2" else min(3072, 6144 // batch))
    else:
        batch, high = 1, _spread(rng, 300, 6000)
    low = high if batch == 1 else rng.randint(max(1, high // 16), high)
    dtype = "bfloat16"
    if model == "gemma2" and kind == "prompt" and batch * high <= 1200 and rng.random() < 0.25:
        dtype = "float32"
    return _case(None, model, kind, batch, low, high, dtype, rng.randint(2, 6) if kind == "pieces" else 1)


def _lengths(case):
    """The sequences' lengths: the same for every seed, the longest among them."""
    rng = random.Random("%d %d %d" % (case["batch"], case["low"], case["high"]))
    return [case["high"]] + [rng.randint(case["low"], case["high"]) for _ in range(case["batch"] - 1)]


def _piece_lengths(case):
    """Unequal pieces that add up to the prompt."""
    n, k = case["high"], case["pieces"]
    rng = random.Random("%d %d" % (n, k))
    cuts = sorted(rng.sample(range(1, n), k - 1)) if k > 2 else [n // 2 + 1]
    cuts = [max(1, (c + n * (i + 1) // k) // 2) for i, c in enumerate(cuts)]
    ends = sorted(set(cuts)) + [n]
    return [b - a for a, b in zip([0] + ends[:-1], ends)]


def _config(case):
    if case["model"] == "gemma2":
        return {"architectures": ["Gemma2ForCausalLM"], "model_type": "gemma2", "hidden_size": WIDTH, "head_dim": HEAD,
                "intermediate_size": FF, "num_attention_heads": HEADS, "num_key_value_heads": KV_HEADS,
                "num_hidden_layers": GEMMA_LAYERS, "vocab_size": VOCAB, "sliding_window": WINDOW, "rope_theta": 10000.0,
                "rms_norm_eps": 1e-6, "query_pre_attn_scalar": HEAD, "attn_logit_softcapping": 50.0,
                "final_logit_softcapping": 30.0, "max_position_embeddings": MOST_CONTEXT, "eos_token_id": 1,
                "hidden_activation": "gelu_pytorch_tanh", "tie_word_embeddings": True, "torch_dtype": "bfloat16"}
    att = {"heads": HEADS, "kv_heads": KV_HEADS, "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5, "mask": {"size": WINDOW}}
    mlp = {"kind": "dense", "ff": FF}
    layers = []
    for i in range(OTHER_LAYERS):
        if case["model"] == "sigalorn":
            if i % 2:
                mixer = {"heads": HEADS, "dim": HEAD // 2, "vdim": HEAD, "tau": 16.0, "rank": 64}
            else:
                mixer = dict(att, rot={"base": 10000.0, "dims": HEAD}, **({"kv_from": i - 2} if i % 4 == 2 else {}))
            layers.append({"type": "gla" if i % 2 else "attention", "mixer": mixer, "mlp": dict(mlp)})
        else:
            scaling = {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}
            left = dict(att, rot={"base": 10000.0, "dims": HEAD, "scaling": scaling})
            right = {"heads": 2 * WIDTH // 64, "vdim": 64, "state": 128, "groups": 1, "norm_groups": 1, "conv": 4}
            scan = {"inner": 2 * WIDTH, "state": 16, "dt_rank": WIDTH // 16, "conv": 4}
            layers.append({"type": "mamba1", "mixer": scan, "mlp": dict(mlp)} if i % 2 else
                          {"type": "parallel", "mixer": {"left": left, "right": right}, "mlp": dict(mlp)})
    c = {"vocab": VOCAB, "width": WIDTH, "embedding": {"scale": 1.0}, "norm": {"eps": 1e-6}, "layers": layers}
    if case["model"] == "sigalorn":
        return dict(c, architecture="Sigalorn", logit_softcap=30.0)
    return dict(c, architecture="Nosolix")


def _tokens(case, seed):
    """Per sequence its token ids (a decode case: and the ids that it is given later)."""
    more = ROOM if case["kind"] == "decode" else 0
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(2, VOCAB, (n + more,), generator=g).tolist() for n in _lengths(case)]


# ---------------------------------------------------------------------------
# a pass
# ---------------------------------------------------------------------------

def prepare(case, seed):
    lens = _lengths(case)
    more = ROOM if case["kind"] == "decode" else 0
    pages = sum((n + more + 63) // 64 * 64 for n in lens)
    engine = janis_b200.from_config(_config(case), seed=seed, dtype=case["dtype"], max_tokens=pages,
                                    max_batch=case["batch"], max_context=max(lens) + more)
    state = {"engine": engine, "case": case, "lens": lens, "tokens": _tokens(case, seed)}
    if case["kind"] == "decode":
        _fill(state)
    return state


def _fill(state):
    """Sequences of the first lengths, by prompt steps that ask for nothing."""
    engine, part, count = state["engine"], [], 0
    state["slots"] = [engine.alloc_slot() for _ in state["lens"]]
    state["done"] = 0
    for slot, n, toks in zip(state["slots"], state["lens"], state["tokens"]):
        if part and count + n > 16384:
            engine.step(part)
            part, count = [], 0
        part.append(StepEntry(slot, toks[:n], ()))
        count += n
    engine.step(part)


def run(state):
    engine, case, lens, tokens = state["engine"], state["case"], state["lens"], state["tokens"]
    if case["kind"] == "decode":
        if state["done"] == ROOM:
            for s in state["slots"]:
                engine.free_slot(s)
            _fill(state)
        k = state["done"]
        state["done"] = k + 1
        return engine.step([StepEntry(s, (t[n + k],), (0,)) for s, n, t in zip(state["slots"], lens, tokens)])
    slots = [engine.alloc_slot() for _ in lens]
    if case["kind"] == "prompt":
        logits = engine.step([StepEntry(s, t, (len(t) - 1,)) for s, t in zip(slots, tokens)])
    else:
        at = 0
        for n in _piece_lengths(case):
            last = at + n == lens[0]
            logits = engine.step([StepEntry(slots[0], tokens[0][at:at + n], (n - 1,) if last else ())])
            at += n
    for s in slots:
        engine.free_slot(s)
    return logits


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    """Every weight read once, the cache's keys, values and states that the step needs read (and states written) once,
    the logits written once; two operations a weight and token, and the attention's and the scans' own."""
    lens, item = _lengths(case), 2 if case["dtype"] == "bfloat16" else 4
    decode = case["kind"] == "decode"
    new = len(lens) if decode else sum(lens)
    matrices = 0
    for name, (shape, _, _) in _specs(case).items():
        if len(shape) == 2 and "embed" not in name and name != "head":
            matrices += shape[0] * shape[1]
    head = VOCAB * WIDTH
    kv = 2 * KV_HEADS * HEAD
    state, steps = 0, 0.0           # floats of state a sequence, operations a token on them
    n_att = {"gemma2": GEMMA_LAYERS, "sigalorn": OTHER_LAYERS // 2, "nosolix": OTHER_LAYERS // 2}[case["model"]]
    if case["model"] == "sigalorn":
        state = OTHER_LAYERS // 2 * HEADS * (HEAD // 2) * HEAD
        steps = 5.0 * state
    elif case["model"] == "nosolix":
        state = OTHER_LAYERS // 2 * 2 * WIDTH * (128 + 16)
        steps = 6.0 * state
    seen = cached = 0
    for i in range(n_att):
        window = WINDOW if case["model"] != "gemma2" or i % 2 == 0 else MOST_CONTEXT
        for n in lens:
            m = min(n + decode, window)
            seen += m if decode else m * (m + 1) // 2 + (n - m) * m
            if not (case["model"] == "sigalorn" and i % 2):         # (the second reads what the first one keeps)
                cached += m * kv
    rows = len(lens)
    nbytes = (matrices + head) * item + cached * item + new * WIDTH * item + rows * VOCAB * 4
    nbytes += rows * state * 4 * (2 if decode else 1)
    flops = 2.0 * matrices * new + 2.0 * head * rows + 4.0 * seen * HEADS * HEAD + steps * new
    if case["model"] == "sigalorn":
        flops += 2.0 * seen * HEADS * HEADS
    return {"bytes": float(nbytes), "flops": flops}


def tolerance(case):
    # Against 64 bits the logits are off by 0.005 to 0.011 in bfloat16 and by 4e-6 in float32 (2-norms); two correct
    # implementations may each be off by as much in directions of their own.
    return {"rel": 3e-5, "max": 3e-4} if case["dtype"] == "float32" else {"rel": 0.025, "max": 0.25}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def exact(case, seed):
    lens = _lengths(case)
    total = sum(lens)
    # 64-bit products of 2.6e9 weights, or a loop over the tokens of four layers: about 20 seconds
    if (case["model"] == "gemma2" and total > 70000) or (case["model"] != "gemma2" and total > 40000):
        return None
    take = 1 if case["kind"] == "decode" else 0
    seqs = [t[:n + take] for t, n in zip(_tokens(case, seed), lens)]
    w = _Weights(_specs(case), seed)
    forward = {"gemma2": _gemma2, "sigalorn": _sigalorn, "nosolix": _nosolix}[case["model"]]
    return forward(_config(case), w, [torch.tensor(s, device="cuda") for s in seqs])


F = torch.float64


def _specs(case):
    """Tensor name -> (shape, standard deviation, mean) of the random weights."""
    s = {}
    if case["model"] == "gemma2":
        s["model.embed_tokens.weight"] = ((VOCAB, WIDTH), 0.02, 0.0)
        for i in range(GEMMA_LAYERS):
            p = "model.layers.%d." % i
            for n in ("input_layernorm", "post_attention_layernorm", "pre_feedforward_layernorm", "post_feedforward_layernorm"):
                s[p + n + ".weight"] = ((WIDTH,), 0.1, 0.0)
            for n, rows, cols in (("self_attn.q", HEADS * HEAD, WIDTH), ("self_attn.k", KV_HEADS * HEAD, WIDTH),
                                  ("self_attn.v", KV_HEADS * HEAD, WIDTH), ("self_attn.o", WIDTH, HEADS * HEAD),
                                  ("mlp.gate", FF, WIDTH), ("mlp.up", FF, WIDTH), ("mlp.down", WIDTH, FF)):
                s[p + n + "_proj.weight"] = ((rows, cols), 0.02, 0.0)
        s["model.norm.weight"] = ((WIDTH,), 0.1, 0.0)
        return s
    s["embed"] = ((VOCAB, WIDTH), 1.0, 0.0)
    s["head"] = ((VOCAB, WIDTH), 1.0 / math.sqrt(WIDTH), 0.0)
    sig = case["model"] == "sigalorn"

    def norm(n):
        s[n] = ((WIDTH,), 0.3, 1.0) if sig else ((WIDTH,), 0.1, 1.0)
        if not sig:
            s[n + ".b"], s[n + ".alpha"] = ((WIDTH,), 0.1, 0.0), ((), 0.05, 0.5)

    def matrix(n, rows, cols, std=0.02, mean=0.0):
        s[n] = ((rows, cols), std, mean)

    def vector(n, size, std, mean=0.0):
        s[n] = ((size,), std, mean)

    norm("final.norm")
    for i, layer in enumerate(_config(case)["layers"]):
        p, m = "l%d." % i, layer["mixer"]
        norm(p + "norm1")
        norm(p + "norm2")
        matrix(p + "mlp.up", FF, WIDTH)
        matrix(p + "mlp.down", WIDTH, FF)
        x = p + "mix."
        if sig:
            norm(p + "norm1b")
            norm(p + "norm2b")
            vector(p + "mlp.up.b", FF, 0.02)
            vector(p + "mlp.down.b", WIDTH, 0.02)
            vector(p + "mlp.act", 2, 0.5)
        if layer["type"] == "gla":
            d = m["heads"] * m["dim"]
            for n, rows in (("q", d), ("k", d), ("v", HEADS * HEAD), ("g", HEADS * HEAD)):
                matrix(x + n, rows, WIDTH)
            matrix(x + "o", WIDTH, HEADS * HEAD)
            matrix(x + "a1", m["rank"], WIDTH)
            matrix(x + "a2", d, m["rank"], 0.2)
            vector(x + "a2.b", d, 1.0)
            vector(x + "norm", HEAD, 0.1)
        elif layer["type"] == "mamba1":
            inner, N, R = m["inner"], m["state"], m["dt_rank"]
            matrix(x + "in", 2 * inner, WIDTH)
            matrix(x + "conv", inner, m["conv"], 0.3)
            vector(x + "conv.b", inner, 0.1)
            matrix(x + "x", R + 2 * N, inner)
            matrix(x + "dt", inner, R, 1.0 / math.sqrt(R))
            vector(x + "dt.b", inner, 1.0, -2.0)
            matrix(x + "A_log", inner, N, 0.5)
            vector(x + "D", inner, 0.5, 1.0)
            matrix(x + "o", WIDTH, inner)
        else:
            if not sig:
                r = m["right"]
                inner, N = r["heads"] * r["vdim"], r["state"]
                vector(x + "left.out", WIDTH, 0.1, 1.0)
                vector(x + "right.out", WIDTH, 0.1, 1.0)
                y = x + "right."
                matrix(y + "in", 2 * inner + 2 * N + r["heads"], WIDTH)
                matrix(y + "conv", inner + 2 * N, r["conv"], 0.3)
                vector(y + "conv.b", inner + 2 * N, 0.1)
                vector(y + "dt_bias", r["heads"], 1.0, -1.0)
                vector(y + "A_log", r["heads"], 0.5)
                vector(y + "D", r["heads"], 0.5, 1.0)
                vector(y + "norm", inner, 0.1, 1.0)
                matrix(y + "o", WIDTH, inner)
                x += "left."
                matrix(x + "g", HEADS * HEAD, WIDTH)
            else:
                matrix(x + "talk", HEADS, HEADS, HEADS ** -0.5)
            matrix(x + "q", HEADS * HEAD, WIDTH)
            matrix(x + "o", WIDTH, HEADS * HEAD)
            if m.get("kv_from") is None:
                matrix(x + "k", KV_HEADS * HEAD, WIDTH)
                matrix(x + "v", KV_HEADS * HEAD, WIDTH)
    return s


def _signed(c):
    c &= (1 << 64) - 1
    return c - (1 << 64) if c >> 63 else c


class _Weights:
    """The random weights of a seed as 64-bit tensors, drawn when asked for."""

    def __init__(self, specs, seed):
        self.specs, self.seed = specs, seed

    def bf16(self, name):
        shape, std, mean = self.specs[name]
        digest = hashlib.sha256(("%d:%s" % (self.seed, name)).encode()).digest()
        key = (int.from_bytes(digest[:8], "little") & ((1 << 63) - 1)) >> 3
        n, out = math.prod(shape), []
        for a in range(0, n, 1 << 24):
            i = torch.arange(a, min(n, a + (1 << 24)), device="cuda", dtype=torch.int64) * 4
            total = torch.zeros_like(i)
            for j in (1, 2, 3):
                z = (i + (j + key)) * _signed(0x9E3779B97F4A7C15)
                z = (z ^ ((z >> 30) & 0x3FFFFFFFF)) * _signed(0xBF58476D1CE4E5B9)
                z = (z ^ ((z >> 27) & 0x1FFFFFFFFF)) * _signed(0x94D049BB133111EB)
                z = z ^ ((z >> 31) & 0x1FFFFFFFF)
                for shift in (0, 16, 32, 48):
                    total += (z >> shift) & 0xFFFF
            x = (total - 6 * 65535).to(torch.float32) * (1.0 / 65536.0) * std
            out.append((x + mean if mean else x).to(torch.bfloat16))
        return torch.cat(out).view(shape)

    def __getitem__(self, name):
        return self.bf16(name).to(F)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _softplus(x):
    return torch.logaddexp(x, torch.zeros_like(x))


def _silu(x):
    return x * torch.sigmoid(x)


def _turn(x, pos, freq):
    """x [T, heads, n]: pairs (i, i + len(freq)) turned by pos * freq."""
    h = freq.numel()
    a = pos.to(F)[:, None, None] * freq.to(F)[None, None, :]
    c, s = torch.cos(a), torch.sin(a)
    u, v = x[..., :h], x[..., h:2 * h]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * h:]], dim=-1)


def _frequencies(rot):
    out = []
    for i in range(rot["dims"] // 2):
        f, sc = rot["base"] ** (-2.0 * i / rot["dims"]), rot.get("scaling")
        if sc:
            wave = 2.0 * math.pi / f
            if wave > sc["original"] / sc["low"]:
                f = f / sc["factor"]
            elif wave >= sc["original"] / sc["high"]:
                t = (sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])
                f = (1.0 - t) * f / sc["factor"] + t * f
        out.append(f)
    return torch.tensor(out, dtype=F, device="cuda")


def _window_attention(q, k, v, scale, window, cap=0.0):
    """q [T, heads, n], k and v [T, kv heads, n]: causal softmax over the last `window` positions (0: all)."""
    T, H = q.shape[:2]
    i = torch.arange(T, device=q.device)
    out = torch.empty_like(q)
    for a in range(0, T, 1024):                     # queries at a time
        rows = i[a:a + 1024, None]
        unseen = i[None, :] > rows
        if window:
            unseen |= i[None, :] <= rows - window
        for h in range(H):
            g = h // (H // k.shape[1])
            s = q[a:a + 1024, h] @ k[:, g].T * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            out[a:a + 1024, h] = torch.softmax(s.masked_fill(unseen, -math.inf), -1) @ v[:, g]
    return out


def _gemma2(cfg, w, seqs):
    eps = cfg["rms_norm_eps"]
    table = w.bf16("model.embed_tokens.weight")
    xs = [table[t].to(F) * math.sqrt(WIDTH) for t in seqs]
    i = torch.arange(HEAD // 2, dtype=F, device="cuda")
    freq = (cfg["rope_theta"] ** (-2.0 * i / HEAD)).to(torch.float32)
    ends = torch.tensor([0] + [x.shape[0] for x in xs]).cumsum(0).tolist()
    x = torch.cat(xs)

    def norm(x, name):
        return _rms(x, eps) * (1.0 + w[name])

    for n in range(GEMMA_LAYERS):
        p = "model.layers.%d." % n
        last = n == GEMMA_LAYERS - 1
        wq, wk, wv, wo = (w[p + "self_attn.%s_proj.weight" % c] for c in "qkvo")
        parts, keep = [], []
        for a, b in zip(ends, ends[1:]):
            y = norm(x[a:b], p + "input_layernorm.weight")
            pos = torch.arange(b - a, device="cuda")
            # angles are products of 32-bit numbers
            ang = (pos.to(torch.float32)[:, None] * freq[None, :]).to(F)[:, None, :]
            c, s = torch.cos(ang), torch.sin(ang)

            def turned(m, heads):
                z = (y @ m.T).view(b - a, heads, HEAD)
                u, v = z[..., :HEAD // 2], z[..., HEAD // 2:]
                return torch.cat([u * c - v * s, v * c + u * s], -1)

            q, k, v = turned(wq, HEADS), turned(wk, KV_HEADS), (y @ wv.T).view(b - a, KV_HEADS, HEAD)
            o = _window_attention(q, k, v, cfg["query_pre_attn_scalar"] ** -0.5, WINDOW if n % 2 == 0 else 0,
                                  cfg["attn_logit_softcapping"])
            parts.append(o.reshape(b - a, HEADS * HEAD) @ wo.T)
            keep.append(b - 1)
        x = x + norm(torch.cat(parts), p + "post_attention_layernorm.weight")
        if last:
            x = x[keep]
        gate, up, down = (w[p + "mlp.%s_proj.weight" % c] for c in ("gate", "up", "down"))
        out = []
        for part in x.split(8192):
            y = norm(part, p + "pre_feedforward_layernorm.weight")
            z = y @ gate.T
            z = 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))
            out.append(part + norm((z * (y @ up.T)) @ down.T, p + "post_feedforward_layernorm.weight"))
        x = torch.cat(out)
    cap = cfg["final_logit_softcapping"]
    return cap * torch.tanh(_project(norm(x, "model.norm.weight"), table) / cap)


def _project(y, table):
    return torch.cat([y @ t.to(F).T for t in table.split(32768)], -1)


def _in_blocks(ws, names):
    return {n: ws[n] for n in names}


def _others(cfg, w, seqs, norm, mix, ff):
    """The frame that Sigalorn and Nosolix share: one sequence after another, the weights of a layer at a time."""
    xs = [w.bf16("embed")[t].to(F) for t in seqs]
    kept = {}
    for i, layer in enumerate(cfg["layers"]):
        p = "l%d." % i
        ws = _in_blocks(w, [n for n in w.specs if n.startswith(p)])
        last = i == len(cfg["layers"]) - 1
        for n, x in enumerate(xs):
            xs[n] = ff(mix(x, ws, p, i, layer, kept, n), ws, p, last)
    y = norm(torch.cat(xs), _in_blocks(w, [n for n in w.specs if n.startswith("final.")]), "final.norm")
    logits = _project(y, w.bf16("head"))
    cap = cfg.get("logit_softcap", 0.0)
    return cap * torch.tanh(logits / cap) if cap else logits


def _sigalorn(cfg, w, seqs):
    eps = cfg["norm"]["eps"]

    def norm(x, ws, n):
        return _rms(x, eps) * ws[n]

    def mix(x, ws, p, i, layer, kept, n):
        m, q_ = layer["mixer"], p + "mix."
        y = norm(x, ws, p + "norm1")
        T, H = x.shape[0], m["heads"]
        if layer["type"] == "gla":
            d, dv = m["dim"], m["vdim"]
            q, k, v = ((y @ ws[q_ + c].T).view(T, H, -1) for c in "qkv")
            z = (y @ ws[q_ + "a1"].T) @ ws[q_ + "a2"].T + ws[q_ + "a2.b"]
            alpha = torch.exp(-_softplus(-z) / m["tau"]).view(T, H, d, 1)
            S, o = torch.zeros(H, d, dv, dtype=F, device=x.device), torch.empty(T, H, dv, dtype=F, device=x.device)
            k, v, q = k[..., None], v[:, :, None, :], q[:, :, None, :] / math.sqrt(d)
            for t in range(T):
                S = torch.addcmul(alpha[t] * S, k[t], v[t])
                torch.matmul(q[t], S, out=o[t].unsqueeze(1))
            o = (_rms(o, eps) * ws[q_ + "norm"]).reshape(T, H * dv) * _silu(y @ ws[q_ + "g"].T)
        else:
            G, size = m["kv_heads"], m["mask"]["size"]
            pos, freq = torch.arange(T, device=x.device), _frequencies(m["rot"])
            if m.get("kv_from") is None:
                kept[n] = [_turn((y @ ws[q_ + c].T).view(T, G, HEAD), pos, freq) for c in "kv"]
            k, v = kept[n]                                     # (four layers: one writes, one reads)
            q = _turn((y @ ws[q_ + "q"].T).view(T, H, HEAD), pos, freq)
            kh, vh = k.repeat_interleave(H // G, 1).transpose(0, 1), v.repeat_interleave(H // G, 1).transpose(0, 1)
            o = torch.empty(T, H, HEAD, dtype=F, device=x.device)
            for a in range(0, T, 1024):
                s = q[a:a + 1024].transpose(0, 1) @ kh.transpose(1, 2) * m["scale"]
                s = torch.einsum("hg,gij->hij", ws[q_ + "talk"], s)
                rows = pos[a:a + 1024, None]
                seen = (pos[None, :] <= rows) & (pos[None, :] // size == rows // size)
                e = torch.exp(s) * seen[None]
                o[a:a + 1024] = ((e / (1.0 + e.sum(-1, keepdim=True))) @ vh).transpose(0, 1)
            o = _turn(o, -pos, freq).reshape(T, H * HEAD)
        return x + norm(o @ ws[q_ + "o"].T, ws, p + "norm1b")

    def ff(x, ws, p, last):
        x = x[-1:] if last else x
        a, b = (_softplus(c) for c in ws[p + "mlp.act"])
        z = norm(x, ws, p + "norm2") @ ws[p + "mlp.up"].T + ws[p + "mlp.up.b"]
        z = torch.where(z > 0, a * z * z + 0.5 * z, (0.5 + b) * (torch.expm1(z.clamp(max=0.0)) - z) + 0.5 * z)
        return x + norm(z @ ws[p + "mlp.down"].T + ws[p + "mlp.down.b"], ws, p + "norm2b")

    return _others(cfg, w, seqs, norm, mix, ff)


def _conv(x, kernel, bias):
    T, taps = x.shape[0], kernel.shape[1]
    out = bias.expand_as(x).clone()
    for j in range(min(taps, T)):
        out[j:] += kernel[:, taps - 1 - j] * x[:T - j]
    return _silu(out)


def _nosolix(cfg, w, seqs):
    eps = cfg["norm"]["eps"]

    def norm(x, ws, n):
        return torch.tanh(ws[n + ".alpha"] * x) * ws[n] + ws[n + ".b"]

    def scan(y, ws, q, m):
        inner, N, R, T = m["inner"], m["state"], m["dt_rank"], y.shape[0]
        u, z = (y @ ws[q + "in"].T).split(inner, -1)
        u = _conv(u, ws[q + "conv"], ws[q + "conv.b"])
        lo, B, C = (u @ ws[q + "x"].T).split([R, N, N], -1)
        delta = _softplus(lo @ ws[q + "dt"].T + ws[q + "dt.b"])
        A, du = -torch.exp(ws[q + "A_log"]), (delta * u)[..., None]
        S, o = torch.zeros(inner, N, dtype=F, device=y.device), torch.empty(T, inner, dtype=F, device=y.device)
        for t in range(T):
            S = torch.addcmul(torch.exp(delta[t][:, None] * A) * S, du[t], B[t][None, :])
            torch.mv(S, C[t], out=o[t])
        return ((o + ws[q + "D"] * u) * _silu(z)) @ ws[q + "o"].T

    def duality(y, ws, q, m):
        H, P, N, T = m["heads"], m["vdim"], m["state"], y.shape[0]
        z, u, B, C, dt = (y @ ws[q + "in"].T).split([H * P, H * P, N, N, H], -1)
        u, B, C = _conv(torch.cat([u, B, C], -1), ws[q + "conv"], ws[q + "conv.b"]).split([H * P, N, N], -1)
        u = u.reshape(T, H, P)
        delta = _softplus(dt + ws[q + "dt_bias"])
        decay = torch.exp(-torch.exp(ws[q + "A_log"]) * delta)[:, None, :, None]
        du = (delta[..., None] * u)[:, None]
        S, o = torch.zeros(N, H, P, dtype=F, device=y.device), torch.empty(T, H * P, dtype=F, device=y.device)
        B = B[:, :, None, None]
        for t in range(T):
            S = torch.addcmul(decay[t] * S, B[t], du[t])
            torch.mv(S.view(N, H * P).T, C[t], out=o[t])
        o = (o.view(T, H, P) + ws[q + "D"][:, None] * u).reshape(T, H * P) * _silu(z)
        return (_rms(o, eps) * ws[q + "norm"]) @ ws[q + "o"].T

    def mix(x, ws, p, i, layer, kept, n):
        m, q_ = layer["mixer"], p + "mix."
        y = norm(x, ws, p + "norm1")
        if layer["type"] == "mamba1":
            return x + scan(y, ws, q_, m)
        T, left, l_ = x.shape[0], m["left"], q_ + "left."
        pos, freq = torch.arange(T, device=x.device), _frequencies(left["rot"])
        q = _turn((y @ ws[l_ + "q"].T).view(T, HEADS, HEAD), pos, freq)
        k = _turn((y @ ws[l_ + "k"].T).view(T, KV_HEADS, HEAD), pos, freq)
        v = (y @ ws[l_ + "v"].T).view(T, KV_HEADS, HEAD)
        o = _window_attention(q, k, v, left["scale"], left["mask"]["size"]).reshape(T, HEADS * HEAD)
        a = (o * torch.sigmoid(y @ ws[l_ + "g"].T)) @ ws[l_ + "o"].T
        b = duality(y, ws, q_ + "right.", m["right"])
        return x + 0.5 * (_rms(a, eps) * ws[l_ + "out"] + _rms(b, eps) * ws[q_ + "right.out"])

    def ff(x, ws, p, last):
        x = x[-1:] if last else x
        return x + torch.relu(norm(x, ws, p + "norm2") @ ws[p + "mlp.up"].T) ** 2 @ ws[p + "mlp.down"].T

    return _others(cfg, w, seqs, norm, mix, ff)
