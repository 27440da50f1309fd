"""What the speed of the library is measured on: generation and replay through `Engine.step` and `Sampler.sample`.

A case is a model (by the name of its shape), a data type, the prompts of one or more turns and the number of single-token
steps after each of them.  One pass takes the sequences through all of it: slots, the prompts' step, the single tokens, the
slots given back.  Weights and token ids are made on the GPU from the seed; sizes come from the case alone.

    feed "greedy", "sampled"   the sampled ids go into the next step on the device, as the generation loop has it
                               ("sampled": temperature 0.8, top-k 40, top-p 0.95)
    feed "given"               the ids of every step come from the host, as in a replay or an evaluation
    want "last", "all"         the logits a prompt's step forms

The Gemma 2 weights make a token's own logit the largest by far (the norms after the branches have small weights), so that
what is sampled does not hang on rounding; the experts' last matrices are small for the same reason (a choice that rounding
turns changes little).  Neither changes what a step computes or reads.
"""
from __future__ import annotations

import math

import torch

from rust_deeplearning_b200 import Engine, SamplingParams
from rust_deeplearning_b200.config.base import architecture_for
from rust_deeplearning_b200.parts.model import Model
from rust_deeplearning_b200.sampling.sampler import Sampler

DEVICE = "cuda:0"
CONTEXT = 8192
L2_BYTES = 126e6

# ---- the shapes ----

GEMMA2_2B = {
    "architectures": ["Gemma2ForCausalLM"], "model_type": "gemma2", "num_hidden_layers": 26, "hidden_size": 2304,
    "num_attention_heads": 8, "num_key_value_heads": 4, "head_dim": 256, "intermediate_size": 9216, "vocab_size": 256000,
    "rms_norm_eps": 1e-6, "rope_theta": 10000.0, "sliding_window": 4096, "query_pre_attn_scalar": 256,
    "attn_logit_softcapping": 50.0, "final_logit_softcapping": 30.0, "max_position_embeddings": CONTEXT,
    "hidden_activation": "gelu_pytorch_tanh", "tie_word_embeddings": True, "bos_token_id": 2, "eos_token_id": 1,
}
GEMMA2_9B = dict(GEMMA2_2B, num_hidden_layers=42, hidden_size=3584, num_attention_heads=16, num_key_value_heads=8,
                 intermediate_size=14336)
# three layers, one key/value head, heads that do not add up to the width: the shape whose logits are compared in 32 bits
GEMMA2_TINY = dict(GEMMA2_2B, num_hidden_layers=3, hidden_size=96, num_attention_heads=6, num_key_value_heads=1, head_dim=32,
                   intermediate_size=160, vocab_size=384, rope_theta=1e6, sliding_window=16, query_pre_attn_scalar=24,
                   attn_logit_softcapping=20.0, final_logit_softcapping=15.0, max_position_embeddings=512)


def _gasetar():
    """Window attention with a norm over the projections, latent attention with sinks, 64 experts of 1,024 beside a shared one."""
    attn = {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 50.0, "mask": {"size": 4096},
            "rot": {"base": 100000.0, "dims": 96, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
    latent = {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5, "rot": {"base": 10000.0, "dims": 64}}
    moe = {"kind": "moe", "expert": {"ff": 1024}, "router": {"experts": 64, "top": 6}, "shared": {"ff": 2304}}
    order = [("attention", attn, {"kind": "dense", "ff": 8448}), ("latent_attention", latent, moe), ("attention", attn, moe), ("attention", attn, moe)]
    return {"architecture": "Gasetar", "width": 2048, "vocab": 32000, "norm": {"eps": 1e-6}, "embedding": {"scale": 2048 ** 0.5},
            "residual_mult": 0.5, "logit_scale": 1.0, "logit_softcap": 30.0, "max_positions": CONTEXT,
            "layers": [{"type": t, "mixer": m, "mlp": f} for t, m, f in order]}


def _dokulorn():
    """Three retention layers and a pair (softmax attention with sinks beside lightning attention), dense feed-forwards of 8,192."""
    decay = [1.0 - 2.0 ** (-5 - 5 * h / 15) for h in range(16)]
    ret = {"heads": 16, "dim": 128, "vdim": 128, "decay": decay, "rot": {"base": 1e6, "dims": 128}}
    par = {"left": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "rot": {"base": 1e4, "dims": 64}, "scale": 1.0, "softcap": 20.0},
           "right": {"heads": 16, "dim": 128, "vdim": 128, "decay": decay}}
    return {"architecture": "Dokulorn", "width": 2048, "vocab": 32000, "norm": {"eps": 1e-6}, "postln_alpha": 2.0, "embedding": {"scale": 10.0},
            "max_positions": CONTEXT, "layers": [{"type": "parallel" if i == 3 else "retention", "mixer": par if i == 3 else ret,
                                                  "mlp": {"kind": "dense", "ff": 8192}} for i in range(4)]}


def _revepel():
    """State space, delta rule, sigmoid-weight attention, the same on shared keys; 32 two-matrix experts of 1,024 beside a shared one."""
    rot = {"base": 10000.0, "dims": 128, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
    mlp = {"kind": "moe", "expert": {"ff": 1024}, "router": {"experts": 32, "top": 4}, "shared": {"ff": 4096}}
    attn = {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 4096}, "rot": rot}
    mixers = [("mamba2", {"heads": 32, "vdim": 64, "state": 128, "groups": 1, "norm_groups": 1, "conv": 4}),
              ("channel_delta", {"heads": 16, "kv_heads": 16, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64, "gate_rank": 64}),
              ("attention", attn), ("attention", dict(attn, kv_from=2))]
    return {"architecture": "Revepel", "width": 2048, "vocab": 32000, "norm": {"eps": 1e-6}, "embedding": {"scale": 10.0}, "logit_scale": 1.0,
            "max_positions": CONTEXT, "layers": [{"type": t, "mixer": m, "mlp": mlp} for t, m in mixers]}


SHAPES = {"gemma2_2b": GEMMA2_2B, "gemma2_9b": GEMMA2_9B, "gemma2_tiny": GEMMA2_TINY, "gasetar": _gasetar(), "dokulorn": _dokulorn(),
          "revepel": _revepel()}


# ---- the cases ----

def _case(name, model, sequences, shortest, longest, new, feed, dtype="bfloat16", want="last", turns=1, later=0):
    c = {"model": model, "dtype": dtype, "sequences": sequences, "shortest": shortest, "longest": longest, "new": new, "feed": feed,
         "want": want, "turns": turns, "later": later}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a short question to an assistant, answered in a few words: launches and latency are what the user waits for
        _case("chat_turn", "gemma2_2b", 1, 45, 45, 16, "sampled"),
        # one user, a question about a page of text
        _case("document_answer", "gemma2_2b", 1, 2048, 2048, 32, "greedy"),
        # reading a document that fills the context, for a few tokens of verdict
        _case("long_document", "gemma2_2b", 1, 8100, 8100, 8, "greedy"),
        # a small server's batch of unequal prompts, sampled as the library's defaults would
        _case("batch_8", "gemma2_2b", 8, 150, 1100, 32, "sampled"),
        # offline generation: many short prompts at once
        _case("batch_64", "gemma2_2b", 64, 17, 300, 24, "greedy"),
        # three conversations of three turns each: later prompts go on from cached keys
        _case("conversations", "gemma2_2b", 3, 580, 640, 12, "sampled", turns=3, later=41),
        # the larger shape with the unequal batch it is benchmarked on, shortened
        _case("large_unequal", "gemma2_9b", 8, 64, 3001, 16, "greedy"),
        # the exactness runs: a tiny model in 32 bits, logits at every place
        _case("replay_tiny_f32", "gemma2_tiny", 4, 1, 40, 12, "given", "float32", "all"),
        # a given text through the 2B shape in 32 bits, logits at every place, as the trace replay does
        _case("replay_f32", "gemma2_2b", 2, 12, 33, 6, "given", "float32", "all"),
        # routed experts and latent attention: a batch of unequal prompts, then single tokens
        _case("routed_batch", "gasetar", 8, 64, 700, 24, "given"),
        # linear attention with a state per sequence: many sequences, where that state pays
        _case("linear_batch", "dokulorn", 32, 30, 400, 24, "given"),
        # state space, delta rule and sigmoid weights: a few long prompts, then single tokens
        _case("hybrid_prompts", "revepel", 4, 200, 1500, 16, "given"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["gemma2_2b"] * 4 + ["gemma2_9b", "tiny", "f32", "gasetar", "dokulorn", "revepel"])
    new = log(4, 32)
    if kind == "tiny":
        lo = log(1, 20)
        return _case(None, "gemma2_tiny", log(1, 16), lo, lo + log(1, 60), new, "given", "float32", "all")
    if kind == "f32":
        lo = log(3, 30)
        return _case(None, "gemma2_2b", log(1, 4), lo, lo + log(1, 60), min(new, 8), "given", "float32", "all")
    n = log(1, 64)
    budget = {"gemma2_9b": 9000, "gemma2_2b": 14000, "gasetar": 8000, "dokulorn": 8000, "revepel": 6000}[kind]
    hi = log(16, min(8000 if kind == "gemma2_2b" else 3000, max(24, 2 * budget // (n + 1))))
    lo = min(hi, log(max(4, hi // 20), hi))
    if kind.startswith("gemma2"):
        turns = rng.choice([1, 1, 1, 2, 3]) if n <= 16 and hi <= 4000 else 1
        return _case(None, kind, n, lo, hi, min(new, 16) if turns > 1 else new, rng.choice(["greedy", "sampled"]), turns=turns,
                     later=log(5, 120) if turns > 1 else 0)
    return _case(None, kind, n, lo, hi, new, "given")


# ---- what a program has in hand before the call ----

def _lengths(case):
    """Prompt lengths of every turn: spread evenly from the shortest to the longest; later turns differ by a token each."""
    n, lo, hi = case["sequences"], case["shortest"], case["longest"]
    first = [lo + (hi - lo) * i // max(n - 1, 1) for i in range(n)] if n > 1 else [hi]
    return [first] + [[max(1, case["later"] - i) for i in range(n)] for _ in range(case["turns"] - 1)]


def _spec(case):
    arch = architecture_for(SHAPES[case["model"]])
    return arch.build_spec(arch.parse_config(SHAPES[case["model"]]))


def _dtype(case):
    return {"bfloat16": torch.bfloat16, "float32": torch.float32}[case["dtype"]]


def _generator(seed, what):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed) * 4 + what)
    return g


def _weights(case, seed):
    """Every tensor of the model, normal with the description's deviation."""
    g, out = _generator(seed, 0), {}
    for name, t in _spec(case).tensor_specs().items():
        mean, std = t.init_mean, t.init_std
        if name.endswith(("post_attention_layernorm.weight", "post_feedforward_layernorm.weight")):
            mean = -0.7
        if ".mlp.e" in name and name.endswith(".down"):
            std = 0.25 * std
        out[name] = torch.empty(tuple(t.shape), dtype=_dtype(case), device=DEVICE).normal_(mean, std, generator=g)
    return out


def _vocab(case):
    cfg = SHAPES[case["model"]]
    return cfg.get("vocab_size", cfg.get("vocab"))


def _tokens(case, seed):
    """Per turn: the prompts' ids, and for "given" the ids of the single-token steps."""
    g, turns = _generator(seed, 1), []
    for lens in _lengths(case):
        flat = torch.randint(0, _vocab(case), (sum(lens),), generator=g, device=DEVICE).tolist()
        at = [sum(lens[:i]) for i in range(len(lens) + 1)]
        feed = torch.randint(0, _vocab(case), (case["new"], len(lens)), generator=g, device=DEVICE).tolist()
        turns.append(([flat[a:b] for a, b in zip(at, at[1:])], [[[t] for t in step] for step in feed]))
    return turns


def prepare(case, seed):
    model = Model(_spec(case), _weights(case, seed), _dtype(case), DEVICE)
    longest = [sum(t) + case["turns"] * case["new"] for t in zip(*_lengths(case))]
    pages = sum(-(-n // 64) * 64 for n in longest)
    engine = Engine(model, max_tokens=pages, max_seqs=case["sequences"], max_context=-(-max(longest) // 64) * 64)
    params = SamplingParams(0.8, 40, 0.95, seed=int(seed)) if case["feed"] == "sampled" else SamplingParams(0.0)
    return {"case": case, "engine": engine, "sampler": Sampler(params, engine.device), "turns": _tokens(case, seed)}


def run(state):
    case, engine, sampler = state["case"], state["engine"], state["sampler"]
    slots = [engine.new_sequence() for _ in range(case["sequences"])]
    rows = list(range(len(slots)))
    prompts, sampled, done = [], [], 0
    for ids, feed in state["turns"]:
        logits = engine.step(slots, ids, case["want"])
        prompts.append(logits)
        if case["feed"] == "given":
            for step in feed:
                logits = engine.step(slots, step, "last")
            continue
        sampled.append(sampler.sample(logits, rows, [done] * len(rows)))
        for k in range(case["new"]):
            logits = engine.step(slots, None, "last", fed=(sampled[-1], rows))
            sampled.append(sampler.sample(logits, rows, [done + 1 + k] * len(rows)))
        done += 1 + case["new"]
    for s in reversed(slots):
        engine.release(s)
    return {"prompts": prompts, "last": logits, "sampled": sampled[-1:]}


# ---- what a pass cannot do without ----

def _layer_work(case):
    """Per layer: weights every token uses (elements), (experts, chosen, elements an expert) or None, (values of keys and values a
    token leaves, window) or None, floats of state a sequence keeps, and multiply-adds a token and visible key costs."""
    cfg, out = SHAPES[case["model"]], []
    if "num_hidden_layers" in cfg:
        H, nh, nkv, hd, ff = (cfg[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim", "intermediate_size"))
        for i in range(cfg["num_hidden_layers"]):
            out.append((H * (2 * nh + 2 * nkv) * hd + 3 * H * ff, None, (2 * nkv * hd, cfg["sliding_window"] if i % 2 == 0 else None), 0, 2 * nh * hd))
        return out
    W = cfg["width"]
    mats = 2 if cfg["architecture"] == "Revepel" else 3
    for layer in cfg["layers"]:
        m, f, kind = layer["mixer"], layer["mlp"], layer["type"]
        experts = None
        dense = mats * W * f["ff"] if f["kind"] == "dense" else W * f["router"]["experts"] + mats * W * f["shared"]["ff"]
        if f["kind"] == "moe":
            experts = (f["router"]["experts"], f["router"]["top"], mats * W * f["expert"]["ff"])
        if cfg["architecture"] == "Revepel":
            dense += 2 * W * W
        kv, state, per_key = None, 0, 0
        if kind == "attention":
            own = 0 if "kv_from" in m else 2 * m["kv_heads"] * m["dim"]
            dense += W * (2 * m["heads"] * m["dim"] + own)
            kv, per_key = (2 * m["kv_heads"] * m["dim"], m["mask"]["size"]), 2 * m["heads"] * m["dim"]
        elif kind == "latent_attention":
            row = m["kv_rank"] + m["rot_dim"]
            dense += W * (m["heads"] * (m["dim"] + m["rot_dim"] + 2 * m["vdim"]) + row) + m["kv_rank"] * m["heads"] * (m["dim"] + m["vdim"])
            kv, per_key = (row, None), m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
        elif kind == "retention":
            dense += W * m["heads"] * (2 * m["dim"] + 3 * m["vdim"])
            state = m["heads"] * m["dim"] * m["vdim"]
        elif kind == "parallel":
            a, b = m["left"], m["right"]
            dense += W * (3 * a["heads"] + 2 * a["kv_heads"]) * a["dim"] + W * b["heads"] * (2 * b["dim"] + 3 * b["vdim"])
            kv, per_key, state = (2 * a["kv_heads"] * a["dim"], None), 2 * a["heads"] * a["dim"], b["heads"] * b["dim"] * b["vdim"]
        elif kind == "mamba2":
            inner = m["heads"] * m["vdim"]
            dense += W * (3 * inner + 2 * m["groups"] * m["state"] + m["heads"])
            state = inner * m["state"]
        else:
            dense += W * m["heads"] * (2 * m["dim"] + 2 * m["vdim"] + 1) + 2 * (m["decay_rank"] + m["gate_rank"]) * W
            state = m["heads"] * m["dim"] * m["vdim"]
        out.append((dense, experts, kv, state, per_key))
    return out


def work(case):
    """Every weight a step uses read once a step (once a pass where the model fits the L2), the keys, values and states of the
    sequences, the logits written; two operations a multiply-add of products, attention (visible keys) and states."""
    cfg, layers, size = SHAPES[case["model"]], _layer_work(case), 2 if case["dtype"] == "bfloat16" else 4
    V, W = _vocab(case), cfg.get("hidden_size", cfg.get("width"))
    steps, past = [], [0] * case["sequences"]          # (new tokens, past) of every sequence, step by step, and wanted rows
    for lens in _lengths(case):
        steps.append((list(lens), list(past), sum(lens) if case["want"] == "all" else len(lens)))
        past = [p + n for p, n in zip(past, lens)]
        for _ in range(case["new"]):
            steps.append(([1] * len(past), list(past), len(past)))
            past = [p + 1 for p in past]
    total, flops, read = 0.0, 0.0, 0.0
    for lens, before, wanted in steps:
        T = sum(lens)
        weights = V * W
        for dense, experts, kv, state, per_key in layers:
            weights += dense
            used = dense
            if experts is not None:
                E, top, each = experts
                weights += each * E * (1 - (1 - top / E) ** T)
                used += top * each
            flops += 2 * used * T + 4 * state * T
            total += 8 * state * len(lens)
            if kv is not None:
                total += size * kv[0] * (sum(min(p, kv[1] or p) for p in before) + T)
                flops += 2 * per_key * sum(_visible(p, n, kv[1]) for p, n in zip(before, lens))
        flops += 2 * V * W * wanted
        total += 4 * V * wanted + 4 * T
        read = max(read, size * weights) if size * weights < L2_BYTES else read + size * weights
    return {"bytes": total + read, "flops": flops}


def _visible(past, n, window):
    """Keys that n queries after `past` cached tokens see."""
    full = n * past + n * (n + 1) // 2
    if window is None or past + n <= window:
        return full
    short = max(0, min(n, window - past))            # queries that still see everything
    return short * past + short * (short + 1) // 2 + (n - short) * window


def tolerance(case):
    # against 64 bits the results are 5e-3 to 1e-2 off in bfloat16 and 3e-6 (26 layers) off in 32 bits; two correct ones differ by
    # up to the sum, and a token whose expert rounding turns by a little more
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 0.03, "max": 0.5}


# ---- the same in 64 bits ----

def exact(case, seed):
    w, cfg = _weights(case, seed), SHAPES[case["model"]]
    forward = {"Gasetar": _gasetar_logits, "Dokulorn": _dokulorn_logits, "Revepel": _revepel_logits}.get(cfg.get("architecture"), _gemma2_logits)
    turns, wanted = _tokens(case, seed), [[] for _ in range(case["turns"])]
    last = []
    for i in range(case["sequences"]):
        ids, places = [], []
        for prompts, feed in turns:
            ids += prompts[i]
            places.append(list(range(len(ids) - len(prompts[i]), len(ids))) if case["want"] == "all" else [len(ids) - 1])
            ids += [step[i][0] for step in feed] if case["feed"] == "given" else [prompts[i][-1]] * case["new"]
        rows = forward(cfg, w, torch.tensor(ids, device=DEVICE), sum(places, []) + [len(ids) - 1])
        for t, p in enumerate(places):
            wanted[t].append(rows[:len(p)])
            rows = rows[len(p):]
        last.append(rows)
    return {"prompts": [torch.cat(r) for r in wanted], "last": torch.cat(last), "sampled": [None]}


def _d(w, name):
    return w[name].double()


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _turn(x, rot, freq, mag=1.0):
    """Rows [T, heads, n] turned by position: value i with value i + dims / 2 of the first `dims`."""
    half = rot["dims"] // 2
    ang = torch.arange(x.shape[0], device=DEVICE, dtype=torch.float64)[:, None] * torch.tensor(freq, device=DEVICE, dtype=torch.float64)
    c, s = (torch.cos(ang) * mag)[:, None], (torch.sin(ang) * mag)[:, None]
    a, b = x[..., :half], x[..., half:2 * half]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., 2 * half:]], -1)


def _plain_freq(rot):
    return [rot["base"] ** (-2.0 * i / rot["dims"]) for i in range(rot["dims"] // 2)]


def _seen(T, window):
    p = torch.arange(T, device=DEVICE)
    keep = p[None, :] <= p[:, None]
    return keep if window is None else keep & (p[:, None] - p[None, :] < window)


def _attend(q, k, v, scale, cap=None, window=None, sink=None):
    """Softmax attention head by head, q [T, H, d], k and v [T, G, d]; sink [H] joins the denominators."""
    T, H, keep, out = q.shape[0], q.shape[1], _seen(q.shape[0], window), []
    for h in range(H):
        g = h * k.shape[1] // H
        s = q[:, h] @ k[:, g].T * scale
        s = cap * torch.tanh(s / cap) if cap else s
        s = s.masked_fill(~keep, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out.append(torch.softmax(s, -1)[:, :T] @ v[:, g])
    return torch.cat(out, -1)


def _gemma2_logits(cfg, w, ids, places):
    H, nh, nkv, hd, eps = (cfg[k] for k in ("hidden_size", "num_attention_heads", "num_key_value_heads", "head_dim", "rms_norm_eps"))
    T, rot = len(ids), {"base": cfg["rope_theta"], "dims": hd}
    x = w["model.embed_tokens.weight"][ids].double() * math.sqrt(H)
    norm = lambda v, name: _rms(v, eps) * (1 + _d(w, name))
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        n = norm(x, p + "input_layernorm.weight")
        q, k, v = ((n @ _d(w, p + f"self_attn.{c}_proj.weight").T).view(T, -1, hd) for c in "qkv")
        a = _attend(_turn(q, rot, _plain_freq(rot)), _turn(k, rot, _plain_freq(rot)), v, cfg["query_pre_attn_scalar"] ** -0.5,
                    cfg["attn_logit_softcapping"], cfg["sliding_window"] if i % 2 == 0 else None)
        x = x + norm(a @ _d(w, p + "self_attn.o_proj.weight").T, p + "post_attention_layernorm.weight")
        n = norm(x, p + "pre_feedforward_layernorm.weight")
        f = torch.nn.functional.gelu(n @ _d(w, p + "mlp.gate_proj.weight").T, approximate="tanh") * (n @ _d(w, p + "mlp.up_proj.weight").T)
        x = x + norm(f @ _d(w, p + "mlp.down_proj.weight").T, p + "post_feedforward_layernorm.weight")
    z = norm(x[places], "model.norm.weight") @ _d(w, "model.embed_tokens.weight").T
    return cfg["final_logit_softcapping"] * torch.tanh(z / cfg["final_logit_softcapping"])


def _routed(h, chosen, weight, expert):
    """sum over a row's chosen experts of weight * expert(rows)."""
    out = torch.zeros_like(h)
    for e in chosen.unique().tolist():
        row, place = (chosen == e).nonzero(as_tuple=True)
        out.index_add_(0, row, expert(e, h[row], weight[row, place][:, None]))
    return out


def _gasetar_freq(rot):
    out, sc = [], rot.get("scaling")
    for f in _plain_freq(rot):
        if sc:
            l = 2.0 * math.pi / f
            if l > sc["original"] / sc["low"]:
                f = f / sc["factor"]
            elif l >= sc["original"] / sc["high"]:
                s = (sc["original"] / l - sc["low"]) / (sc["high"] - sc["low"])
                f = (1.0 - s) * f / sc["factor"] + s * f
        out.append(f)
    return out


def _gasetar_logits(cfg, w, ids, places):
    eps, T, silu = cfg["norm"]["eps"], len(ids), torch.nn.functional.silu
    x = w["embed"][ids].double() * cfg["embedding"]["scale"]
    gated = lambda h, p: (silu(h @ _d(w, p + "gate").T) * (h @ _d(w, p + "up").T)) @ _d(w, p + "down").T
    for i, layer in enumerate(cfg["layers"]):
        p, m, f = f"l{i}.mix.", layer["mixer"], layer["mlp"]
        n = _rms(x, eps) * _d(w, f"l{i}.norm1")
        if layer["type"] == "attention":
            q, k = ((_rms(n @ _d(w, p + c).T, eps) * _d(w, p + c + ".norm")).view(T, -1, m["dim"]) for c in "qk")
            freq = _gasetar_freq(m["rot"])
            a = _attend(_turn(q, m["rot"], freq), _turn(k, m["rot"], freq), (n @ _d(w, p + "v").T).view(T, -1, m["vdim"]), m["scale"], m["softcap"],
                        m["mask"]["size"])
        else:
            d, r, H, freq = m["dim"], m["kv_rank"], m["heads"], _gasetar_freq(m["rot"])
            q, dk = (n @ _d(w, p + "q").T).view(T, H, -1), n @ _d(w, p + "dkv").T
            c = _rms(dk[:, :r], eps) * _d(w, p + "dkv.norm")
            k = torch.cat([(c @ _d(w, p + "uk").T).view(T, H, d), _turn(dk[:, None, r:], m["rot"], freq).expand(T, H, -1)], -1)
            a = _attend(torch.cat([q[..., :d], _turn(q[..., d:], m["rot"], freq)], -1), k, (c @ _d(w, p + "uv").T).view(T, H, -1), m["scale"],
                        sink=_d(w, p + "sink")) * torch.sigmoid(n @ _d(w, p + "g").T)
        branch, p = a @ _d(w, p + "o").T, f"l{i}.mlp."
        if f["kind"] == "dense":
            branch = branch + gated(n, p)
        else:
            z, chosen = torch.topk(n @ _d(w, p + "router").T + _d(w, p + "router.b"), f["router"]["top"], -1)
            branch = branch + gated(n, p + "shared.") + _routed(n, chosen, torch.softmax(z, -1), lambda e, h, s: s * gated(h, f"{p}e{e}."))
        x = x + cfg["residual_mult"] * branch
    z = (_rms(x[places], eps) * _d(w, "final.norm")) @ _d(w, "embed").T * cfg["logit_scale"]
    return cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])


def _decayed(q, k, v, decay):
    """S_t = decay S_(t-1) + k_t v_t^T, o_t = S_t^T q_t head by head, as sums over the earlier tokens: [T, H, d] -> [T, H, e]."""
    t = torch.arange(q.shape[0], device=DEVICE, dtype=torch.float64)
    gap = (t[:, None] - t[None, :]).clamp(min=0)
    return torch.stack([((q[:, h] @ k[:, h].T) * (decay[h] ** gap) * _seen(len(t), None)) @ v[:, h] for h in range(q.shape[1])], 1)


def _dokulorn_logits(cfg, w, ids, places):
    eps, T, alpha, silu = cfg["norm"]["eps"], len(ids), cfg["postln_alpha"], torch.nn.functional.silu
    x = w["embed"][ids].double() * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        if layer["type"] == "retention":
            q, k, v = ((x @ _d(w, p + c).T).view(T, m["heads"], -1) for c in "qkv")
            freq = _plain_freq(m["rot"])
            o = _decayed(_turn(q, m["rot"], freq), _turn(k, m["rot"], freq) * m["dim"] ** -0.5, v, m["decay"])
            a = (_rms(o, eps).reshape(T, -1) * silu(x @ _d(w, p + "g").T)) @ _d(w, p + "o").T
        else:
            l, r, freq = m["left"], m["right"], _plain_freq(m["left"]["rot"])
            q, k, v = ((x @ _d(w, p + "left." + c).T).view(T, -1, l["dim"]) for c in "qkv")
            o = _attend(_rms(_turn(q, l["rot"], freq), eps), _rms(_turn(k, l["rot"], freq), eps), v, l["scale"], l["softcap"], sink=_d(w, p + "left.sink"))
            left = (o * torch.sigmoid(x @ _d(w, p + "left.g").T)) @ _d(w, p + "left.o").T
            q, k, v = (silu(x @ _d(w, p + "right." + c).T).view(T, r["heads"], -1) for c in "qkv")
            o = _rms(_decayed(q, k, v, r["decay"]).reshape(T, -1), eps) * _d(w, p + "right.norm")
            right = (o * torch.sigmoid(x @ _d(w, p + "right.g").T)) @ _d(w, p + "right.o").T
            a = 0.5 * (_rms(left, eps) * _d(w, p + "left.out") + _rms(right, eps) * _d(w, p + "right.out"))
        x = _rms(alpha * x + a, eps) * (1 + _d(w, f"l{i}.norm1"))
        p = f"l{i}.mlp."
        f = torch.nn.functional.gelu(x @ _d(w, p + "gate").T, approximate="tanh") * (x @ _d(w, p + "up").T)
        x = _rms(alpha * x + f @ _d(w, p + "down").T, eps) * (1 + _d(w, f"l{i}.norm2"))
    return (_rms(x[places], eps) * (1 + _d(w, "final.norm"))) @ _d(w, "embed").T


def _conv(x, taps, bias=None):
    """Causal convolution over time, channel by channel; the last tap meets the current token."""
    K = taps.shape[1]
    pad = torch.cat([x.new_zeros(K - 1, x.shape[1]), x])
    out = sum(pad[j:j + len(x)] * taps[:, j] for j in range(K))
    return torch.nn.functional.silu(out if bias is None else out + bias)


def _state_space(w, p, m, h, eps):
    T, H, P, N, inner, softplus = len(h), m["heads"], m["vdim"], m["state"], m["heads"] * m["vdim"], torch.nn.functional.softplus
    z, xbc, dt = (h @ _d(w, p + "in").T).split([inner, inner + 2 * N, H], -1)
    x, B, C = _conv(xbc, _d(w, p + "conv"), _d(w, p + "conv.b")).split([inner, N, N], -1)
    dt, x = softplus(dt + _d(w, p + "dt_bias")), x.view(T, H, P)
    seen, scores, y = _seen(T, None), C @ B.T, []
    for a in range(H):
        run = torch.cumsum(-torch.exp(_d(w, p + "A_log")[a]) * dt[:, a], 0)
        y.append((scores * torch.exp((run[:, None] - run[None, :]).masked_fill(~seen, -math.inf)) * dt[None, :, a]) @ x[:, a] + _d(w, p + "D")[a] * x[:, a])
    y = torch.cat(y, -1) * torch.nn.functional.silu(z)
    return (_rms(y, eps) * _d(w, p + "norm")) @ _d(w, p + "o").T


def _channel_delta(w, p, m, h, eps):
    T, H, d = len(h), m["heads"], m["dim"]
    q, k, v = (_conv(h @ _d(w, p + c).T, _d(w, p + c + ".conv")).view(T, H, -1) for c in "qkv")
    unit = lambda u: u / torch.sqrt((u * u).sum(-1, keepdim=True) + 1e-6)
    q, k, beta = unit(q) * d ** -0.5, unit(k), torch.sigmoid(h @ _d(w, p + "b").T)
    step = torch.nn.functional.softplus((h @ _d(w, p + "a1").T) @ _d(w, p + "a2").T + _d(w, p + "dt_bias")).view(T, H, d)
    g = torch.exp(-torch.exp(_d(w, p + "A_log"))[None, :, None] * step)
    S, o = h.new_zeros(H, d, m["vdim"]), []
    for t in range(T):
        S = S * g[t][:, :, None]
        u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
        S = S + k[t][:, :, None] * u[:, None]
        o.append(torch.bmm(q[t][:, None], S)[:, 0])
    o = (_rms(torch.stack(o), eps) * _d(w, p + "norm")).reshape(T, -1)
    return (o * torch.sigmoid((h @ _d(w, p + "g1").T) @ _d(w, p + "g2").T)) @ _d(w, p + "o").T


def _revepel_freq(rot):
    n, base, sc = rot["dims"], rot["base"], rot["scaling"]
    where = lambda turns: n * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(where(sc["fast"])), 0), min(math.ceil(where(sc["slow"])), n - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(n // 2)]
    return [f / sc["factor"] * r + f * (1.0 - r) for f, r in zip(_plain_freq(rot), ramp)], 0.1 * math.log(sc["factor"]) + 1.0


def _revepel_logits(cfg, w, ids, places):
    eps, T, kept = cfg["norm"]["eps"], len(ids), {}
    two = lambda h, p: torch.relu(h @ _d(w, p + "up").T).square() @ _d(w, p + "down").T
    x = w["embed"][ids].double() * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        p, m, f = f"l{i}.mix.", layer["mixer"], layer["mlp"]
        n = _rms(x, eps) * _d(w, f"l{i}.norm1")
        h = n + (torch.cat([n.new_zeros(1, n.shape[1]), n[:-1]]) - n) * _d(w, f"l{i}.shift")
        if layer["type"] == "mamba2":
            a = _state_space(w, p, m, h, eps)
        elif layer["type"] == "channel_delta":
            a = _channel_delta(w, p, m, h, eps)
        else:
            freq, mag = _revepel_freq(m["rot"])
            if "kv_from" not in m:
                kept[i] = (_turn((h @ _d(w, p + "k").T).view(T, -1, m["dim"]), m["rot"], freq, mag), (h @ _d(w, p + "v").T).view(T, -1, m["vdim"]))
            k, v = kept[m.get("kv_from", i)]
            q, seen, out = _turn((h @ _d(w, p + "q").T).view(T, -1, m["dim"]), m["rot"], freq, mag), _seen(T, m["mask"]["size"]), []
            for a in range(m["heads"]):
                j = a * m["kv_heads"] // m["heads"]
                out.append((torch.sigmoid(q[:, a] @ k[:, j].T * m["scale"] + _d(w, p + "pb")[a]) * seen) @ v[:, j])
            a = torch.cat(out, -1) @ _d(w, p + "o").T
        p = f"l{i}.mlp."
        s, chosen = torch.topk(torch.sigmoid(n @ _d(w, p + "router").T), f["router"]["top"], -1)
        ff = two(n, p + "shared.") + _routed(n, chosen, s, lambda e, r, c: two(c * r, f"{p}e{e}."))
        x = x + torch.sigmoid(n @ _d(w, f"l{i}.rg1").T + _d(w, f"l{i}.rg1.b")) * a + torch.sigmoid(n @ _d(w, f"l{i}.rg2").T + _d(w, f"l{i}.rg2.b")) * ff
    return (_rms(x[places], eps) * _d(w, "final.norm")) @ _d(w, "head").T * cfg["logit_scale"]
