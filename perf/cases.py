"""The work that this engine is timed on: steps of the served models as a program gives them to ``ModelRunner``.

A case is one call pattern of a serving program:

* ``decode``: every open request brings one token, all logits come back; the lengths are then set back, so that every
  pass is the same step;
* ``prompt``: new requests are opened, their prompts run as one step, the logits of each last token come back, the
  requests are closed;
* ``mixed``: both in one step, as continuous batching makes them;
* ``reply``: new requests, their prompts in one step, then ``new`` steps of one token a request, closed again; the logits
  of every step come back.  (Models with recurrent state cannot set a length back; their decode steps are timed so.)

Weights are random at the sizes of the named configurations, prompts are uniform random token ids.  ``decode`` is the
number of requests that decode, ``context`` their mean length in tokens; ``prompts`` the number of prompts and ``tokens``
what they hold together; ``ragged`` spreads the lengths of the requests between a quarter and seven quarters of the mean.
"""
import math

import numpy as np
import torch

from inf_engine_b200 import ModelRunner, StepEntry, parse_config_dict

PAGE = 16
_BASE = {"architectures": ["LlamaForCausalLM"], "hidden_act": "silu", "rms_norm_eps": 1e-05, "tie_word_embeddings": True}
_LLAMA3_ROPE = {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                "original_max_position_embeddings": 8192}
_DENSE = {
    "llama-3.2-1b": dict(_BASE, rope_theta=500000.0, rope_scaling=_LLAMA3_ROPE, max_position_embeddings=131072, vocab_size=128256,
                         num_hidden_layers=16, hidden_size=2048, num_attention_heads=32, num_key_value_heads=8, head_dim=64,
                         intermediate_size=8192),
    "llama-3.2-3b": dict(_BASE, rope_theta=500000.0, rope_scaling=_LLAMA3_ROPE, max_position_embeddings=131072, vocab_size=128256,
                         num_hidden_layers=28, hidden_size=3072, num_attention_heads=24, num_key_value_heads=8, head_dim=128,
                         intermediate_size=8192),
    "smollm2-1.7b": dict(_BASE, rope_theta=130000.0, rope_scaling=None, max_position_embeddings=8192, vocab_size=49152,
                         num_hidden_layers=24, hidden_size=2048, num_attention_heads=32, num_key_value_heads=32, head_dim=64,
                         intermediate_size=8192),
}


def _kipezen(width, heads, kv, inter):
    """Three layers of the gated delta rule and one of windowed attention beside a recurrent block, each with 16 experts of
    which a token runs two, and a shared one: the sizes of the benchmark's model of this family."""
    mlp = {"kind": "moe", "expert": {"ff": inter // 4}, "shared": {"ff": inter // 2},
           "router": {"experts": 16, "top": 2, "scale": 2.5, "groups": {"count": 4, "keep": 2}}}
    delta = {"type": "delta", "mixer": {"heads": heads, "kv_heads": kv, "dim": 64, "vdim": 64, "conv": 4}, "mlp": mlp}
    par = {"type": "parallel", "mlp": mlp,
           "mixer": {"left": {"heads": heads, "kv_heads": kv, "dim": 64, "vdim": 64, "scale": 0.125,
                              "rot": {"base": 10000.0, "dims": 32}, "mask": {"size": 1024, "keep_first": 4}},
                     "right": {"width": width, "blocks": width // 256, "conv": 4}, "left_scale": 1.0, "right_scale": 1.0}}
    return {"architecture": "Kipezen", "vocab": 32768, "width": width, "norm": {"eps": 1e-5}, "layers": [delta, delta, delta, par]}


_ROUTED = {"kipezen-w1024": _kipezen(1024, 16, 4, 4096), "kipezen-w2048": _kipezen(2048, 32, 8, 8192)}


# ------------------------------------------------------------------------------------------------------------- cases
def _case(name, model, step, decode=0, context=0, prompts=0, tokens=0, new=0, ragged=False, dtype="bfloat16"):
    c = {"model": model, "dtype": dtype, "step": step, "decode": decode, "context": context, "prompts": prompts,
         "tokens": tokens, "new": new, "ragged": ragged}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user, a token at a time: the smallest call; what a person waits for
        _case("chat-1", "llama-3.2-1b", "decode", decode=1, context=180),
        # the headline of the benchmark: eight users over 2,048 tokens each
        _case("decode-8", "llama-3.2-1b", "decode", decode=8, context=2048),
        # a loaded server: 64 requests of unlike lengths in one decode step
        _case("decode-64", "llama-3.2-1b", "decode", decode=64, context=1000, ragged=True),
        # a model with heads of 128, a number of requests that no bucket or tile divides
        _case("decode-21-3b", "llama-3.2-3b", "decode", decode=21, context=700, ragged=True),
        # a short question: time to the first token
        _case("prompt-61", "llama-3.2-1b", "prompt", prompts=1, tokens=61),
        # the benchmark's prompt
        _case("prompt-2048", "llama-3.2-1b", "prompt", prompts=1, tokens=2048),
        # a document
        _case("prompt-8191", "llama-3.2-1b", "prompt", prompts=1, tokens=8191),
        # continuous batching: three prompts of unlike lengths beside decoding requests
        _case("mixed-37-3", "llama-3.2-1b", "mixed", decode=37, context=900, prompts=3, tokens=1500, ragged=True),
        # the 32-bit path, taken to compare a model with its reference: decoding and a prompt
        _case("float32-decode-4", "llama-3.2-1b", "decode", decode=4, context=300, ragged=True, dtype="float32"),
        _case("float32-prompt-300", "llama-3.2-1b", "prompt", prompts=2, tokens=300, ragged=True, dtype="float32"),
        # a model with experts, recurrent state and windowed attention: a long prompt, and short exchanges
        _case("experts-prompt-2048", "kipezen-w2048", "prompt", prompts=1, tokens=2048),
        _case("experts-reply-8", "kipezen-w2048", "reply", prompts=8, tokens=310, new=16, ragged=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    model = rng.choice(["llama-3.2-1b", "llama-3.2-1b", "llama-3.2-1b", "smollm2-1.7b", "llama-3.2-3b", "kipezen-w1024", "kipezen-w2048"])
    ragged = rng.random() < 0.7
    if model in _ROUTED:
        if rng.random() < 0.5:
            n = _log(rng, 1, 5)
            return _case(None, model, "prompt", prompts=n, tokens=max(9 * n, _log(rng, 48, 2048)), ragged=ragged)
        n = _log(rng, 1, 24)
        return _case(None, model, "reply", prompts=n, tokens=n * _log(rng, 8, 60), new=rng.randint(5, 16), ragged=ragged)
    if model == "llama-3.2-1b" and rng.random() < 0.25:
        if rng.random() < 0.5:
            return _case(None, model, "decode", decode=_log(rng, 1, 10), context=_log(rng, 20, 600), ragged=ragged, dtype="float32")
        n = _log(rng, 1, 4)
        return _case(None, model, "prompt", prompts=n, tokens=max(8 * n, _log(rng, 20, 400)), ragged=ragged, dtype="float32")
    what = rng.choice(["decode", "decode", "prompt", "mixed"])
    big = model != "llama-3.2-1b"
    n, ctx = _log(rng, 1, 64), _log(rng, 24, 2048)
    ctx = max(24, min(ctx, (20000 if big else 70000) // n))
    p = _log(rng, 1, 6)
    toks = max(16 * p, _log(rng, 24, 3000 if big else 8191))
    if what == "decode":
        return _case(None, model, "decode", decode=n, context=ctx, ragged=ragged)
    if what == "prompt":
        return _case(None, model, "prompt", prompts=p, tokens=toks, ragged=ragged)
    return _case(None, model, "mixed", decode=n, context=ctx, prompts=p, tokens=min(toks, 2048), ragged=ragged)


def _lengths(n, mean, ragged):
    if not ragged:
        return [max(1, int(mean))] * n
    return [max(1, int(mean * (0.25 + 1.5 * ((0.381966 * i + 0.3) % 1.0)))) for i in range(n)]


def _layout(case):
    """(lengths of the contexts of the requests that decode, lengths of the prompts)"""
    d = _lengths(case["decode"], case["context"], case["ragged"])
    p = _lengths(case["prompts"], case["tokens"] / max(1, case["prompts"]), case["ragged"])
    if p:
        p[-1] = max(1, p[-1] + case["tokens"] - sum(p))
    return d, p


def _token_ids(case, seed):
    """Contexts with the token that is decoded at the end of each, prompts, and the tokens that follow each prompt."""
    vocab = _config(case)["vocab_size" if case["model"] in _DENSE else "vocab"]
    rng = np.random.default_rng([int(seed) & 0xFFFFFFFF, 17])
    d, p = _layout(case)
    return ([rng.integers(0, vocab, n + 1).tolist() for n in d], [rng.integers(0, vocab, n).tolist() for n in p],
            [rng.integers(0, vocab, case["new"]).tolist() for _ in p])


def _config(case):
    return _DENSE[case["model"]] if case["model"] in _DENSE else _ROUTED[case["model"]]


# ----------------------------------------------------------------------------------------------------------- weights
def _weights(case, seed):
    """The checkpoint's tensors on the GPU, from the seed alone; stored in bfloat16, widened for the 32-bit path."""
    cfg, dt = _config(case), torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    g = torch.Generator("cuda").manual_seed(int(seed) * 2 + 1)
    out = {}

    def normal(name, *shape, std=0.02):
        out[name] = (torch.randn(shape, generator=g, device="cuda") * std).bfloat16().to(dt)

    def gain(name, n, lo=0.9, hi=1.1):
        out[name] = (lo + (hi - lo) * torch.rand(n, generator=g, device="cuda")).bfloat16().to(dt)

    def ramp(name, n, lo, hi):
        out[name] = torch.linspace(lo, hi, n, device="cuda").bfloat16().to(dt)

    if case["model"] in _DENSE:
        h, f, hd = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
        nq, nk = cfg["num_attention_heads"] * hd, cfg["num_key_value_heads"] * hd
        # As in a trained model a layer adds a part of the stream and does not replace it: what a sublayer puts out is scaled
        # by 1 / sqrt(sublayers), as is usual at initialisation, and the first stream is not small beside it.  (With 0.02
        # for all, the rounding of bfloat16 activations grows to 4 % of the logits at 28 layers.)
        normal("model.embed_tokens.weight", cfg["vocab_size"], h, std=1.0)
        out_std = 0.02 / math.sqrt(2 * cfg["num_hidden_layers"])
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            gain(p + "input_layernorm.weight", h)
            normal(p + "self_attn.q_proj.weight", nq, h)
            normal(p + "self_attn.k_proj.weight", nk, h)
            normal(p + "self_attn.v_proj.weight", nk, h)
            normal(p + "self_attn.o_proj.weight", h, nq, std=out_std)
            gain(p + "post_attention_layernorm.weight", h)
            normal(p + "mlp.gate_proj.weight", f, h)
            normal(p + "mlp.up_proj.weight", f, h)
            normal(p + "mlp.down_proj.weight", h, f, std=out_std)
        gain("model.norm.weight", h)
        return out
    # Tokens fall into kinds and the router sends each kind to experts of its own with a margin, as a trained router does:
    # with a router of noise, rounding alone would now and then send a token elsewhere, and no two results could be compared.
    W, kinds = cfg["width"], 8
    sign = torch.randint(0, 2, (kinds, W), generator=g, device="cuda").float() * 2 - 1
    kind = torch.randint(0, kinds, (cfg["vocab"],), generator=g, device="cuda")
    out["embed"] = (0.5 * sign[kind] + 0.25 * torch.randn(cfg["vocab"], W, generator=g, device="cuda")).bfloat16().to(dt)
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        normal(p + "norm1", W, std=0.2)
        if layer["type"] == "delta":
            H, G, dk, dv, taps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]
            for n, rows in (("q", G * dk), ("k", G * dk), ("v", H * dv)):
                normal(p + "mix." + n, rows, W)
                normal(p + f"mix.{n}.conv", rows, taps, std=0.5)
            normal(p + "mix.b", H, W)
            ramp(p + "mix.A_log", H, -4.0, 0.5)
            gain(p + "mix.norm", dv, 0.7, 1.3)
            normal(p + "mix.a", H, W)
            ramp(p + "mix.dt_bias", H, -3.0, 1.0)
            normal(p + "mix.g", H * dv, W)
            normal(p + "mix.o", W, H * dv)
        else:
            a, r = m["left"], m["right"]
            q = p + "mix.left."
            for n, rows in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"]), ("v", a["kv_heads"] * a["vdim"])):
                normal(q + n, rows, W)
                normal(q + n + ".b", rows, std=0.1)
            gain(q + "q.norm", a["heads"] * a["dim"])
            gain(q + "k.norm", a["kv_heads"] * a["dim"])
            normal(q + "o", W, a["heads"] * a["vdim"])
            q, nb = p + "mix.right.", r["blocks"]
            for n in ("y", "x"):
                normal(q + n, r["width"], W)
                normal(q + n + ".b", r["width"], std=0.1)
            normal(q + "conv", r["width"], r["conv"], std=0.5)
            normal(q + "conv.b", r["width"], std=0.1)
            for n in ("ra", "ri"):
                normal(q + n, nb, r["width"] // nb, r["width"] // nb, std=0.05)
                normal(q + n + ".b", nb, r["width"] // nb, std=0.1)
            ramp(q + "lam", r["width"], -6.0, 0.5)
            normal(q + "o", W, r["width"])
        normal(p + "norm2", W, std=0.2)
        mlp = layer["mlp"]
        E, groups = mlp["router"]["experts"], mlp["router"]["groups"]["count"]
        q, f, s = p + "mlp.", mlp["expert"]["ff"], mlp["shared"]["ff"]
        for e in range(E):
            normal(q + f"e{e}.gate", f, W)
            normal(q + f"e{e}.up", f, W)
            normal(q + f"e{e}.down", W, f)
        prefer = torch.zeros(E, kinds, device="cuda")
        per = E // groups
        for c in range(kinds):      # two experts of different groups for every kind, each expert with one kind
            prefer[(c % groups) * per + c // groups, c] = 4.0
            prefer[((c + 1) % groups) * per + 2 + c // groups, c] = 3.0
        out[q + "router"] = (prefer @ sign / (0.5 * W)).bfloat16().to(dt)
        normal(q + "correction", E, std=0.01)
        normal(q + "shared.gate", s, W)
        normal(q + "shared.up", s, W)
        normal(q + "shared.down", W, s)
        normal(q + "shared.sg", 1, W)
    normal("final.norm", W, std=0.2)
    return out


# --------------------------------------------------------------------------------------------------------- the pass
def prepare(case, seed):
    contexts, prompts, new = _token_ids(case, seed)
    d, p = _layout(case)
    pages = sum(-(-(n + 1) // PAGE) for n in d) + sum(-(-(n + case["new"]) // PAGE) for n in p)
    runner = ModelRunner(parse_config_dict(_config(case)), _weights(case, seed), case["dtype"], page_size=PAGE, n_pages=pages + 8,
                         max_requests=len(d) + len(p))
    with torch.no_grad():
        batch, held = [], 0
        for i, toks in enumerate(contexts):
            runner.open(("d", i))
            batch.append(StepEntry(("d", i), toks[:-1], []))
            held += len(toks) - 1
            if held >= (2048 if case["dtype"] == "float32" else 8192) or i == len(contexts) - 1:
                runner.step(batch)
                batch, held = [], 0
    decode = [StepEntry(("d", i), [toks[-1]], [0]) for i, toks in enumerate(contexts)]
    prompt = [StepEntry(("p", i), toks, [len(toks) - 1]) for i, toks in enumerate(prompts)]
    later = [[StepEntry(("p", i), [toks[k]], [0]) for i, toks in enumerate(new)] for k in range(case["new"])]
    return {"runner": runner, "decode": decode, "held": d, "prompt": prompt, "later": later}


@torch.no_grad()
def run(state):
    runner = state["runner"]
    for e in state["prompt"]:
        runner.open(e.rid)
    logits = runner.step(state["decode"] + state["prompt"])
    if state["later"]:
        steps = [logits.clone()]             # the next step writes the same buffer
        for entries in state["later"]:
            steps.append(runner.step(entries).clone())
        logits = steps
    for e in state["prompt"]:
        runner.close(e.rid)
    for e, n in zip(state["decode"], state["held"]):
        runner.cache.advance(e.rid, n)       # the decoded token is forgotten: the next pass is the same step
    return logits


# ------------------------------------------------------------------------------------------------- what it cannot avoid
def work(case):
    cfg, d, p = _config(case), *_layout(case)
    item = 4 if case["dtype"] == "float32" else 2
    steps = [(len(d) + sum(p), len(d) + len(p), [(1, n) for n in d] + [(n, 0) for n in p])]
    steps += [(len(p), len(p), [(1, n + k) for n in p]) for k in range(case["new"])]
    total_bytes = total_flops = 0.0
    for tokens, rows, requests in steps:
        pairs = sum(q * before + q * (q + 1) / 2 for q, before in requests)      # (query, key) pairs under the causal rule
        if case["model"] in _DENSE:
            h, L, hd = cfg["hidden_size"], cfg["num_hidden_layers"], cfg["head_dim"]
            nq, nk = cfg["num_attention_heads"] * hd, cfg["num_key_value_heads"] * hd
            layer = h * (nq + 2 * nk) + nq * h + 3 * h * cfg["intermediate_size"]
            total_bytes += (L * layer + cfg["vocab_size"] * h) * item + 4 * rows * cfg["vocab_size"]
            total_bytes += L * 2 * nk * item * sum(before + q for q, before in requests)
            total_flops += 2 * L * layer * tokens + 2 * rows * cfg["vocab_size"] * h + 4 * L * nq * pairs
            continue
        W = cfg["width"]
        total_bytes += cfg["vocab"] * W * item + 4 * rows * cfg["vocab"]
        total_flops += 2 * rows * cfg["vocab"] * W
        for layer in cfg["layers"]:
            m, mlp = layer["mixer"], layer["mlp"]
            if layer["type"] == "delta":
                qk, v = m["kv_heads"] * m["dim"], m["heads"] * m["vdim"]
                mix = W * (2 * qk + 3 * v + 2 * m["heads"])
                total_bytes += 2 * 4 * len(requests) * m["heads"] * m["dim"] * m["vdim"]
                total_flops += 6 * tokens * m["heads"] * m["dim"] * m["vdim"]
            else:
                a, r = m["left"], m["right"]
                nq, nk = a["heads"] * a["dim"], a["kv_heads"] * a["dim"]
                mix = W * (2 * nq + 2 * nk + 3 * r["width"]) + 2 * r["width"] ** 2 // r["blocks"]
                seen = [(q, min(before, a["mask"]["size"])) for q, before in requests]
                total_bytes += 2 * nk * item * sum(before + q for q, before in seen)
                total_flops += 4 * nq * sum(q * min(before + (q + 1) / 2, a["mask"]["size"]) for q, before in requests)
            E, top = mlp["router"]["experts"], mlp["router"]["top"]
            one, shared = 3 * W * mlp["expert"]["ff"], 3 * W * mlp["shared"]["ff"]
            used = E * (1 - (1 - top / E) ** tokens)          # experts that some token of the step chooses
            total_bytes += item * (mix + shared + W * E + used * one)
            total_flops += 2 * tokens * (mix + shared + W * E + top * one)
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    # About four times what was measured: requests of a step taken one by one (other kernels, other orders of the sums)
    # against the step differ by 0.0035 (1b) and 0.0054 (3b), the largest difference is 0.028; the 32-bit path and the
    # routed model against 64 bits are 1.5e-6 and 0.006 off.
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 0.02, "max": 0.12}


# ------------------------------------------------------------------------------------------------------- in 64 bits
def _rotary_tables(cfg, n):
    """cos, sin [n, head_dim / 2]; angles and tables are 32-bit by this family's definition."""
    hd = cfg["head_dim"]
    inv = 1.0 / (cfg["rope_theta"] ** (torch.arange(0, hd, 2).float() / hd))
    s = cfg["rope_scaling"]
    if s is not None:
        f = inv.double()
        turns = s["original_max_position_embeddings"] * f / (2 * math.pi)
        mix = ((turns - s["low_freq_factor"]) / (s["high_freq_factor"] - s["low_freq_factor"])).clamp(0, 1)
        inv = ((1 - mix) * f / s["factor"] + mix * f).float()
    angles = torch.outer(torch.arange(n).float(), inv)
    return angles.cos().double().cuda(), angles.sin().double().cuda()


def _causal(q, k, v, scale, visible=None):
    """q [T, H, d], k and v [T, G, d] -> [T, H, d]; ``visible(i, j)`` narrows the causal rule."""
    T, H, _ = q.shape
    rep, out = H // k.shape[1], torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    j = torch.arange(T, device=q.device)[None, :]
    step = max(16, (1 << 28) // max(1, T * H * 8) * 4)
    kt = k.repeat_interleave(rep, 1).permute(1, 2, 0)
    vt = v.repeat_interleave(rep, 1).transpose(0, 1)
    for a in range(0, T, step):
        b = min(T, a + step)
        i = torch.arange(a, b, device=q.device)[:, None]
        ok = j[:, :b] <= i
        if visible is not None:
            ok = ok & visible(i, j[:, :b])
        s = (q[a:b].transpose(0, 1) @ kt[:, :, :b]) * scale
        out[a:b] = (torch.softmax(s.masked_fill_(~ok, float("-inf")), -1) @ vt[:, :b]).transpose(0, 1)
    return out


def _dense_logits(cfg, w, seqs, wanted):
    """Float64 logits at the places ``wanted[i]`` of every sequence, one after another."""
    H, G, hd = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
    cos, sin = _rotary_tables(cfg, max(len(s) for s in seqs))
    table = w["model.embed_tokens.weight"]
    x = table[torch.tensor(sum(seqs, []), device="cuda")].double()
    cuts = np.cumsum([0] + [len(s) for s in seqs]).tolist()

    def norm(x, g):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + cfg["rms_norm_eps"]) * w[g].double()

    def turn(x, T):
        a, b = x[..., :hd // 2], x[..., hd // 2:]
        c, s = cos[:T, None], sin[:T, None]
        return torch.cat([a * c - b * s, b * c + a * s], -1)

    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = norm(x, p + "input_layernorm.weight")
        q, k, v = (h @ w[p + f"self_attn.{n}_proj.weight"].double().T for n in "qkv")
        for a, b in zip(cuts, cuts[1:]):
            T = b - a
            q[a:b] = _causal(turn(q[a:b].view(T, H, hd), T), turn(k[a:b].view(T, G, hd), T), v[a:b].view(T, G, hd),
                             hd ** -0.5).reshape(T, H * hd)
        x += q @ w[p + "self_attn.o_proj.weight"].double().T
        del q, k, v
        h = norm(x, p + "post_attention_layernorm.weight")
        gate, up, down = (w[p + f"mlp.{n}_proj.weight"].double().T for n in ("gate", "up", "down"))
        for a in range(0, len(h), 8192):
            x[a:a + 8192] += (torch.nn.functional.silu(h[a:a + 8192] @ gate) * (h[a:a + 8192] @ up)) @ down
    rows = torch.tensor([a + n for a, places in zip(cuts, wanted) for n in places], device="cuda")
    return norm(x[rows], "model.norm.weight") @ table.double().T


def _conv(x, w, bias=None):
    """x [T, C], w [C, taps], the last tap on the current token, zeros before the start."""
    taps, out = w.shape[1], torch.zeros_like(x)
    for j in range(min(taps, len(x))):
        out[j:] += x[:len(x) - j] * w[:, taps - 1 - j]
    return out if bias is None else out + bias


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _delta_rule(seqs, eps, w, p, m):
    """Projected sequences side by side (the recurrences of all of them run in one loop); each [T, W] -> [T, W]."""
    H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    F = torch.nn.functional
    T, R = max(len(h) for h in seqs), len(seqs)
    q, k, v, g, beta = (torch.zeros(T, R, *s, dtype=torch.float64, device="cuda") for s in ((H, dk), (H, dk), (H, dv), (H,), (H,)))
    for r, h in enumerate(seqs):
        n = len(h)
        a, b, c = (F.silu(_conv(h @ w[p + x].T, w[p + x + ".conv"])).view(n, -1, d) for x, d in (("q", dk), ("k", dk), ("v", dv)))
        q[:n, r] = (a / torch.sqrt((a * a).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5).repeat_interleave(H // G, 1)
        k[:n, r] = (b / torch.sqrt((b * b).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
        v[:n, r] = c
        beta[:n, r] = torch.sigmoid(h @ w[p + "b"].T)
        g[:n, r] = torch.exp(-torch.exp(w[p + "A_log"]) * F.softplus(h @ w[p + "a"].T + w[p + "dt_bias"]))
    S, out = torch.zeros(R, H, dk, dv, dtype=torch.float64, device="cuda"), torch.empty_like(v)
    for t in range(T):
        S = S * g[t, :, :, None, None]
        u = beta[t, :, :, None] * (v[t] - (k[t, :, :, None, :] @ S)[:, :, 0])
        S = S + k[t, :, :, :, None] * u[:, :, None, :]
        out[t] = (q[t, :, :, None, :] @ S)[:, :, 0]
    return [((_unit(out[:len(h), r], eps) * w[p + "norm"] * F.silu(h @ w[p + "g"].T).view(-1, H, dv)).reshape(len(h), H * dv)) @ w[p + "o"].T
            for r, h in enumerate(seqs)]


def _window_attention(h, eps, w, p, m):
    H, G, d, dv, T = m["heads"], m["kv_heads"], m["dim"], m["vdim"], len(h)
    q, k, v = (h @ w[p + n].T + w[p + n + ".b"] for n in "qkv")
    q, k = (_unit(q, eps) * w[p + "q.norm"]).view(T, H, d), (_unit(k, eps) * w[p + "k.norm"]).view(T, G, d)
    dims = m["rot"]["dims"]
    f = m["rot"]["base"] ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims)
    ang = torch.arange(T, dtype=torch.float64, device="cuda")[:, None] * f
    c, s = ang.cos()[:, None], ang.sin()[:, None]

    def turn(x):
        a, b, y = x[..., 0:dims:2], x[..., 1:dims:2], x.clone()
        y[..., 0:dims:2], y[..., 1:dims:2] = a * c - b * s, b * c + a * s
        return y

    size, keep = m["mask"]["size"], m["mask"]["keep_first"]
    o = _causal(turn(q), turn(k), v.view(T, G, dv), m["scale"], lambda i, j: (i - j < size) | (j < keep))
    return o.reshape(T, H * dv) @ w[p + "o"].T


def _recurrent_block(seqs, w, p, m):
    Wd, nb, F = m["width"], m["blocks"], torch.nn.functional
    T, R = max(len(h) for h in seqs), len(seqs)
    a, u = (torch.zeros(T, R, Wd, dtype=torch.float64, device="cuda") for _ in range(2))
    for r, h in enumerate(seqs):
        x = _conv(h @ w[p + "x"].T + w[p + "x.b"], w[p + "conv"], w[p + "conv.b"])
        xb = x.view(len(h), nb, Wd // nb)
        gr, gi = (torch.sigmoid(torch.einsum("boi,tbi->tbo", w[p + n], xb) + w[p + n + ".b"]).reshape(len(h), Wd) for n in ("ra", "ri"))
        decay = torch.exp(-8.0 * gr * F.softplus(w[p + "lam"]))
        a[:len(h), r], u[:len(h), r] = decay, torch.sqrt(1.0 - decay * decay) * gi * x
    S, out = torch.zeros(R, Wd, dtype=torch.float64, device="cuda"), torch.empty_like(u)
    for t in range(T):
        S = a[t] * S + u[t]
        out[t] = S
    return [(out[:len(h), r] * F.gelu(h @ w[p + "y"].T + w[p + "y.b"], approximate="tanh")) @ w[p + "o"].T for r, h in enumerate(seqs)]


def _experts(h, w, p, m):
    F, r = torch.nn.functional, m["router"]

    def expert(x, q):
        return (F.silu(x @ w[q + "gate"].T) * (x @ w[q + "up"].T)) @ w[q + "down"].T

    s = torch.sigmoid(h @ w[p + "router"].T)
    choice = s + w[p + "correction"]
    grouped = choice.view(len(h), r["groups"]["count"], -1)
    best = grouped.topk(2, -1).values.sum(-1).topk(r["groups"]["keep"], -1).indices
    allowed = torch.zeros_like(grouped[..., 0], dtype=torch.bool).scatter_(1, best, True)
    ids = grouped.masked_fill(~allowed[..., None], float("-inf")).view(len(h), -1).topk(r["top"], -1).indices
    wt = s.gather(1, ids)
    wt = wt / (wt.sum(-1, keepdim=True) + 1e-20) * r["scale"]
    out = torch.sigmoid(h @ w[p + "shared.sg"].T) * expert(h, p + "shared.")
    for e in range(r["experts"]):
        tok, slot = (ids == e).nonzero(as_tuple=True)
        if len(tok):
            out[tok] += wt[tok, slot][:, None] * expert(h[tok], p + f"e{e}.")
    return out


def _routed_logits(cfg, w, seqs, wanted):
    eps = cfg["norm"]["eps"]
    xs = [w["embed"][torch.tensor(s, device="cuda")].double() for s in seqs]
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        wl = {k: v.double() for k, v in w.items() if k.startswith(p)}
        if layer["type"] == "delta":
            ys = _delta_rule(xs, eps, wl, p + "mix.", m)
        else:
            rec = _recurrent_block(xs, wl, p + "mix.right.", m["right"])
            ys = [m["left_scale"] * _window_attention(x, eps, wl, p + "mix.left.", m["left"]) + m["right_scale"] * r for x, r in zip(xs, rec)]
        xs = [x + _unit(y, eps) * (1 + wl[p + "norm1"]) for x, y in zip(xs, ys)]
        xs = [x + _unit(_experts(x, wl, p + "mlp.", layer["mlp"]), eps) * (1 + wl[p + "norm2"]) for x in xs]
    rows = torch.cat([x[torch.tensor(n, device="cuda")] for x, n in zip(xs, wanted)])
    return (_unit(rows, eps) * (1 + w["final.norm"].double())) @ w["embed"].double().T


@torch.no_grad()
def exact(case, seed):
    contexts, prompts, new = _token_ids(case, seed)
    w, cfg = _weights(case, seed), _config(case)
    seqs = contexts + [a + b for a, b in zip(prompts, new)]
    wanted = [[len(t) - 1] for t in contexts] + [[len(t) - 1 + k for k in range(case["new"] + 1)] for t in prompts]
    logits = (_dense_logits if case["model"] in _DENSE else _routed_logits)(cfg, w, seqs, wanted)
    if case["step"] != "reply":
        return logits
    steps = logits.view(len(prompts), case["new"] + 1, -1)
    return [steps[:, k].contiguous() for k in range(case["new"] + 1)]
