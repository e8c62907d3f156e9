"""What this framework is timed on: requests served from their prompts to their last token.

A case names a model by its layer sizes, a dtype, a number of requests, their prompt lengths (spread evenly between
``low`` and ``high``) and how many tokens each of them draws. One pass hands the requests to an engine that already
holds the weights and the recorded steps, as a server's loop or ``LLM.generate`` does, runs it until they have
finished, and returns the tokens and the logits that each of them was drawn from. ``entry = "trace"`` feeds given
tokens through ``Replayer`` in portions and single steps instead, as ``bin/trace_run`` does.

The weights are random, with one property of a trained model: it is sure of its next token. The embedding's rows carry
the stream (each layer adds a fraction of them), and row t + SHIFT of the output head is row t of the embedding, so
the next token after t is t + SHIFT by a wide margin. Drawn tokens therefore do not hang on the last bit of a sum.
"""

import math

import torch

from tinyserve_b200 import LLM, DecoderModel, Replayer, SamplingParams
from tinyserve_b200.config import config_from_dict

SHIFT = 7919
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
BUDGET = 2048                # tokens a step may carry (the engine's default)

# The dense decoder at the layer sizes of the repository's benchmark: 0.6B and 8B.
DENSE = {
    "0.6b": dict(layers=28, width=1024, heads=16, kv_heads=8, dim=128, ff=3072, vocab=151936),
    "8b": dict(layers=36, width=4096, heads=32, kv_heads=8, dim=128, ff=12288, vocab=151936),
}
# Two of the layered designs at the sizes their benchmark uses (width 1,024).
ATTENTION = {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "scale": 128 ** -0.5}


def guzovik_config():
    windowed = {**ATTENTION, "mask": {"size": 512}}
    latent = {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5,
              "mask": {"size": 1024}, "rot": {"dims": 64, "base": 1e6}}
    moe = {"kind": "moe", "router": {"experts": 16, "top": 3}, "expert": {"ff": 768}, "shared": {"ff": 768}}
    shared = {"type": "attention", "mlp": moe, "mixer": windowed, "weights_of": 2}
    return {"architecture": "Guzovik", "vocab": 32768, "width": 1024, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
            "max_positions": 8192,
            "layers": [{"type": "attention", "mlp": {"kind": "dense", "ff": 3072, "limit": 7.0}, "mixer": windowed},
                       {"type": "latent_attention", "mlp": moe, "mixer": latent},
                       {"type": "attention", "mlp": moe, "mixer": windowed}, shared,
                       {"type": "latent_attention", "mlp": moe, "mixer": latent}, dict(shared)]}


def fegilix_config():
    attn = {**ATTENTION, "rot": {"dims": 128, "base": 1e6}}
    mlp = {"kind": "dense", "ff": 3072}
    mlstm = {"type": "mlstm", "mlp": None, "mixer": {"heads": 8, "dim": 128, "vdim": 128, "gate_cap": 15.0}}
    delta = {"type": "channel_delta", "mlp": None, "mixer": {"heads": 8, "kv_heads": 4, "dim": 128, "vdim": 128, "conv": 4,
                                                             "step_rank": 64, "gate_rank": 64}}
    return {"architecture": "Fegilix", "vocab": 32768, "width": 1024, "norm": {"eps": 1e-5}, "streams": 2,
            "logit_softcap": 30.0, "max_positions": 8192,
            "layers": [mlstm, mlstm, {"type": "attention", "mlp": mlp, "mixer": attn}, delta, mlstm,
                       {"type": "attention", "mlp": mlp, "mixer": {**attn, "kv_from": 2}}]}


def dense_config(s):
    return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "vocab_size": s["vocab"], "hidden_size": s["width"],
            "intermediate_size": s["ff"], "num_hidden_layers": s["layers"], "num_attention_heads": s["heads"],
            "num_key_value_heads": s["kv_heads"], "head_dim": s["dim"], "hidden_act": "silu", "rms_norm_eps": 1e-6,
            "rope_theta": 1e6, "max_position_embeddings": 40960, "tie_word_embeddings": False}


def config_of(case):
    return {"guzovik": guzovik_config, "fegilix": fegilix_config}.get(case["model"], lambda: dense_config(DENSE[case["model"]]))()


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    def case(name, model, dtype, requests, low, high, new, **more):
        return {"name": name, "entry": "engine", "model": model, "dtype": dtype, "requests": requests, "low": low, "high": high,
                "new": new, "chunk": 0, "temperature": 0.0, **more}

    return [
        # one person at a prompt: a short question, the answer token by token (latency of the smallest step)
        case("chat_1", "0.6b", "bfloat16", 1, 37, 37, 48),
        # a handful of conversations with some history, answered together
        case("chat_8", "0.6b", "bfloat16", 8, 700, 1100, 24),
        # a full batch of short jobs, drawn with a temperature
        case("batch_64", "0.6b", "bfloat16", 64, 40, 400, 12, temperature=0.8),
        # one prompt that fills a step: time to the first token
        case("prompt_2048", "0.6b", "bfloat16", 1, 2048, 2048, 1),
        # documents of odd lengths that are only scored: one token each
        case("score_5", "0.6b", "bfloat16", 5, 61, 901, 1),
        # a long document cut into portions of the step's budget
        case("long_9001", "0.6b", "bfloat16", 1, 9001, 9001, 4, chunk=BUDGET),
        # the command line's default dtype, a short question
        case("chat_1_32bit", "0.6b", "float32", 1, 45, 45, 12),
        # given tokens replayed in 32 bits, portions and single tokens mixed, logits of several places
        {"name": "trace_32bit", "entry": "trace", "model": "0.6b", "dtype": "float32", "requests": 3, "low": 70, "high": 150,
         "new": 6, "chunk": 64, "temperature": 0.0},
        # continuous batching with chunked prompts at the larger sizes
        case("mixed_16_8b", "8b", "bfloat16", 16, 60, 700, 12, chunk=512),
        # one conversation at the larger sizes
        case("chat_1_8b", "8b", "bfloat16", 1, 120, 120, 16),
        # a design with routed experts and latent attention
        case("experts_4", "guzovik", "bfloat16", 4, 150, 800, 16),
        # a design with recurrent layers and several lanes of the stream
        case("recurrent_3", "fegilix", "bfloat16", 3, 100, 650, 16),
    ]


def draw(rng):
    def spread(low, high):          # evenly over the logarithm
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["chat", "chat", "batch", "prompt", "long", "32bit", "trace", "8b", "guzovik", "fegilix"])
    case = {"entry": "engine", "model": "0.6b", "dtype": "bfloat16", "requests": 1, "chunk": 0,
            "temperature": rng.choice([0.0, 0.8])}
    most, new = 1100, rng.randint(8, 48)
    if kind == "chat":
        case["requests"] = spread(1, 16)
    elif kind == "batch":
        case["requests"], most, new = spread(16, 64), 400, rng.randint(4, 16)
    elif kind == "prompt":
        case["requests"], most, new = spread(1, 8), BUDGET, 1
    elif kind == "long":
        most, new, case["chunk"] = 9001, rng.randint(1, 8), rng.choice([512, 1000, BUDGET])
    elif kind == "32bit":
        case.update(dtype="float32", requests=spread(1, 4))
        most, new = 150, rng.randint(2, 12)
    elif kind == "trace":
        case.update(entry="trace", dtype="float32", requests=rng.randint(1, 4), chunk=rng.choice([16, 37, 64]), temperature=0.0)
        most, new = 150, rng.randint(2, 8)
    elif kind == "8b":
        case.update(model="8b", requests=spread(1, 8), chunk=rng.choice([0, 512]))
        most, new = 700, rng.randint(4, 12)
    else:
        case.update(model=kind, requests=spread(1, 8))
        most, new = 800, rng.randint(4, 24)
    low = BUDGET + 1 if kind == "long" else 16
    a, b = sorted((spread(low, most), spread(low, most)))
    return {**case, "low": a, "high": b, "new": new}


def prompt_lengths(case):
    """Between ``low`` and ``high``, in an order that is neither rising nor falling."""
    return [case["low"] + int((i * 0.6180339887 % 1.0) * (case["high"] - case["low"])) if i else case["high"]
            for i in range(case["requests"])]


def prompts_of(case, seed):
    g = torch.Generator().manual_seed(1000 + seed)
    vocab = config_of(case).get("vocab") or config_of(case)["vocab_size"]
    return [torch.randint(0, vocab, (n,), generator=g).tolist() for n in prompt_lengths(case)]


# ---------------------------------------------------------------------------------------------- the weights
def weight_shapes(case):
    """(name, shape, mean, deviation) of every tensor, matrices that share an input stacked as the models bind them."""
    c = config_of(case)
    out = []
    matrix = 0.02

    def add(name, *shape, mean=0.0, std=matrix):
        out.append((name, shape, mean, std))

    if case["model"] in DENSE:
        s = DENSE[case["model"]]
        h, ff, q, kv = s["width"], s["ff"], s["heads"] * s["dim"], s["kv_heads"] * s["dim"]
        matrix = 0.02 * (1024 / h) ** 0.5
        for i in range(s["layers"]):
            p = f"model.layers.{i}."
            add(p + "input_layernorm.weight", h, mean=1.0)
            add(p + "self_attn.qkv_proj.weight", q + 2 * kv, h, std=matrix)
            add(p + "self_attn.o_proj.weight", h, q, std=matrix)
            add(p + "self_attn.q_norm.weight", s["dim"], mean=1.0)
            add(p + "self_attn.k_norm.weight", s["dim"], mean=1.0)
            add(p + "post_attention_layernorm.weight", h, mean=1.0)
            add(p + "mlp.gate_up_proj.weight", 2 * ff, h, std=matrix)
            add(p + "mlp.down_proj.weight", h, ff, std=matrix)
        add("model.norm.weight", h, mean=1.0)
        return out
    h = c["width"]
    for i, layer in enumerate(c["layers"]):
        if layer.get("weights_of") is not None:
            continue
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        x = p + "mix."
        if case["model"] == "guzovik":
            add(p + "norm1", h)
            if layer["type"] == "attention":
                add(x + "qkvg", (m["heads"] + 2 * m["kv_heads"]) * m["dim"] + m["heads"], h)
            else:
                add(x + "q+down", m["heads"] * (m["dim"] + m["rot_dim"]) + m["kv_rank"] + m["rot_dim"], h)
                add(x + "dkv.norm", m["kv_rank"], mean=1.0)
                add(x + "uk", m["heads"] * m["dim"], m["kv_rank"])
                add(x + "uv", m["heads"] * m["vdim"], m["kv_rank"])
            add(x + "o", h, m["heads"] * m["vdim"])
            for n in ("norm1b", "norm2", "norm2b"):
                add(p + n, h)
            for n in ("ls1", "ls2"):
                add(p + n, h, mean=0.3, std=0.03)
            if mlp["kind"] == "dense":
                add(p + "mlp.gate+up", 2 * mlp["ff"], h)
                add(p + "mlp.down", h, mlp["ff"])
            else:
                e, ff = mlp["router"]["experts"], mlp["expert"]["ff"]
                add(p + "mlp.router", e, h, std=0.06)
                add(p + "mlp.experts.gate+up", 2 * e * ff, h)
                add(p + "mlp.experts.down", e * h, ff)
                add(p + "mlp.shared.gate+up", 2 * mlp["shared"]["ff"], h)
                add(p + "mlp.shared.down", h, mlp["shared"]["ff"])
            continue
        heads, d, dv = m["heads"], m["dim"], m["vdim"]
        for k in (1, 2) if mlp else (1,):
            add(p + f"norm{k}", h, mean=1.0)
            add(p + f"hc{k}.in", 2, mean=0.7, std=0.1)
            add(p + f"hc{k}.out", 2, mean=0.7, std=0.1)
            add(p + f"hc{k}.mix", 2, 2, std=0.1)
        if layer["type"] == "mlstm":
            add(x + "qkvg", 2 * heads * d + 2 * heads * dv, h)
            add(x + "if", 2 * heads, h)
            add(x + "if.b", 2 * heads, std=1.0)
            add(x + "norm", heads * dv, mean=1.0)
        elif layer["type"] == "attention":
            if m.get("kv_from") is None:
                add(x + "qkvg", (heads + 2 * m["kv_heads"]) * d + heads * dv, h)
                add(x + "k.norm", d, mean=1.0)
            else:
                add(x + "qg", heads * (d + dv), h)
            add(x + "q.norm", d, mean=1.0)
            add(x + "sink", heads, std=1.0)
        else:
            c_qkv = 2 * m["kv_heads"] * d + heads * dv
            add(x + "qkv", c_qkv, h)
            add(x + "qkv.conv", c_qkv, m["conv"], std=0.3)
            add(x + "b", heads, h)
            add(x + "A_log", heads, std=0.5)
            add(x + "norm", dv, mean=1.0)
            add(x + "a1", m["step_rank"], h)
            add(x + "a2", heads * d, m["step_rank"])
            add(x + "dt_bias", heads * d, std=1.0)
            add(x + "g1", m["gate_rank"], h)
            add(x + "g2", heads * dv, m["gate_rank"])
        add(x + "o", h, heads * dv)
        if mlp:
            add(p + "mlp.gate+up", 2 * mlp["ff"], h)
            add(p + "mlp.down", h, mlp["ff"])
    add("final.norm", h, mean=1.0 if case["model"] == "fegilix" else 0.0)
    return out


def weights_of(case, seed):
    c, dtype = config_of(case), DTYPES[case["dtype"]]
    dense = case["model"] in DENSE
    vocab, h = (c["vocab_size"], c["hidden_size"]) if dense else (c["vocab"], c["width"])
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = {}
    for name, shape, mean, std in weight_shapes(case):
        w[name] = torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(mean, std, generator=g).to(dtype)
        if name.endswith(".mix") and shape == (2, 2):
            w[name] += torch.eye(2, dtype=dtype, device="cuda")
    table = torch.empty((vocab, h), dtype=torch.bfloat16, device="cuda").normal_(0.0, 1.0, generator=g).to(dtype)
    w["model.embed_tokens.weight" if dense else "embed"] = table
    w["lm_head.weight" if dense else "head"] = torch.roll(table, SHIFT, 0) * 0.125
    return w


# ------------------------------------------------------------------------------------------------ one pass
def trace_steps(case, seed):
    """Steps of (request, tokens, wanted places): every request starts one step after the one before it, brings its
    prompt in portions of ``chunk`` tokens and then single tokens; logits of each portion's first and last place."""
    given = [p + [(p[-1] + SHIFT * (j + 1)) % DENSE[case["model"]]["vocab"] for j in range(case["new"])]
             for p in prompts_of(case, seed)]
    cuts = []
    for p in given:
        n = len(p) - case["new"]
        at = list(range(0, n, case["chunk"])) + list(range(n, len(p) + 1))
        cuts.append([(a, b) for a, b in zip(at, at[1:])])
    steps = []
    for s in range(max(i + len(c) for i, c in enumerate(cuts))):
        entries = []
        for i, c in enumerate(cuts):
            if 0 <= s - i < len(c):
                a, b = c[s - i]
                entries.append((i, a, given[i][a:b], sorted({0, b - a - 1})))
        steps.append((entries, [i for i, c in enumerate(cuts) if s - i == len(c) - 1]))
    return steps, given


def prepare(case, seed):
    model = DecoderModel(config_from_dict(config_of(case)), weights_of(case, seed), DTYPES[case["dtype"]], "cuda")
    if case["entry"] == "trace":
        steps, given = trace_steps(case, seed)
        room = sum(-(-len(p) // 64) * 64 for p in given)
        return {"case": case, "steps": steps, "replayer": Replayer(model, room, max_live=len(given))}
    prompts = prompts_of(case, seed)
    pages = sum(-(-(len(p) + case["new"]) // 16) for p in prompts)
    llm = LLM(model, num_pages=pages, max_num_seqs=len(prompts), max_batch_tokens=case["chunk"] or BUDGET,
              chunked_prefill=bool(case["chunk"]), record_logits=True)
    sampling = [SamplingParams(case["temperature"], 0.95, seed=i) if case["temperature"] else None for i in range(len(prompts))]
    return {"case": case, "prompts": prompts, "engine": llm.engine, "sampling": sampling}


def run(state):
    case = state["case"]
    if case["entry"] == "trace":
        rows = []
        for entries, end in state["steps"]:
            logits = state["replayer"].run_step([(str(i), tokens, places) for i, _, tokens, places in entries],
                                                end=[str(i) for i in end])
            rows.append(logits.clone())
        return {"logits": torch.cat(rows)}
    engine = state["engine"]
    ids = [engine.add_request(p, case["new"], sampling=s) for p, s in zip(state["prompts"], state["sampling"])]
    while engine.has_work():
        engine.step()
    tokens = [engine.requests[i].output for i in ids]
    rows = {i: [] for i in ids}
    for i, _, row in engine.logits_log:
        rows[i].append(row)
    engine.logits_log.clear()
    for i in ids:
        engine.release(i)
    return {"tokens": torch.tensor(tokens), "logits": torch.stack([row for i in ids for row in rows[i]])}


# ------------------------------------------------------------------- the same in 64 bits, from the formulas
def rms(x, weight, eps):
    x = x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps)
    return x if weight is None else x * weight


def turn(x, pos, base, dims, neighbours=False):
    """``x [T, H, D]``: the first ``dims`` elements of a head turn, in pairs (i, i + dims / 2) or neighbours."""
    f = base ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=x.device) / dims)
    a = (pos.double()[:, None] * f)[:, None, :]
    c, s = a.cos(), a.sin()
    out = x.clone()
    u, v = (slice(0, dims, 2), slice(1, dims, 2)) if neighbours else (slice(0, dims // 2), slice(dims // 2, dims))
    out[..., u], out[..., v] = x[..., u] * c - x[..., v] * s, x[..., v] * c + x[..., u] * s
    return out


def attend(q, k, v, scale, window=None, sink=None):
    """Causal softmax attention of one sequence, heads in groups; ``sink [H]``: one more score that carries no value."""
    t, heads, groups = q.shape[0], q.shape[1], k.shape[1]
    rep = heads // groups
    k, v = k.permute(1, 2, 0), v.transpose(0, 1)
    j = torch.arange(t, device=q.device)
    out = torch.empty(t, heads, v.shape[-1], dtype=q.dtype, device=q.device)
    for a in range(0, t, 512):
        b = min(a + 512, t)
        first = 0 if window is None else max(0, a - window + 1)
        i = j[a:b, None]
        hidden = j[None, first:b] > i
        if window is not None:
            hidden = hidden | (j[None, first:b] <= i - window)
        for g in range(groups):
            s = torch.matmul(q[a:b, g * rep:(g + 1) * rep].transpose(0, 1), k[g, :, first:b]) * scale
            s = s.masked_fill(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[g * rep:(g + 1) * rep, None, None].expand(-1, b - a, 1)], -1)
            p = torch.softmax(s, -1)[..., : b - first]
            out[a:b, g * rep:(g + 1) * rep] = torch.matmul(p, v[g, first:b]).transpose(0, 1)
    return out


def silu(z):
    return z * torch.sigmoid(z)


class Sequences:
    """Several token sequences in one ``[T, ...]`` tensor."""

    def __init__(self, ids):
        self.parts, at = [], 0
        for p in ids:
            self.parts.append(slice(at, at + len(p)))
            at += len(p)
        self.ids = torch.tensor([t for p in ids for t in p], device="cuda")
        self.pos = torch.cat([torch.arange(len(p), device="cuda") for p in ids])

    def each(self, f, *x):
        return torch.cat([f(*(y[p] for y in x)) for p in self.parts])


def dense_stream(case, w, seqs):
    s = DENSE[case["model"]]
    nq, nkv, d, eps = s["heads"], s["kv_heads"], s["dim"], 1e-6
    x = w("model.embed_tokens.weight", seqs.ids)
    for i in range(s["layers"]):
        p = f"model.layers.{i}."
        h = rms(x, w(p + "input_layernorm.weight"), eps)
        qkv = (h @ w(p + "self_attn.qkv_proj.weight").T).view(len(x), nq + 2 * nkv, d)
        q = turn(rms(qkv[:, :nq], w(p + "self_attn.q_norm.weight"), eps), seqs.pos, 1e6, d)
        k = turn(rms(qkv[:, nq:nq + nkv], w(p + "self_attn.k_norm.weight"), eps), seqs.pos, 1e6, d)
        a = seqs.each(lambda q, k, v: attend(q, k, v, d ** -0.5), q, k, qkv[:, nq + nkv:])
        x = x + a.reshape(len(x), -1) @ w(p + "self_attn.o_proj.weight").T
        gate, up = (rms(x, w(p + "post_attention_layernorm.weight"), eps) @ w(p + "mlp.gate_up_proj.weight").T).chunk(2, -1)
        x = x + (silu(gate) * up) @ w(p + "mlp.down_proj.weight").T
    return rms(x, w("model.norm.weight"), eps)


def guzovik_stream(case, w, seqs):
    c = config_of(case)
    eps = c["norm"]["eps"]
    x = w("embed", seqs.ids) * c["embedding"]["scale"]
    t = len(x)
    for i, layer in enumerate(c["layers"]):
        p, m, mlp = f"l{layer.get('weights_of', i)}.", layer["mixer"], layer["mlp"]
        u, heads, d = p + "mix.", m["heads"], m["dim"]
        h = rms(x, 1.0 + w(p + "norm1"), eps)
        window = m["mask"]["size"]
        if layer["type"] == "attention":
            n, g = heads * d, m["kv_heads"] * d
            q, k, v, gate = (h @ w(u + "qkvg").T).split([n, g, g, heads], -1)
            zero = torch.zeros(heads, dtype=x.dtype, device=x.device)
            y = seqs.each(lambda q, k, v: attend(q, k, v, m["scale"], window, zero), q.view(t, heads, d), k.view(t, -1, d), v.view(t, -1, d))
            y = y * torch.sigmoid(gate)[:, :, None]
        else:
            dr, rank = m["rot_dim"], m["kv_rank"]
            q, lat, kr = (h @ w(u + "q+down").T).split([heads * (d + dr), rank, dr], -1)
            q = q.view(t, heads, d + dr)
            lat = rms(lat, w(u + "dkv.norm"), eps)
            kr = turn(kr[:, None], seqs.pos, m["rot"]["base"], m["rot"]["dims"], True).expand(t, heads, dr)
            q = torch.cat([q[..., :d], turn(q[..., d:], seqs.pos, m["rot"]["base"], m["rot"]["dims"], True)], -1)
            k = torch.cat([(lat @ w(u + "uk").T).view(t, heads, d), kr], -1)
            v = (lat @ w(u + "uv").T).view(t, heads, m["vdim"])
            y = seqs.each(lambda q, k, v: attend(q, k, v, m["scale"], window), q, k, v)
        x = x + rms(y.reshape(t, -1) @ w(u + "o").T, 1.0 + w(p + "norm1b"), eps) * w(p + "ls1")
        h = rms(x, 1.0 + w(p + "norm2"), eps)
        u = p + "mlp."
        if mlp["kind"] == "dense":
            gate, up = (h @ w(u + "gate+up").T).chunk(2, -1)
            gate, up = gate.clamp(max=mlp["limit"]), up.clamp(-mlp["limit"], mlp["limit"])
            y = (gate * torch.sigmoid(1.702 * gate) * (up + 1.0)) @ w(u + "down").T
        else:
            best, ids = (h @ w(u + "router").T).topk(mlp["router"]["top"], -1)
            share = torch.softmax(best, -1)
            gate, up = (h @ w(u + "shared.gate+up").T).chunk(2, -1)
            y = (silu(gate) * up) @ w(u + "shared.down").T
            e, ff = mlp["router"]["experts"], mlp["expert"]["ff"]
            both, down = w(u + "experts.gate+up").view(e, 2 * ff, -1), w(u + "experts.down").view(e, -1, ff)
            for n in range(e):
                row, place = (ids == n).nonzero(as_tuple=True)
                gate, up = (h[row] @ both[n].T).chunk(2, -1)
                y = y.index_add(0, row, ((silu(gate) * up) @ down[n].T) * share[row, place, None])
        x = x + rms(y, 1.0 + w(p + "norm2b"), eps) * w(p + "ls2")
    return rms(x, 1.0 + w("final.norm"), eps)


def matrix_memory(q, k, v, log_i, log_f):
    """S <- f S + i k v^T, n <- f n + i k, o = S^T q / max(|n q|, 1), kept in the scale of a running maximum."""
    s = torch.zeros(*k.shape[1:], v.shape[-1], dtype=q.dtype, device=q.device)
    n, m, out = torch.zeros_like(k[0]), torch.zeros_like(log_i[0]), []
    for a, b, c, i, f in zip(q, k, v, log_i, log_f):
        top = torch.maximum(f + m, i)
        keep, take, m = torch.exp(f + m - top), torch.exp(i - top), top
        s = keep[:, None, None] * s + take[:, None, None] * (b[:, :, None] * c[:, None, :])
        n = keep[:, None] * n + take[:, None] * b
        den = torch.maximum((n * a).sum(-1).abs(), torch.exp(-m)) + 1e-6
        out.append((s * a[:, :, None]).sum(1) / den[:, None])
    return torch.stack(out)


def delta_rule(q, k, v, beta, decay):
    """S <- decay S; S <- S + k (beta (v - S^T k))^T; o = S^T q."""
    s, out = torch.zeros(*k.shape[1:], v.shape[-1], dtype=q.dtype, device=q.device), []
    for a, b, c, e, f in zip(q, k, v, beta, decay):
        s = f[:, :, None] * s
        s = s + b[:, :, None] * (e[:, None] * (c - (s * b[:, :, None]).sum(1)))[:, None, :]
        out.append((s * a[:, :, None]).sum(1))
    return torch.stack(out)


def convolve(x, taps):
    k = taps.shape[1]
    pad = torch.cat([x.new_zeros(k - 1, x.shape[1]), x])
    return silu(sum(pad[j:j + len(x)] * taps[:, j] for j in range(k)))


def fegilix_stream(case, w, seqs):
    c = config_of(case)
    eps, t = c["norm"]["eps"], len(seqs.ids)
    lanes = [w("embed", seqs.ids)] * 2
    kept = {}

    def mix(i, layer, h):
        m, u = layer["mixer"], f"l{i}.mix."
        heads, d, dv = m["heads"], m["dim"], m["vdim"]
        if layer["type"] == "attention":
            own = m.get("kv_from") is None
            n, g = heads * d, m.get("kv_heads", heads) * d
            got = (h @ w(u + ("qkvg" if own else "qg")).T).split([n, g, g, n] if own else [n, n], -1)
            q = turn(rms(got[0].view(t, heads, d), w(u + "q.norm"), eps), seqs.pos, m["rot"]["base"], d)
            if own:
                kept[i] = (turn(rms(got[1].view(t, -1, d), w(u + "k.norm"), eps), seqs.pos, m["rot"]["base"], d), got[2].view(t, -1, d))
            k, v = kept[i if own else m["kv_from"]]
            sink = w(u + "sink")
            y = seqs.each(lambda q, k, v: attend(q, k, v, m["scale"], None, sink), q, k, v).reshape(t, -1) * torch.sigmoid(got[-1])
        elif layer["type"] == "mlstm":
            q, k, v, gate = (z.view(t, heads, -1) for z in (h @ w(u + "qkvg").T).chunk(4, -1))
            i_f = m["gate_cap"] * torch.tanh((h @ w(u + "if").T + w(u + "if.b")) / m["gate_cap"])
            y = seqs.each(matrix_memory, q * d ** -0.5, k, v, i_f[:, :heads], torch.nn.functional.logsigmoid(i_f[:, heads:]))
            y = rms(y, None, eps).reshape(t, -1) * w(u + "norm") * torch.sigmoid(gate.reshape(t, -1))
        else:
            g = m["kv_heads"]
            qkv = seqs.each(lambda z: convolve(z, w(u + "qkv.conv")), h @ w(u + "qkv").T)
            q, k, v = (z.reshape(t, -1, d) for z in qkv.split([g * d, g * d, heads * dv], -1))
            q, k = (z / torch.sqrt(z.pow(2).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
            q, k = (q * d ** -0.5).repeat_interleave(heads // g, 1), k.repeat_interleave(heads // g, 1)
            step = torch.nn.functional.softplus((h @ w(u + "a1").T) @ w(u + "a2").T + w(u + "dt_bias")).view(t, heads, d)
            y = seqs.each(delta_rule, q, k, v, torch.sigmoid(h @ w(u + "b").T), torch.exp(-torch.exp(w(u + "A_log"))[:, None] * step))
            y = rms(y, w(u + "norm"), eps).reshape(t, -1) * torch.sigmoid((h @ w(u + "g1").T) @ w(u + "g2").T)
        return y @ w(u + "o").T

    def feed(i, h):
        gate, up = (h @ w(f"l{i}.mlp.gate+up").T).chunk(2, -1)
        return (torch.nn.functional.gelu(gate, approximate="tanh") * up) @ w(f"l{i}.mlp.down").T

    for i, layer in enumerate(c["layers"]):
        for k in (1, 2) if layer["mlp"] else (1,):
            take, put, across = (w(f"l{i}.hc{k}.{n}") for n in ("in", "out", "mix"))
            h = rms(take[0] * lanes[0] + take[1] * lanes[1], w(f"l{i}.norm{k}"), eps)
            y = mix(i, layer, h) if k == 1 else feed(i, h)
            lanes = [across[0, j] * lanes[0] + across[1, j] * lanes[1] + put[j] * y for j in range(2)]
    return rms(lanes[0] + lanes[1], w("final.norm"), eps)


@torch.inference_mode()
def exact(case, seed):
    tensors = weights_of(case, seed)

    def w(name, rows=None):
        return (tensors[name] if rows is None else tensors[name][rows]).double()

    stream = {"guzovik": guzovik_stream, "fegilix": fegilix_stream}.get(case["model"], dense_stream)
    head = w("lm_head.weight" if case["model"] in DENSE else "head")
    vocab = head.shape[0]

    def logits_at(ids, places):
        seqs = Sequences(ids)
        rows = torch.tensor([seqs.parts[i].start + p for i, p in places], device="cuda")
        z = stream(case, w, seqs)[rows] @ head.T
        return 30.0 * torch.tanh(z / 30.0) if case["model"] == "fegilix" else z

    if case["entry"] == "trace":
        steps, given = trace_steps(case, seed)
        return {"logits": logits_at(given, [(i, a + p) for entries, _ in steps for i, a, _, places in entries for p in places])}
    prompts, new = prompts_of(case, seed), case["new"]
    drawn = [[(p[-1] + SHIFT * (j + 1)) % vocab for j in range(new)] for p in prompts]
    while True:
        z = logits_at([p + d[:-1] for p, d in zip(prompts, drawn)], [(i, len(p) - 1 + j) for i, p in enumerate(prompts) for j in range(new)])
        best = z.argmax(-1).view(len(prompts), new).tolist()
        if best == drawn:
            return {"tokens": torch.tensor(drawn), "logits": z}
        drawn = best         # a token that is not the expected one: once more with what was drawn instead


# ----------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Every step reads the weights once (they are larger than the L2 cache) and the rows of the cache that its queries
    see; the logits are written. Steps: the prompts at the step's budget, then one for each further token."""
    shapes = weight_shapes(case)
    size = 4 if case["dtype"] == "float32" else 2
    c = config_of(case)
    dense = case["model"] in DENSE
    vocab, h = (c["vocab_size"], c["hidden_size"]) if dense else (c["vocab"], c["width"])
    lengths, new = prompt_lengths(case), case["new"]
    if case["entry"] == "trace":
        steps, given = trace_steps(case, 0)
        step_tokens = [sum(len(t) for _, _, t, _ in entries) for entries, _ in steps]
        rows = sum(len(places) for entries, _ in steps for _, _, _, places in entries)
        lengths, new, head_reads = [len(g) for g in given], 1, len(steps)
    else:
        per_step = case["chunk"] or BUDGET
        step_tokens = [min(per_step, sum(lengths) - a) for a in range(0, sum(lengths), per_step)] + [len(lengths)] * (new - 1)
        rows, head_reads = len(lengths) * new, new
    tokens = sum(step_tokens)
    bytes_, flops = 0.0, 0.0
    for name, shape, _, _ in shapes:
        n, uses = math.prod(shape), 1
        if not dense:       # a layer that runs on another's tensors reads them again
            uses += sum(f"l{layer.get('weights_of')}." == name.split(".")[0] + "." for layer in c["layers"])
        if ".experts." in name:
            bytes_ += uses * size * n / 16 * sum(min(16.0, 3.0 * t) for t in step_tokens)
            flops += uses * 2.0 * n * tokens * 3 / 16
        else:
            bytes_ += uses * size * n * len(step_tokens)
            flops += uses * 2.0 * n * tokens if len(shape) == 2 else 0.0
    bytes_ += vocab * h * size * head_reads + tokens * h * size + 4.0 * rows * vocab
    flops += 2.0 * rows * vocab * h
    if dense:
        s = DENSE[case["model"]]
        layers, heads, kv, d, span = s["layers"], s["heads"], 2 * s["kv_heads"] * s["dim"], s["dim"], 1 << 30
    elif case["model"] == "guzovik":
        layers, heads, kv, d, span = 6, 16, 1536, 128, 683      # four windows of 512 and two of 1,024 positions
    else:
        layers, heads, kv, d, span = 2, 16, 2048, 128, 1 << 30
    for n in lengths:
        seen = [min(p + 1, span) for p in range(n + new - 1)]
        flops += 4.0 * layers * heads * d * sum(seen)
        bytes_ += layers * kv * size * (n + sum(seen[n:]))
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 0.03, "max": 0.5}
