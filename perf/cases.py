"""Steps of served models whose speed is followed: what is run, on what, and how exact it has to be.

Every case is a model with random weights behind an ``Engine`` and one piece of work that a serving program
has it do:

* ``decode``: one more token for each of a batch of requests that hold cached tokens;
* ``prompt``: a new request's whole prompt, logits at its last token;
* ``portion``: the next stretch of a long prompt, on what the cache already holds of it;
* ``mixed``: portions of two prompts beside the single tokens of running requests (continuous batching);
* ``score``: a text's logits at every token (how likely a model finds it), the use of the float32 path;
* ``turn``: whole short requests: a batch of prompts, then a few tokens for each, one step a token.

Models: the layer sizes of Llama 3.2 1B and 3B and of Llama 3.1 8B (some with fewer layers than those models have:
all layers of a model are alike), and two designs whose layers differ: Zeladra (attention over a cached latent, a state-space
mixer, windowed attention with kept first positions, two residual streams) and Pegurax (attention inside chunks
beside a gated delta rule, a selective scan).  Between them they hold every kind of mixer whose prompt and
single-token forms differ: paged keys and values, one latent a token, and states of fixed size.

``exact`` computes the same logits in 64 bits from the same weights, in whole sequences and without a cache.
"""

from __future__ import annotations

import math

import torch

PAGE = 64
VOCAB = 128256

#: layer sizes of the Llama shapes (width, query heads, key/value heads, head size, feed-forward width, factor of the rotation's scaling)
LLAMA = {
    "llama-1b": (2048, 32, 8, 64, 8192, 32.0),
    "llama-3b": (3072, 24, 8, 128, 8192, 32.0),
    "llama-8b": (4096, 32, 8, 128, 14336, 8.0),
}
#: width, heads, key/value heads, head size, feed-forward width, window or chunk of the two other designs
DESIGN = {
    "zeladra": (2048, 32, 8, 64, 8192, 1024),
    "pegurax": (2048, 32, 8, 64, 8192, 1024),
}


def listed():
    return [
        # the smallest step: one chat request on the smallest model, all its layers
        dict(name="decode 1b b1", model="llama-1b", dtype="bf16", layers=16, mode="decode", batch=1, context=300),
        # the benchmark's decode: batch 8 at a context of 4,096
        dict(name="decode 8b b8 ctx4096", model="llama-8b", dtype="bf16", layers=8, mode="decode", batch=8, context=4096),
        # a full batch of requests of all lengths
        dict(name="decode 3b b64 ragged", model="llama-3b", dtype="bf16", layers=8, mode="decode", batch=64, context=1400),
        # two readers of long documents
        dict(name="decode 1b b2 ctx30000", model="llama-1b", dtype="bf16", layers=8, mode="decode", batch=2, context=30000),
        # the benchmark's prompt
        dict(name="prompt 8b 2048", model="llama-8b", dtype="bf16", layers=8, mode="prompt", tokens=2048),
        # a step of continuous batching: two portions beside twenty running requests
        dict(name="mixed 3b 700+20", model="llama-3b", dtype="bf16", layers=8, mode="mixed", tokens=700, batch=20, context=900),
        # the last portion of a long document
        dict(name="portion 8b 512 on 16384", model="llama-8b", dtype="bf16", layers=4, mode="portion", tokens=512, context=16384),
        # likelihood of a text in float32, and a few float32 requests being decoded
        dict(name="score 1b f32 777", model="llama-1b", dtype="f32", layers=4, mode="score", tokens=777),
        dict(name="decode 1b f32 b5", model="llama-1b", dtype="f32", layers=4, mode="decode", batch=5, context=500),
        # the designs with layers of several kinds: prompts, one of them of an odd length, and whole short requests
        dict(name="prompt zeladra 2048", model="zeladra", dtype="bf16", layers=6, mode="prompt", tokens=2048),
        dict(name="prompt pegurax 1501", model="pegurax", dtype="bf16", layers=4, mode="prompt", tokens=1501),
        dict(name="turn zeladra b4 200+12", model="zeladra", dtype="bf16", layers=3, mode="turn", batch=4, tokens=200, new=12),
    ]


def _log(rng, lo, hi):
    """A whole number from ``lo`` to ``hi``, spread evenly over its logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    """One more case: any model and piece of work of the list, at sizes up to those of the list."""
    kind = rng.choice(["decode", "decode", "long", "prompt", "portion", "mixed", "f32", "f32", "design", "design", "design"])
    model = rng.choice(["llama-1b", "llama-3b", "llama-8b"])
    if kind == "decode":
        batch = _log(rng, 1, 64)
        context = _log(rng, 20, min(4096, 64000 // batch))
        return dict(model=model, dtype="bf16", layers=rng.randint(4, 8), mode="decode", batch=batch, context=context)
    if kind == "long":
        return dict(model="llama-1b", dtype="bf16", layers=rng.randint(4, 8), mode="decode", batch=rng.randint(1, 2),
                    context=_log(rng, 4096, 30000))
    if kind == "prompt":
        return dict(model=model, dtype="bf16", layers=rng.randint(4, 8), mode="prompt", tokens=_log(rng, 9, 2048))
    if kind == "portion":
        return dict(model=model, dtype="bf16", layers=rng.randint(2, 4), mode="portion", tokens=_log(rng, 16, 512),
                    context=_log(rng, 300, 16384))
    if kind == "mixed":
        return dict(model=model, dtype="bf16", layers=rng.randint(4, 8), mode="mixed", tokens=_log(rng, 32, 1000),
                    batch=rng.randint(2, 30), context=_log(rng, 60, 1200))
    if kind == "f32":
        model = rng.choice(["llama-1b", "llama-3b"])
        if rng.random() < 0.5:
            return dict(model=model, dtype="f32", layers=rng.randint(2, 4), mode="score", tokens=_log(rng, 5, 600))
        return dict(model=model, dtype="f32", layers=rng.randint(2, 4), mode="decode", batch=_log(rng, 1, 16),
                    context=_log(rng, 20, 700))
    model = rng.choice(["zeladra", "pegurax"])
    layers = 3 * rng.randint(1, 2) if model == "zeladra" else 2 * rng.randint(1, 2)
    if rng.random() < 0.5:
        return dict(model=model, dtype="bf16", layers=layers, mode="prompt", tokens=_log(rng, 40, 2048))
    return dict(model=model, dtype="bf16", layers=layers, mode="turn", batch=_log(rng, 1, 8), tokens=_log(rng, 10, 300),
                new=rng.randint(4, 12))


# -- what a case's model is ----------------------------------------------------------------------


def _llama_config(case):
    width, heads, kv, size, ffn, factor = LLAMA[case["model"]]
    return dict(architectures=["LlamaForCausalLM"], hidden_size=width, intermediate_size=ffn,
                num_hidden_layers=case["layers"], num_attention_heads=heads, num_key_value_heads=kv, head_dim=size,
                rms_norm_eps=1e-5, vocab_size=VOCAB, tie_word_embeddings=False, rope_theta=500000.0,
                rope_scaling=dict(factor=factor, low_freq_factor=1.0, high_freq_factor=4.0,
                                  original_max_position_embeddings=8192, rope_type="llama3"),
                max_position_embeddings=131072)


def _zeladra_config(case):
    width, heads, kv, d, ffn, window = DESIGN["zeladra"]
    latent = dict(heads=heads, dim=d, rot_dim=d // 2, vdim=d, q_rank=width * 3 // 4, kv_rank=4 * d, scale=(d * 3 // 2) ** -0.5,
                  rot=dict(dims=d // 2, base=500000.0, scaling=dict(factor=4.0, original=8192, fast=32.0, slow=1.0)))
    ssm = dict(heads=2 * width // 64, vdim=64, state=128, groups=8, conv=4, norm_groups=8)
    att = dict(heads=heads, kv_heads=kv, dim=d, vdim=d, scale=d ** -0.5, rot=dict(dims=d, base=500000.0),
               mask=dict(size=window, keep_first=4))
    layers = []
    for i in range(case["layers"]):
        kind = ("latent_attention", "mamba2", "attention")[i % 3]
        mixer = dict(dict(latent_attention=latent, mamba2=ssm, attention=att)[kind])
        if kind == "latent_attention" and i:
            mixer["kv_from"] = 0  # it reads the first latent layer's cache
        layers.append(dict(type=kind, mixer=mixer, mlp=dict(kind="dense", ff=ffn)))
    return dict(architecture="Zeladra", vocab=VOCAB, width=width, norm=dict(eps=1e-5), embedding=dict(scale=1.0), streams=2,
                layers=layers)


def _pegurax_config(case):
    width, heads, kv, d, ffn, chunk = DESIGN["pegurax"]
    left = dict(heads=heads // 2, kv_heads=kv // 2, dim=d, vdim=d, scale=d ** -0.5, mask=dict(size=chunk),
                rot=dict(dims=d, base=500000.0, scaling=dict(factor=8.0, original=8192, fast=32.0, slow=1.0)))
    right = dict(heads=heads // 2, kv_heads=kv // 2, dim=d, vdim=d, conv=4)
    scan = dict(inner=width, state=16, dt_rank=width // 16, conv=4)
    layers = []
    for i in range(case["layers"]):
        mlp = dict(kind="dense", ff=ffn)
        if i % 2 == 0:
            layers.append(dict(type="parallel", mixer=dict(left=dict(left), right=dict(right), left_scale=0.8, right_scale=0.5),
                               mlp=mlp))
        else:
            layers.append(dict(type="mamba1", mixer=dict(scan), mlp=mlp))
    return dict(architecture="Pegurax", vocab=VOCAB, width=width, norm=dict(eps=1e-5), embedding=dict(scale=1.0), layers=layers)


def _config(case):
    return {"zeladra": _zeladra_config, "pegurax": _pegurax_config}.get(case["model"], _llama_config)(case)


def _tensors(case):
    """Names, shapes and laws of a checkpoint: ("normal", deviation), ("near one",) or ("uniform", from, to)."""
    out = []

    def matrix(name, *shape):
        # The maps into the residual stream are smaller, by the root of their number, and the stream starts with
        # deviation 1: no single layer drowns the others, as in a trained model.
        last = name.removesuffix(".weight").rpartition(".")[2]
        deep = last in ("o", "down", "o_proj", "down_proj")
        out.append((name, shape, ("normal", 1.0 if "embed" in name else 0.02 / math.sqrt(2 * case["layers"]) if deep else 0.02)))

    def norm(name, n):
        out.append((name, (n,), ("near one",)))

    def uniform(name, shape, lo, hi):
        out.append((name, shape, ("uniform", lo, hi)))

    if case["model"] in LLAMA:
        w, heads, kv, d, ffn, _ = LLAMA[case["model"]]
        matrix("model.embed_tokens.weight", VOCAB, w)
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            norm(p + "input_layernorm.weight", w)
            matrix(p + "self_attn.q_proj.weight", heads * d, w)
            matrix(p + "self_attn.k_proj.weight", kv * d, w)
            matrix(p + "self_attn.v_proj.weight", kv * d, w)
            matrix(p + "self_attn.o_proj.weight", w, heads * d)
            norm(p + "post_attention_layernorm.weight", w)
            matrix(p + "mlp.gate_proj.weight", ffn, w)
            matrix(p + "mlp.up_proj.weight", ffn, w)
            matrix(p + "mlp.down_proj.weight", w, ffn)
        norm("model.norm.weight", w)
        matrix("lm_head.weight", VOCAB, w)
        return out
    config = _config(case)
    w, zeladra = config["width"], case["model"] == "zeladra"
    matrix("embed", VOCAB, w)
    for i, layer in enumerate(config["layers"]):
        p, x, m = f"l{i}.", f"l{i}.mix.", layer["mixer"]
        for n in ("norm1", "norm2") if zeladra else ("norm1", "norm1b", "ls1", "norm2", "norm2b", "ls2"):
            norm(p + n, w)
        if zeladra:
            out.append((p + "norm1.b", (w,), ("normal", 0.02)))
            out.append((p + "norm2.b", (w,), ("normal", 0.02)))
            for q in ("hc1.", "hc2."):
                uniform(p + q + "in", (2,), 0.3, 0.9)
                uniform(p + q + "out", (2,), 0.5, 1.0)
                uniform(p + q + "mix", (2, 2), 0.1, 0.7)
        if layer["type"] == "latent_attention":
            h, d, r, e, rank = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            matrix(x + "dq", m["q_rank"], w)
            norm(x + "dq.norm", m["q_rank"])
            matrix(x + "uq", h * (d + r), m["q_rank"])
            if "kv_from" not in m:
                matrix(x + "dkv", rank + r, w)
                norm(x + "dkv.norm", rank)
            matrix(x + "uk", h * d, rank)
            matrix(x + "uv", h * e, rank)
            matrix(x + "g", h, w)
            matrix(x + "o", w, h * e)
        elif layer["type"] == "mamba2":
            h, inner = m["heads"], m["heads"] * m["vdim"]
            channels = inner + 2 * m["groups"] * m["state"]
            matrix(x + "in", inner + channels + h, w)
            out.append((x + "conv", (channels, m["conv"]), ("normal", 0.3)))
            out.append((x + "conv.b", (channels,), ("normal", 0.1)))
            uniform(x + "dt_bias", (h,), -3.0, 0.5)
            uniform(x + "A_log", (h,), -1.0, 1.5)
            norm(x + "D", h)
            norm(x + "norm", inner)
            matrix(x + "o", w, inner)
        elif layer["type"] == "attention":
            d = m["dim"]
            matrix(x + "q", m["heads"] * d, w)
            matrix(x + "k", m["kv_heads"] * d, w)
            matrix(x + "v", m["kv_heads"] * d, w)
            matrix(x + "o", w, m["heads"] * d)
        elif layer["type"] == "parallel":
            l, r = m["left"], m["right"]
            d = l["dim"]
            matrix(x + "left.q", l["heads"] * d, w)
            matrix(x + "left.k", l["kv_heads"] * d, w)
            matrix(x + "left.v", l["kv_heads"] * d, w)
            matrix(x + "left.o", w, l["heads"] * d)
            norm(x + "left.q.norm", l["heads"] * d)
            norm(x + "left.k.norm", l["kv_heads"] * d)
            for n, rows in (("q", r["kv_heads"] * d), ("k", r["kv_heads"] * d), ("v", r["heads"] * d)):
                matrix(x + "right." + n, rows, w)
                out.append((x + "right." + n + ".conv", (rows, r["conv"]), ("normal", 0.3)))
            matrix(x + "right.b", r["heads"], w)
            matrix(x + "right.a", r["heads"], w)
            matrix(x + "right.g", r["heads"] * d, w)
            matrix(x + "right.o", w, r["heads"] * d)
            uniform(x + "right.A_log", (r["heads"],), -2.0, 0.5)
            uniform(x + "right.dt_bias", (r["heads"],), -3.0, 0.5)
            norm(x + "right.norm", d)
        else:  # mamba1
            inner, n, rank = m["inner"], m["state"], m["dt_rank"]
            matrix(x + "in", 2 * inner, w)
            out.append((x + "conv", (inner, m["conv"]), ("normal", 0.3)))
            out.append((x + "conv.b", (inner,), ("normal", 0.1)))
            matrix(x + "x", rank + 2 * n, inner)
            matrix(x + "dt", inner, rank)
            uniform(x + "dt.b", (inner,), -4.0, 0.0)
            uniform(x + "A_log", (inner, n), -1.0, 1.5)
            norm(x + "D", inner)
            matrix(x + "o", w, inner)
        matrix(p + "mlp.gate", layer["mlp"]["ff"], w)
        matrix(p + "mlp.up", layer["mlp"]["ff"], w)
        matrix(p + "mlp.down", w, layer["mlp"]["ff"])
    norm("final.norm", w)
    if zeladra:
        out.append(("final.norm.b", (w,), ("normal", 0.02)))
        matrix("head", VOCAB, w)
    return out


def _weights(case, seed):
    """The checkpoint: matrices in the model's type, vectors of norms, gates and decays in the same."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = torch.float32 if case["dtype"] == "f32" else torch.bfloat16
    out = {}
    for name, shape, law in _tensors(case):
        if law[0] == "normal":
            out[name] = torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, law[1], generator=gen)
        elif law[0] == "uniform":
            out[name] = torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(law[1], law[2], generator=gen).to(dtype)
        else:
            out[name] = (1.0 + torch.empty(shape, dtype=torch.float32, device="cuda").normal_(0.0, 0.1, generator=gen)).to(dtype)
    return out


# -- what a case's requests are --------------------------------------------------------------------


def _requests(case):
    """Per request: (tokens in the cache before the pass, tokens the pass brings)."""
    mode = case["mode"]
    if mode == "decode":
        n, ctx = case["batch"], case["context"]
        # one or eight requests of equal length stand for a benchmark's batch, the others are of all lengths
        if n in (1, 2, 8):
            return [(ctx, 1)] * n
        return [(max(1, round(ctx * (0.2 + 0.8 * ((i * 0.6180339887) % 1.0)))), 1) for i in range(n)]
    if mode in ("prompt", "score"):
        return [(0, case["tokens"])]
    if mode == "portion":
        return [(case["context"], case["tokens"])]
    if mode == "turn":
        return [(0, max(2, case["tokens"] - 7 * i)) for i in range(case["batch"])]
    first = max(2, case["tokens"] * 5 // 8)
    second = max(2, case["tokens"] - first)
    ctx = case["context"]
    singles = [(max(1, round(ctx * (0.2 + 0.8 * ((i * 0.6180339887) % 1.0)))), 1) for i in range(case["batch"])]
    return [(0, first), (ctx // 2, second)] + singles


def _texts(case, seed):
    """Every request's whole text: cached tokens, the pass's, and for ``turn`` the tokens that follow."""
    gen = torch.Generator().manual_seed(seed + 1)
    more = case.get("new", 0)
    return [torch.randint(0, VOCAB, (cached + new + more,), generator=gen).tolist() for cached, new in _requests(case)]


def prepare(case, seed):
    from fastgen_b200.config import model_args_from_config
    from fastgen_b200.csrc.ops import Ops
    from fastgen_b200.engine import Engine, Model, StepEntry

    device = torch.device("cuda:0")
    torch.cuda.set_device(device)
    model = Model(model_args_from_config(_config(case)), Ops(torch.float32 if case["dtype"] == "f32" else torch.bfloat16, device))
    model.bind(_weights(case, seed))
    requests, texts = _requests(case), _texts(case, seed)
    longest = max(len(t) for t in texts)
    batch = len(requests)
    engine = Engine(model, page_size=PAGE, n_pages=sum(-(-len(t) // PAGE) + 1 for t in texts), max_requests=batch,
                    max_length=longest + PAGE, num_cuda_graphs=2, max_step_tokens=2048)
    state = dict(engine=engine, case=case)
    if case["mode"] in ("prompt", "score"):
        n = case["tokens"]
        want = list(range(n)) if case["mode"] == "score" else [n - 1]
        state["entries"] = [StepEntry("p", texts[0], want)]
        return state
    if case["mode"] == "turn":
        state["first"] = [StepEntry(i, t[:n], [n - 1]) for i, (t, (_, n)) in enumerate(zip(texts, requests))]
        state["then"] = [[StepEntry(i, [t[n + s]], [0]) for i, (t, (_, n)) in enumerate(zip(texts, requests))]
                         for s in range(case["new"])]
        return state
    # the cached tokens go through the model in portions, then room is taken for the pass's tokens
    for i, (t, (cached, _)) in enumerate(zip(texts, requests)):
        engine.admit(i)
        for s in range(0, cached, 2048):
            engine.step([StepEntry(i, t[s : min(s + 2048, cached)], [])])
    for i, (cached, new) in enumerate(requests):
        engine.cache.reserve(engine.cache.get(i), cached + new)
    state["entries"] = [StepEntry(i, t[c : c + n], [n - 1]) for i, (t, (c, n)) in enumerate(zip(texts, requests))]
    return state


def run(state):
    engine, mode = state["engine"], state["case"]["mode"]
    if mode in ("prompt", "score"):
        engine.admit("p")
        logits = engine.step(state["entries"])
        engine.release("p")
        return logits
    if mode == "turn":
        for e in state["first"]:
            engine.admit(e.request_id)
        out = [engine.step(state["first"]).clone()]
        for entries in state["then"]:
            out.append(engine.step(entries).clone())
        for e in state["first"]:
            engine.release(e.request_id)
        return torch.stack(out)
    # the step of a caller that keeps the lengths itself: the same tokens of the same requests each time
    return engine.step_reserved(state["entries"])


# -- what a pass cannot do without -------------------------------------------------------------------


def work(case):
    """Every weight a step uses once a step, the cached entries a step's queries see, the logits; two
    operations a multiplication of the products, the scores and the recurrences."""
    requests = _requests(case)
    elt = 4 if case["dtype"] == "f32" else 2
    config = _config(case)
    sizes = {name: math.prod(shape) for name, shape, _ in _tensors(case)}
    head = sizes.get("lm_head.weight", sizes.get("head", sizes["embed"] if "embed" in sizes else 0))
    tables = [n for n in ("model.embed_tokens.weight", "embed", "lm_head.weight", "head") if n in sizes]
    inner = sum(v for n, v in sizes.items() if n not in tables)
    width = config["hidden_size"] if case["model"] in LLAMA else config["width"]
    steps = [requests]
    if case["mode"] == "turn":
        steps += [[(c + n + s, 1) for c, n in requests] for s in range(case["new"])]
    total_bytes = total_flops = 0.0
    for step in steps:
        tokens = sum(n for _, n in step)
        wanted = case["tokens"] if case["mode"] == "score" else len(step)
        total_bytes += elt * (inner + head + tokens * width) + 4.0 * wanted * VOCAB
        total_flops += 2.0 * inner * tokens + 2.0 * head * wanted
        for i in range(case["layers"]):
            b, f = _mixer_work(case, config, i, step, elt)
            total_bytes += b
            total_flops += f
    return {"bytes": total_bytes, "flops": total_flops}


def _pairs(cached, new, window=None):
    """Query-key pairs of ``new`` tokens behind ``cached`` ones."""
    whole = new * cached + new * (new + 1) / 2
    return whole if window is None else min(whole, new * float(window))


def _mixer_work(case, config, i, step, elt):
    if case["model"] in LLAMA:
        _, heads, kv, d, _, _ = LLAMA[case["model"]]
        return (sum(2.0 * kv * d * elt * (c + n) for c, n in step), sum(4.0 * heads * d * _pairs(c, n) for c, n in step))
    layer = config["layers"][i]
    m, kind = layer["mixer"], layer["type"]
    if kind == "latent_attention":
        entry = m["kv_rank"] + m["rot_dim"]
        return (sum(float(entry) * elt * (c + n) for c, n in step),
                sum(2.0 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]) * _pairs(c, n) for c, n in step))
    if kind == "attention":
        window = m["mask"]["size"] + m["mask"]["keep_first"]
        return (sum(2.0 * m["kv_heads"] * m["dim"] * elt * min(c + n, window + n) for c, n in step),
                sum(4.0 * m["heads"] * m["dim"] * _pairs(c, n, window) for c, n in step))
    if kind == "mamba2":
        numbers = m["heads"] * m["state"] * m["vdim"]
        return 8.0 * numbers * len(step), sum(6.0 * numbers * n for _, n in step)
    if kind == "mamba1":
        numbers = m["inner"] * m["state"]
        return 8.0 * numbers * len(step), sum(6.0 * numbers * n for _, n in step)
    l, r = m["left"], m["right"]
    numbers = r["heads"] * r["dim"] * r["vdim"]
    return (sum(2.0 * l["kv_heads"] * l["dim"] * elt * min(c + n, l["mask"]["size"] + n) for c, n in step) + 8.0 * numbers * len(step),
            sum(4.0 * l["heads"] * l["dim"] * _pairs(c, n, l["mask"]["size"]) + 8.0 * numbers * n for c, n in step))


def tolerance(case):
    """About four times what the logits are off against 64 bits: float32 1.5e-6; bfloat16 0.003 to 0.007 on the
    Llama shapes, up to 0.012 where decays and norms over small vectors feed on rounded values."""
    if case["dtype"] == "f32":
        return {"rel": 7e-6}
    return {"rel": 0.02 if case["model"] in LLAMA else 0.03}


# -- the same in 64 bits -----------------------------------------------------------------------------

D = torch.float64


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _centred(x, eps):
    c = x - x.mean(-1, keepdim=True)
    return c / torch.sqrt((c * c).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.logaddexp(x, torch.zeros_like(x))


def _llama_freqs(config):
    d, s = config["head_dim"], config["rope_scaling"]
    f = config["rope_theta"] ** (-torch.arange(0, d, 2, dtype=D, device="cuda") / d)
    wave = 2 * math.pi / f
    low, high, old = s["low_freq_factor"], s["high_freq_factor"], s["original_max_position_embeddings"]
    smooth = ((old / wave - low) / (high - low)).clamp(0, 1)  # 0: slow pairs, divided; 1: fast pairs, kept
    return (1 - smooth) * f / s["factor"] + smooth * f


def _yarn(rot):
    dims, base, s = rot["dims"], float(rot["base"]), rot.get("scaling")
    i = torch.arange(dims // 2, dtype=D, device="cuda")
    f = base ** (-2.0 * i / dims)
    if not s:
        return f, 1.0

    def at(turns):
        return dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))

    lo, hi = max(math.floor(at(s["fast"])), 0), min(math.ceil(at(s["slow"])), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / s["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def _turn(x, freqs, magnitude=1.0, halves=True):
    """``x`` [T, heads, 2P]: the pairs (i, i + P), or (2i, 2i + 1), of position p turn by p freqs[i]."""
    ang = torch.arange(x.shape[0], dtype=D, device=x.device)[:, None, None] * freqs
    c, s = torch.cos(ang) * magnitude, torch.sin(ang) * magnitude
    if halves:
        a, b = x.chunk(2, dim=-1)
        return torch.cat([a * c - b * s, b * c + a * s], dim=-1)
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, b * c + a * s], dim=-1).reshape(x.shape)


def _attend(q, k, v, scale, seen=None, sink=False):
    """``q`` [T, H, d], ``k`` [T, G, d], ``v`` [T, G, e] -> [T, H * e]; ``seen(i, j)`` narrows what is causal;
    ``sink``: one more summand, 1, in the sum of weights."""
    t, heads, _ = q.shape
    rep = heads // k.shape[1]
    j = torch.arange(t, device=q.device)[None, :]
    out = torch.empty(t, heads, v.shape[2], dtype=D, device=q.device)
    step = max(16, min(t, (1 << 28) // (t * heads)))
    kk, vv = k.permute(1, 2, 0), v.permute(1, 0, 2)  # [G, d, T], [G, T, e]
    for s in range(0, t, step):
        e = min(t, s + step)
        i = torch.arange(s, e, device=q.device)[:, None]
        qq = q[s:e].permute(1, 0, 2).reshape(k.shape[1], rep * (e - s), -1)
        z = torch.bmm(qq, kk[:, :, :e]).mul_(scale).reshape(heads, e - s, e)
        ok = j[:, :e] <= i
        if seen is not None:
            ok = ok & seen(i, j[:, :e])
        z.masked_fill_(~ok, -math.inf)
        top = z.max(-1, keepdim=True).values
        if sink:
            top = top.clamp(min=0.0)
        z.sub_(top).exp_()
        total = z.sum(-1, keepdim=True)
        if sink:
            total = total + torch.exp(-top)
        z.div_(total)
        o = torch.bmm(z.reshape(k.shape[1], rep * (e - s), e), vv[:, :e])
        out[s:e] = o.reshape(heads, e - s, -1).permute(1, 0, 2)
    return out.reshape(t, -1)


def _conv(x, taps, bias=None):
    t, n = x.shape[0], taps.shape[1]
    padded = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
    y = sum(padded[j : j + t] * taps[:, j] for j in range(n))
    return y if bias is None else y + bias


def _latent(h, w, m, eps, entries):
    t = h.shape[0]
    heads, d, r, e, rank = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    f, mag = _yarn(m["rot"])
    if entries is None:
        low = h @ w["dkv"].T
        entries = (_rms(low[:, :rank], eps) * w["dkv.norm"], _turn(low[:, None, rank:], f, mag, halves=False))
    c, turned = entries
    q = ((_rms(h @ w["dq"].T, eps) * w["dq.norm"]) @ w["uq"].T).reshape(t, heads, d + r)
    q = torch.cat([q[..., :d], _turn(q[..., d:], f, mag, halves=False)], dim=-1)
    k = torch.cat([(c @ w["uk"].T).reshape(t, heads, d), turned.expand(t, heads, r)], dim=-1)
    v = (c @ w["uv"].T).reshape(t, heads, e)
    o = _attend(q, k, v, m["scale"]).reshape(t, heads, e) * torch.sigmoid(h @ w["g"].T)[:, :, None]
    return o.reshape(t, -1) @ w["o"].T, entries


def _windowed(h, w, m):
    t, d = h.shape[0], m["dim"]
    f, mag = _yarn(m["rot"])
    q = _turn((h @ w["q"].T).reshape(t, -1, d), f, mag, halves=False)
    k = _turn((h @ w["k"].T).reshape(t, -1, d), f, mag, halves=False)
    size, keep = m["mask"]["size"], m["mask"]["keep_first"]
    o = _attend(q, k, (h @ w["v"].T).reshape(t, -1, d), m["scale"], lambda i, j: (i - j < size) | (j < keep))
    return o @ w["o"].T


def _mamba2(h, w, m, eps):
    t = h.shape[0]
    heads, p, n, groups = m["heads"], m["vdim"], m["state"], m["groups"]
    inner = heads * p
    proj = h @ w["in"].T
    z, xbc, dt = proj[:, :inner], proj[:, inner : 2 * inner + 2 * groups * n], proj[:, 2 * inner + 2 * groups * n :]
    xbc = _silu(_conv(xbc, w["conv"], w["conv.b"]))
    x = xbc[:, :inner].reshape(t, heads, p)
    b = xbc[:, inner : inner + groups * n].reshape(t, groups, n).repeat_interleave(heads // groups, dim=1)
    c = xbc[:, inner + groups * n :].reshape(t, groups, n).repeat_interleave(heads // groups, dim=1)
    dt = _softplus(dt + w["dt_bias"])
    decay = torch.exp(-torch.exp(w["A_log"]) * dt)
    xd = x * dt[:, :, None]
    state = x.new_zeros(heads, n, p)
    y = torch.empty_like(x)
    for s in range(t):
        state = torch.baddbmm(state * decay[s][:, None, None], b[s][:, :, None], xd[s][:, None, :])
        y[s] = torch.bmm(c[s][:, None, :], state)[:, 0]
    y = (y + w["D"][:, None] * x).reshape(t, inner) * _silu(z)
    parts = m["norm_groups"]
    return (_rms(y.reshape(t, parts, -1), eps).reshape(t, inner) * w["norm"]) @ w["o"].T


def _chunked(h, w, m, eps):
    t, d, size = h.shape[0], m["dim"], m["mask"]["size"]
    f, mag = _yarn(m["rot"])
    q = _turn((_rms(h @ w["q"].T, eps) * w["q.norm"]).reshape(t, -1, d), f, mag)
    k = _turn((_rms(h @ w["k"].T, eps) * w["k.norm"]).reshape(t, -1, d), f, mag)
    return _attend(q, k, (h @ w["v"].T).reshape(t, -1, d), m["scale"], lambda i, j: i // size == j // size, sink=True) @ w["o"].T


def _delta(h, w, m, eps):
    t, heads, d = h.shape[0], m["heads"], m["dim"]
    rep = heads // m["kv_heads"]
    q, k, v = (_silu(_conv(h @ w[n].T, w[n + ".conv"])).reshape(t, -1, d) for n in "qkv")
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    q, k = q.repeat_interleave(rep, dim=1), k.repeat_interleave(rep, dim=1)
    beta = torch.sigmoid(h @ w["b"].T)
    g = torch.exp(-torch.exp(w["A_log"]) * _softplus(h @ w["a"].T + w["dt_bias"]))
    state = h.new_zeros(heads, d, d)
    out = torch.empty_like(v)
    for s in range(t):
        state = state * g[s][:, None, None]
        u = beta[s][:, None] * (v[s] - torch.bmm(k[s][:, None, :], state)[:, 0])
        state = torch.baddbmm(state, k[s][:, :, None], u[:, None, :])
        out[s] = torch.bmm(q[s][:, None, :], state)[:, 0]
    out = _rms(out, eps) * w["norm"] * _silu(h @ w["g"].T).reshape(t, heads, d)
    return out.reshape(t, -1) @ w["o"].T


def _mamba1(h, w, m):
    t, inner, n, rank = h.shape[0], m["inner"], m["state"], m["dt_rank"]
    proj = h @ w["in"].T
    x = _silu(_conv(proj[:, :inner], w["conv"], w["conv.b"]))
    low = x @ w["x"].T
    dt = _softplus(low[:, :rank] @ w["dt"].T + w["dt.b"])
    b, c = low[:, rank : rank + n], low[:, rank + n :]
    a = -torch.exp(w["A_log"])
    state = h.new_zeros(inner, n)
    y = torch.empty_like(x)
    for s in range(t):
        state = torch.exp(dt[s][:, None] * a) * state + (dt[s] * x[s])[:, None] * b[s]
        y[s] = state @ c[s]
    return ((y + w["D"] * x) * _silu(proj[:, inner:])) @ w["o"].T


def _llama_layer(x, w, config, freqs):
    t, d, eps = x.shape[0], config["head_dim"], config["rms_norm_eps"]
    h = _rms(x, eps) * w["input_layernorm.weight"]
    q = _turn((h @ w["self_attn.q_proj.weight"].T).reshape(t, -1, d), freqs)
    k = _turn((h @ w["self_attn.k_proj.weight"].T).reshape(t, -1, d), freqs)
    v = (h @ w["self_attn.v_proj.weight"].T).reshape(t, -1, d)
    x = x + _attend(q, k, v, d ** -0.5) @ w["self_attn.o_proj.weight"].T
    h = _rms(x, eps) * w["post_attention_layernorm.weight"]
    return x + (_silu(h @ w["mlp.gate_proj.weight"].T) * (h @ w["mlp.up_proj.weight"].T)) @ w["mlp.down_proj.weight"].T


def _mlp(h, w, act):
    return (act(h @ w["mlp.gate"].T) * (h @ w["mlp.up"].T)) @ w["mlp.down"].T


def _of(weights, prefix):
    return {n[len(prefix):]: v for n, v in weights.items() if n.startswith(prefix)}


def exact(case, seed):
    weights = _weights(case, seed)
    texts, requests, config = _texts(case, seed), _requests(case), _config(case)
    table = weights["model.embed_tokens.weight" if case["model"] in LLAMA else "embed"]
    xs = [table[torch.tensor(t, device="cuda")].to(D) for t in texts]
    latents = {}
    if case["model"] == "zeladra":
        xs = [torch.stack([x, x]) for x in xs]  # two residual streams
    freqs = _llama_freqs(config) if case["model"] in LLAMA else None
    for i in range(case["layers"]):
        w = {n: v.to(D) for n, v in _of(weights, (f"model.layers.{i}." if case["model"] in LLAMA else f"l{i}.")).items()}
        for r, x in enumerate(xs):
            if case["model"] in LLAMA:
                xs[r] = _llama_layer(x, w, config, freqs)
                continue
            layer, eps, mix = config["layers"][i], config["norm"]["eps"], _of(w, "mix.")
            m = layer["mixer"]
            if case["model"] == "zeladra":
                for q in "12":
                    a, b, c = w[f"hc{q}.in"], w[f"hc{q}.out"], w[f"hc{q}.mix"]
                    h = _centred(a[0] * x[0] + a[1] * x[1], eps) * w[f"norm{q}"] + w[f"norm{q}.b"]
                    if q == "2":
                        y = _mlp(h, w, _silu)
                    elif layer["type"] == "latent_attention":
                        y, latents[r] = _latent(h, mix, m, eps, latents[r] if "kv_from" in m else None)
                    elif layer["type"] == "mamba2":
                        y = _mamba2(h, mix, m, eps)
                    else:
                        y = _windowed(h, mix, m)
                    x = torch.stack([c[0, s] * x[0] + c[1, s] * x[1] + b[s] * y for s in range(2)])
                xs[r] = x
                continue
            h = _centred(x, eps) * w["norm1"]
            if layer["type"] == "parallel":
                y = (m["left_scale"] * _chunked(h, _of(mix, "left."), m["left"], eps)
                     + m["right_scale"] * _delta(h, _of(mix, "right."), m["right"], eps))
            else:
                y = _mamba1(h, mix, m)
            x = x + _centred(y, eps) * w["norm1b"] * w["ls1"]
            y = _mlp(_centred(x, eps) * w["norm2"], w, torch.relu)
            xs[r] = x + _centred(y, eps) * w["norm2b"] * w["ls2"]
    # the rows whose logits a pass returns
    rows = []
    for x, (cached, new) in zip(xs, requests):
        x = x[0] + x[1] if case["model"] == "zeladra" else x
        if case["mode"] == "score":
            rows.append(x)
        elif case["mode"] == "turn":
            rows.append(x[new - 1 : new + case["new"]])
        else:
            rows.append(x[cached + new - 1][None])
    x = torch.stack(rows, dim=1) if case["mode"] == "turn" else torch.cat(rows)
    if case["model"] in LLAMA:
        x, head = _rms(x, config["rms_norm_eps"]) * weights["model.norm.weight"].to(D), weights["lm_head.weight"]
    elif case["model"] == "zeladra":
        x, head = _centred(x, 1e-5) * weights["final.norm"].to(D) + weights["final.norm.b"].to(D), weights["head"]
    else:
        x, head = _centred(x, 1e-5) * weights["final.norm"].to(D), table
    return x @ head.to(D).T
