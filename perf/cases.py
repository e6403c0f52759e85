"""The work whose speed matters: steps of real models through the library's public entry points.

A case is a model (sizes as in the library's configurations and benchmark, layers of each kind it
has), a kind of call and the sequences of that call:

    prompt     ``Engine.step`` of prompts that start together: the logits of each one's last token
    decode     ``Engine.decode_step``: one given token for every sequence, a sampled one each; the
               logits that were sampled from
    generate   ``GenerationEngine.generate``: greedy tokens of a batch of prompts, and the logits of
               the last of them

Weights are random, drawn at the spread at which activations keep a trained model's sizes; token ids are
uniform.  ``shortest`` and ``longest`` bound the sequences' lengths (in tokens, before the call; spaced
evenly over their logarithm).
"""

import gc
import math

import torch

from strata_inference_b200 import Engine, GenerationConfig, GenerationEngine, spec_from_config

# width, feed-forward, heads, key/value heads, head width, vocabulary
SIZES = {
    "tiny": (64, 128, 4, 2, 16, 256),
    "1b": (2048, 8192, 16, 8, 128, 32000),
    "2b": (2304, 9216, 8, 4, 256, 256000),
    "9b": (3584, 14336, 16, 8, 256, 256000),
}
GROWTH = 1024       # tokens a decoded sequence may grow by before another takes its place
WARM_STEPS = 3      # decode steps before the first timed one: a server records its steps at start-up


def case(name, model, size, layers, dtype, call, sequences, shortest, longest, new=1, temperature=0.0,
         top_k=0, top_p=1.0):
    made = {"model": model, "size": size, "layers": layers, "dtype": dtype, "call": call,
            "sequences": sequences, "shortest": shortest, "longest": longest, "new": new,
            "temperature": temperature, "top_k": top_k, "top_p": top_p}
    return dict(made, name=name) if name else made


def listed():
    return [
        # the smallest request there is: a toy model in 32-bit, as a test suite or a tutorial runs it
        case("tiny_generate_f32", "gemma2", "tiny", 2, "float32", "generate", 3, 5, 13, new=8),
        # one user at the end of a long conversation
        case("gemma2_2b_decode_1", "gemma2", "2b", 26, "bfloat16", "decode", 1, 7001, 7001),
        # a small server's batch with long contexts: the benchmark's headline
        case("gemma2_2b_decode_8", "gemma2", "2b", 26, "bfloat16", "decode", 8, 5300, 7001),
        # a full server's batch, sampled as chat front ends sample
        case("gemma2_2b_decode_64", "gemma2", "2b", 26, "bfloat16", "decode", 64, 150, 3001,
             temperature=0.8, top_k=40, top_p=0.95),
        # three short questions: latency until the first token
        case("gemma2_2b_prompt_short", "gemma2", "2b", 26, "bfloat16", "prompt", 3, 19, 83),
        # the benchmark's prompt
        case("gemma2_2b_prompt_2048", "gemma2", "2b", 26, "bfloat16", "prompt", 1, 2048, 2048),
        # an unequal batch of documents on a larger model
        case("gemma2_9b_prompt_8", "gemma2", "9b", 12, "bfloat16", "prompt", 8, 128, 4096),
        # the 32-bit check of a model's logits
        case("gemma2_2b_prompt_f32", "gemma2", "2b", 6, "float32", "prompt", 2, 301, 700),
        # recurrent layers in turn with attention: a prompt, a batch of decoded tokens
        case("karupel_2b_prompt_2048", "karupel", "2b", 4, "bfloat16", "prompt", 1, 2048, 2048),
        case("karupel_1b_decode_32", "karupel", "1b", 8, "bfloat16", "decode", 32, 200, 2500),
        # routed experts: a batch of prompts, a small batch of decoded tokens
        case("kerolorn_1b_prompt_4", "kerolorn", "1b", 4, "bfloat16", "prompt", 4, 250, 1777),
        case("kerolorn_1b_decode_8", "kerolorn", "1b", 4, "bfloat16", "decode", 8, 300, 3001),
    ]


def draw(rng):
    """One more case of the same ranges: every model and call, sizes over their logarithm."""
    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model = rng.choice(["gemma2", "gemma2", "gemma2", "karupel", "kerolorn"])
    size = rng.choice(["1b", "2b", "2b", "9b"] if model == "gemma2" else ["1b", "2b"])
    call = rng.choice(["prompt", "decode"])
    layers = rng.choice([4, 6, 8])
    dtype = "float32" if model == "gemma2" and size != "9b" and rng.random() < 0.2 else "bfloat16"
    n = between(1, 64)
    if call == "prompt":
        n = min(n, 16)
        longest = between(3, min(4096, (1500 if dtype == "float32" else 12000) // n))
        return case("", model, size, layers, dtype, call, n, between(max(1, longest // 20), longest), longest)
    longest = between(60, min(7000, (4000 if dtype == "float32" else 100000) // n))
    sampled = rng.choice([(0.0, 0, 1.0), (0.0, 0, 1.0), (1.0, 0, 1.0), (0.8, 40, 0.95), (0.7, 0, 0.9)])
    return case("", model, size, layers, dtype, call, n, between(max(10, longest // 20), longest), longest, 1,
                *sampled)


# ---- models ---------------------------------------------------------------------------------------------

def config_of(c):
    """The config.json of a case's model."""
    width, ff, heads, kv, hd, vocab = SIZES[c["size"]]
    if c["model"] == "gemma2":
        tiny = c["size"] == "tiny"
        return {"architectures": ["Gemma2ForCausalLM"], "model_type": "gemma2", "num_hidden_layers": c["layers"],
                "hidden_size": width, "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": hd,
                "intermediate_size": ff, "vocab_size": vocab, "rope_theta": 10000.0,
                "sliding_window": 8 if tiny else 4096, "query_pre_attn_scalar": hd,
                "attn_logit_softcapping": 50.0, "final_logit_softcapping": 30.0, "rms_norm_eps": 1e-6,
                "max_position_embeddings": 128 if tiny else 8192, "hidden_activation": "gelu_pytorch_tanh",
                "tie_word_embeddings": True}
    if c["model"] == "karupel":
        mlp = {"kind": "dense", "ff": ff}
        attention = {"type": "attention", "mlp": mlp, "mixer": {
            "heads": heads, "kv_heads": kv, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "v_mix": True,
            "rot": {"base": 10000.0, "dims": hd // 2, "scaling": {"factor": 2.0}}}}
        delta = {"type": "delta", "mlp": mlp,
                 "mixer": {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": hd, "conv": 4}}
        memory = {"type": "mlstm", "mlp": mlp, "mixer": {"heads": heads, "dim": 128, "vdim": hd, "gate_cap": 15.0}}
        pattern = [delta, attention, memory, attention]
        return {"architecture": "Karupel", "vocab": vocab, "width": width, "norm": {"eps": 1e-6},
                "layers": [pattern[i % 4] for i in range(c["layers"])]}
    layer = {"type": "attention",
             "mixer": {"heads": heads, "kv_heads": kv, "dim": hd, "vdim": hd, "scale": hd ** -0.5,
                       "mask": {"size": 1024, "keep_first": 64},
                       "rot": {"base": 1000000.0, "dims": hd,
                               "scaling": {"factor": 16.0, "original": 4096, "fast": 32.0, "slow": 1.0}}},
             "mlp": {"kind": "moe", "router": {"experts": 32, "top": 4, "scale": 2.0}, "expert": {"ff": ff // 8},
                     "shared": {"ff": ff // 2}}}
    return {"architecture": "Kerolorn", "vocab": vocab, "width": width, "norm": {"eps": 1e-6}, "canon": {"taps": 4},
            "logit_scale": 0.5, "layers": [layer] * c["layers"]}


def tensors_of(c):
    """(name, shape, spread, mean) of every stored tensor."""
    cfg = config_of(c)
    W, ff, heads, kv, hd, V = SIZES[c["size"]]
    out = []

    def matrix(name, rows, cols, spread=None):
        out.append((name, (rows, cols), W ** -0.5 if spread is None else spread, 0.0))

    def vector(name, n, spread, mean=0.0):
        out.append((name, (n,) if n else (), spread, mean))

    if c["model"] == "gemma2":
        std = 0.08 if c["size"] == "tiny" else 0.02
        matrix("model.embed_tokens.weight", V, W, std)
        for i in range(c["layers"]):
            p = f"model.layers.{i}."
            for site in ("input", "post_attention", "pre_feedforward", "post_feedforward"):
                vector(p + site + "_layernorm.weight", W, 0.1)
            for n, rows, cols in (("self_attn.q_proj", heads * hd, W), ("self_attn.k_proj", kv * hd, W),
                                  ("self_attn.v_proj", kv * hd, W), ("self_attn.o_proj", W, heads * hd),
                                  ("mlp.gate_proj", ff, W), ("mlp.up_proj", ff, W), ("mlp.down_proj", W, ff)):
                matrix(p + n + ".weight", rows, cols, std)
        vector("model.norm.weight", W, 0.1)
        return out
    matrix("embed", V, W, 1.0)
    for i, layer in enumerate(cfg["layers"]):
        m, p, q = layer["mixer"], f"l{i}.mix.", f"l{i}.mlp."
        H, D, U = m["heads"], m["dim"], m["vdim"]
        G = m.get("kv_heads", H)
        vector(f"l{i}.norm1", W, 0.1, 0.0 if c["model"] == "karupel" else 1.0)
        vector(f"l{i}.norm2", W, 0.1, 0.0 if c["model"] == "karupel" else 1.0)
        matrix(p + "q", H * D if layer["type"] != "delta" else G * D, W)
        matrix(p + "k", G * D, W)
        matrix(p + "v", (H if layer["type"] == "delta" else G) * U, W)
        matrix(p + "o", W, H * U, (H * U) ** -0.5)
        if c["model"] == "kerolorn":
            vector(f"l{i}.norm1b", W, 0.1, 1.0)
            vector(f"l{i}.norm2b", W, 0.1, 1.0)
            matrix(f"l{i}.canon1", W, cfg["canon"]["taps"], 0.3)
            vector(p + "temp", H, 0.1, 1.0)
            mlp = layer["mlp"]
            E, F, S = mlp["router"]["experts"], mlp["expert"]["ff"], mlp["shared"]["ff"]
            matrix(q + "router", E, W, 3.0 * W ** -0.5)     # (a trained router's scores are far apart)
            vector(q + "correction", E, 0.01)
            for e in range(E):
                matrix(q + f"e{e}.gate", F, W)
                matrix(q + f"e{e}.up", F, W)
                matrix(q + f"e{e}.down", W, F, F ** -0.5)
            matrix(q + "shared.gate", S, W)
            matrix(q + "shared.up", S, W)
            matrix(q + "shared.down", W, S, S ** -0.5)
            matrix(q + "shared.sg", 1, W)
            continue
        if layer["type"] == "delta":
            for n, rows in (("q", G * D), ("k", G * D), ("v", H * U)):
                matrix(p + n + ".conv", rows, m["conv"], 0.6)
            matrix(p + "b", H, W)
            matrix(p + "a", H, W)
            vector(p + "A_log", H, 0.5, -1.0)
            vector(p + "dt_bias", H, 0.5)
            vector(p + "norm", U, 0.1, 1.0)
            matrix(p + "g", H * U, W)
        elif layer["type"] == "attention":
            for n, rows in (("q", H * D), ("k", G * D), ("v", G * U)):
                vector(p + n + ".b", rows, 0.2)
            vector(p + "q.norm", D, 0.1, 1.0)
            vector(p + "k.norm", D, 0.1, 1.0)
            vector(p + "vmix", 0, 0.1, 0.5)
            matrix(p + "g", H, W)
        else:
            matrix(p + "i", H, W)
            matrix(p + "f", H, W)
            vector(p + "i.b", H, 0.5)
            vector(p + "f.b", H, 0.5, 2.0)
            vector(p + "norm", H * U, 0.1, 1.0)
            matrix(p + "g", H * U, W)
        matrix(q + "gate", ff, W)
        matrix(q + "up", ff, W)
        matrix(q + "down", W, ff, ff ** -0.5)
    vector("final.norm", W, 0.1, 0.0 if c["model"] == "karupel" else 1.0)
    if c["model"] == "kerolorn":
        matrix("head", V, W)
    return out


def weights_of(c, seed):
    """The stored tensors by name, drawn on the device."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype = getattr(torch, c["dtype"])
    out = {}
    for name, shape, spread, mean in tensors_of(c):
        t = torch.randn(shape, generator=g, device="cuda", dtype=dtype).mul_(spread)
        out[name] = t.add_(mean) if mean else t
    return out


def lengths_of(c):
    n, lo, hi = c["sequences"], c["shortest"], c["longest"]
    return [hi if n == 1 else int(round(lo * (hi / lo) ** (i / (n - 1)))) for i in range(n)]


def tokens_of(c, seed):
    """Token ids of every sequence: its own and the ones that are fed to it afterwards."""
    g = torch.Generator().manual_seed(seed)
    vocab = SIZES[c["size"]][5]
    return [torch.randint(0, vocab, (n + GROWTH,), generator=g).tolist() for n in lengths_of(c)]


# ---- a pass ---------------------------------------------------------------------------------------------

def begin(state):
    """Fresh sequences that hold their contexts (all but the steps that warm the engine up)."""
    engine, lengths = state["engine"], state["lengths"]
    state["slots"] = [engine.new_sequence() for _ in lengths]
    for at in range(0, len(lengths), 8):
        engine.step([(s, ids[:n - WARM_STEPS]) for s, ids, n in
                     list(zip(state["slots"], state["ids"], lengths))[at:at + 8]])
    state["fed"] = -WARM_STEPS


def prepare(c, seed):
    gc.collect()        # (an engine and its recorded steps refer to each other)
    lengths, ids = lengths_of(c), tokens_of(c, seed)
    most = c["longest"] + (GROWTH if c["call"] == "decode" else c["new"])
    spec = spec_from_config(config_of(c))[1]
    grow = GROWTH if c["call"] == "decode" else c["new"]
    engine = Engine(spec, weights_of(c, seed), dtype=c["dtype"], max_seq_len=most, max_slots=c["sequences"],
                    max_tokens=sum(-(-(n + grow) // 64) * 64 for n in lengths))
    state = {"engine": engine, "case": c, "lengths": lengths, "ids": ids}
    if c["call"] == "decode":
        begin(state)
        for _ in range(WARM_STEPS):
            run(state)
    else:
        state["prompts"] = [t[:n] for t, n in zip(ids, lengths)]
        if c["call"] == "generate":
            state["generation"] = GenerationEngine(engine)
        other = [list(reversed(p)) for p in state["prompts"]]
        for _ in range(WARM_STEPS):
            run(dict(state, prompts=other))
    return state


def run(state):
    engine, c = state["engine"], state["case"]
    if c["call"] == "generate":
        outs = state["generation"].generate(state["prompts"], GenerationConfig(max_tokens=c["new"]))
        return {"tokens": torch.tensor([o.token_ids for o in outs]), "logits": engine.last_logits}
    if c["call"] == "prompt":
        slots = [engine.new_sequence() for _ in state["prompts"]]
        logits = engine.step(list(zip(slots, state["prompts"])))
        for s in slots:
            engine.end_sequence(s)
        return {"logits": logits}
    if state["fed"] >= GROWTH - 1:       # these sequences have reached their ends: the next ones
        for s in state["slots"]:
            engine.end_sequence(s)
        begin(state)
    at = state["fed"]
    fed = [ids[n + at] for ids, n in zip(state["ids"], state["lengths"])]
    engine.decode_step(state["slots"], fed, c["temperature"], c["top_k"], c["top_p"])
    state["fed"] += 1
    return {"logits": engine.last_logits}


# ---- what a pass needs, and how far results may be apart ------------------------------------------------

def work(c):
    cfg = config_of(c)
    W, ff, heads, kv, hd, V = SIZES[c["size"]]
    esize = 4 if c["dtype"] == "float32" else 2
    lengths, n = lengths_of(c), c["sequences"]
    rows = sum(lengths) if c["call"] != "decode" else n
    steps = c["new"] - 1 if c["call"] == "generate" else 0
    read = used = 0                                  # elements of weights: that are read, that a row meets
    for name, shape, _, _ in tensors_of(c):
        size = math.prod(shape)
        if name in ("embed", "model.embed_tokens.weight"):
            continue
        if ".mlp.e" in name:                         # a routed expert
            r = cfg["layers"][0]["mlp"]["router"]
            used += size * r["top"] / r["experts"]
            read += size * min(1.0, rows * r["top"] / r["experts"])
        elif name != "head":
            used += size
            read += size
    head = V * W
    nbytes = esize * (read + head) + rows * W * esize + 4 * n * V
    flops = 2.0 * used * rows + 2.0 * head * n
    for i in range(c["layers"]):
        window, cell, state = 0, 0, 0
        if c["model"] == "gemma2":
            window = cfg["sliding_window"] if i % 2 == 0 else 0
            cell = 2 * kv * hd
        else:
            m = cfg["layers"][i]["mixer"]
            window = m["mask"]["size"] + m["mask"]["keep_first"] if m.get("mask") else 0
            if cfg["layers"][i]["type"] == "attention":
                cell = 2 * kv * hd
            else:
                state = m["heads"] * m["dim"] * m["vdim"]
        for length in lengths:
            if cell and c["call"] == "decode":
                seen = min(length + 1, window or length + 1)
                flops += 4.0 * seen * heads * hd
                nbytes += esize * cell * (seen + 1)
            elif cell:
                over = max(0, length - window) if window else 0
                flops += 4.0 * heads * hd * (length * (length + 1) / 2 - over * (over + 1) / 2)
                nbytes += esize * cell * length
            else:
                flops += 6.0 * state * (1 if c["call"] == "decode" else length)
                nbytes += 4 * state * (2 if c["call"] == "decode" else 1)
    return {"bytes": float(nbytes * (1 + steps)), "flops": float(flops + steps * (2.0 * used + 2.0 * head) * n)}


def tolerance(c):
    # Seen against 64 bits: 2.7e-6 to 4e-6 in 32-bit; in bfloat16, whose roundings any change of a sum's
    # order moves, 0.006 to 0.021 (the same pass twice: 0.006).
    if c["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-4}
    return {"rel": 0.03, "max": 0.3}


# ---- the same in 64 bits --------------------------------------------------------------------------------

def unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def silu(x):
    return x * torch.sigmoid(x)


def attend(q, k, v, scale, cap=0.0, window=0, keep=0):
    """q[T, H, d], k[T, G, d], v[T, G, u] -> [T, H * u]: causal, grouped, capped, windowed."""
    T, H = q.shape[:2]
    pos = torch.arange(T, device=q.device)
    out = q.new_empty(T, H, v.shape[2])
    for lo in range(0, T, 2048):
        hi = min(T, lo + 2048)
        far = pos[lo:hi, None] - pos[None, :hi]
        hidden = far < 0
        if window:
            hidden = hidden | ((far >= window) & (pos[None, :hi] >= keep))
        for h in range(H):
            g = h * k.shape[1] // H
            s = q[lo:hi, h] @ k[:hi, g].T * (scale[h] if torch.is_tensor(scale) else scale)
            if cap:
                s = cap * torch.tanh(s / cap)
            out[lo:hi, h] = torch.softmax(s.masked_fill_(hidden, -math.inf), -1) @ v[:hi, g]
    return out.reshape(T, -1)


def turn_halves(x, dims, freq):
    """Rotate the first ``dims`` entries of x[T, heads, d], entry i with entry i + dims / 2."""
    ang = torch.arange(x.shape[0], device=x.device, dtype=x.dtype)[:, None] * freq
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    a, b = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., dims:]], -1)


def gemma2_layer(xs, w, i, cfg):
    p, eps, hd = f"model.layers.{i}.", cfg["rms_norm_eps"], cfg["head_dim"]
    heads, kv = cfg["num_attention_heads"], cfg["num_key_value_heads"]
    half = torch.arange(hd // 2, dtype=torch.float32, device="cuda")
    freq = torch.pow(cfg["rope_theta"], -2.0 * half / hd).double()

    def norm(x, site):
        return unit(x, eps) * (1 + w(p + site + "_layernorm.weight"))

    def one(x):
        h = norm(x, "input")
        q, k, v = ((h @ w(p + f"self_attn.{n}_proj.weight").T).view(len(h), -1, hd) for n in "qkv")
        q, k = turn_halves(q, hd, freq), turn_halves(k, hd, freq)
        y = attend(q, k, v, cfg["query_pre_attn_scalar"] ** -0.5, cfg["attn_logit_softcapping"],
                   cfg["sliding_window"] if i % 2 == 0 else 0)
        x = x + norm(y @ w(p + "self_attn.o_proj.weight").T, "post_attention")
        h = norm(x, "pre_feedforward")
        gate = torch.nn.functional.gelu(h @ w(p + "mlp.gate_proj.weight").T, approximate="tanh")
        y = (gate * (h @ w(p + "mlp.up_proj.weight").T)) @ w(p + "mlp.down_proj.weight").T
        return x + norm(y, "post_feedforward")

    assert heads % kv == 0
    return [one(x) for x in xs]


def scan(parts, step, shape):
    """Run ``step(S, inputs of token t) -> (S, out)`` over all sequences side by side: ``parts``, per
    sequence, the tensors whose first dimension is the token; shorter sequences end in zeros."""
    T = max(len(p[0]) for p in parts)
    stacked = [torch.stack([torch.cat([p[j], p[j].new_zeros(T - len(p[j]), *p[j].shape[1:])]) for p in parts], 1)
               for j in range(len(parts[0]))]
    S = [stacked[0].new_zeros(len(parts), *s) for s in shape]
    outs = []
    for t in range(T):
        S, o = step(S, *(x[t] for x in stacked))
        outs.append(o)
    out = torch.stack(outs, 1)
    return [out[b, :len(p[0])] for b, p in enumerate(parts)]


def delta_step(S, q, k, v, beta, g):
    S = S[0] * g[..., None, None]
    u = beta[..., None] * (v - (S * k[..., None]).sum(-2))
    S = S + k[..., None] * u[..., None, :]
    return [S], (S * q[..., None]).sum(-2)


def memory_step(state, q, k, v, ig, fg):
    S, n, mx = state
    new = torch.maximum(fg + mx, ig)
    keep, take = torch.exp(fg + mx - new)[..., None], torch.exp(ig - new)[..., None]
    S = keep[..., None] * S + (take * k)[..., None] * v[..., None, :]
    n = keep * n + take * k
    den = torch.maximum((n * q).sum(-1).abs(), torch.exp(-new)) + 1e-6
    return [S, n, new], (S * q[..., None]).sum(-2) / den[..., None]


def conv(x, w):
    """y[t] = sum_j w[:, j] x[t - taps + 1 + j], zeros before the start."""
    taps = w.shape[1]
    padded = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(padded[j:j + len(x)] * w[:, j] for j in range(taps))


def karupel_layer(xs, w, i, cfg, first):
    layer, eps, p = cfg["layers"][i], cfg["norm"]["eps"], f"l{i}.mix."
    m = layer["mixer"]
    H, D, U, F = m["heads"], m["dim"], m["vdim"], torch.nn.functional
    G = m.get("kv_heads", H)
    if layer["type"] == "delta":
        parts = []
        for x in xs:
            q, k, v = (silu(conv(x @ w(p + n).T, w(p + n + ".conv"))).view(len(x), -1, d)
                       for n, d in (("q", D), ("k", D), ("v", U)))
            q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
            q, k = (t.repeat_interleave(H // G, 1) for t in (q * D ** -0.5, k))
            parts.append((q, k, v, torch.sigmoid(x @ w(p + "b").T),
                          torch.exp(-torch.exp(w(p + "A_log")) * F.softplus(x @ w(p + "a").T + w(p + "dt_bias")))))
        outs = scan(parts, delta_step, [(H, D, U)])
        ys = [(unit(o, eps) * w(p + "norm") * silu(x @ w(p + "g").T).view(len(x), H, U)).reshape(len(x), -1)
              for x, o in zip(xs, outs)]
    elif layer["type"] == "mlstm":
        cap, parts = m["gate_cap"], []
        for x in xs:
            q, k, v = ((x @ w(p + n).T).view(len(x), H, -1) for n in "qkv")
            ig, fg = (cap * torch.tanh((x @ w(p + n).T + w(p + n + ".b")) / cap) for n in "if")
            parts.append((q * D ** -0.5, k, v, ig, F.logsigmoid(fg)))
        outs = scan(parts, memory_step, [(H, D, U), (H, D), (H,)])
        ys = [unit(o, eps).reshape(len(x), -1) * w(p + "norm") * torch.sigmoid(x @ w(p + "g").T)
              for x, o in zip(xs, outs)]
    else:
        ys = []
        rot = m["rot"]
        half = torch.arange(rot["dims"] // 2, dtype=torch.float64, device="cuda")
        freq = rot["base"] ** (-2.0 * half / rot["dims"]) / rot["scaling"]["factor"]
        for b, x in enumerate(xs):
            q, k, v = ((x @ w(p + n).T + w(p + n + ".b")).view(len(x), -1, d)
                       for n, d in (("q", D), ("k", D), ("v", U)))
            q, k = (turn_halves(unit(t, eps) * w(p + n + ".norm"), rot["dims"], freq)
                    for t, n in ((q, "q"), (k, "k")))
            v_first = first.setdefault(b, v)
            if v_first is not v:
                v = (1 - w(p + "vmix")) * v + w(p + "vmix") * v_first
            gate = torch.sigmoid(x @ w(p + "g").T).repeat_interleave(U, 1)
            ys.append(attend(q, k, v, m["scale"]) * gate)
    out, q = [], f"l{i}.mlp."
    for x, y in zip(xs, ys):
        x = x + unit(y @ w(p + "o").T, eps) * (1 + w(f"l{i}.norm1"))
        y = (silu(x @ w(q + "gate").T) * (x @ w(q + "up").T)) @ w(q + "down").T
        out.append(x + unit(y, eps) * (1 + w(f"l{i}.norm2")))
    return out


def yarn(dims, base, s):
    """Frequencies of the dims / 2 pairs and the factor on cosine and sine."""
    def index_of(turns):
        return dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))

    lo, hi = max(math.floor(index_of(s["fast"])), 0), min(math.ceil(index_of(s["slow"])), dims - 1)
    i = torch.arange(dims // 2, dtype=torch.float64, device="cuda")
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    plain = base ** (-2.0 * i / dims)
    return plain / s["factor"] * ramp + plain * (1 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def kerolorn_layer(xs, w, i, cfg):
    layer, eps, p, e = cfg["layers"][i], cfg["norm"]["eps"], f"l{i}.mix.", f"l{i}.mlp."
    m, mlp = layer["mixer"], layer["mlp"]
    freq, magnitude = yarn(m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"])
    out = []

    def turn_pairs(x):
        ang = torch.arange(len(x), device="cuda", dtype=torch.float64)[:, None] * freq
        c, s = magnitude * torch.cos(ang)[:, None], magnitude * torch.sin(ang)[:, None]
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)

    def gated(h, n):
        return (silu(h @ w(n + "gate").T) * (h @ w(n + "up").T)) @ w(n + "down").T

    for x in xs:
        h = unit(x, eps) * w(f"l{i}.norm1")
        h = h + conv(h, w(f"l{i}.canon1"))
        q, k, v = ((h @ w(p + n).T).view(len(h), -1, d) for n, d in (("q", m["dim"]), ("k", m["dim"]), ("v", m["vdim"])))
        q, k = unit(turn_pairs(q), eps), unit(turn_pairs(k), eps)
        y = attend(q, k, v, m["scale"] * w(p + "temp"), 0.0, m["mask"]["size"], m["mask"]["keep_first"])
        x = x + unit(y @ w(p + "o").T, eps) * w(f"l{i}.norm1b")
        h = unit(x, eps) * w(f"l{i}.norm2")
        score = torch.softmax(h @ w(e + "router").T, -1)
        chosen = (score + w(e + "correction")).topk(mlp["router"]["top"], -1).indices
        weight = torch.zeros_like(score).scatter(1, chosen, score.gather(1, chosen) * mlp["router"]["scale"])
        y = torch.sigmoid(h @ w(e + "shared.sg").T) * gated(h, e + "shared.")
        for n in range(mlp["router"]["experts"]):
            rows = weight[:, n].nonzero()[:, 0]
            if len(rows):
                y[rows] += weight[rows, n, None] * gated(h[rows], e + f"e{n}.")
        out.append(x + unit(y, eps) * w(f"l{i}.norm2b"))
    return out


def last_logits(c, cfg, stored, sequences):
    """Logits of each sequence's last token."""
    def w(name):
        return stored[name].double()

    def rows_of(table, ids):
        return stored[table][torch.tensor(ids, device="cuda")].double()

    gemma2 = c["model"] == "gemma2"
    table = "model.embed_tokens.weight" if gemma2 else "embed"
    xs = [rows_of(table, ids) for ids in sequences]
    first = {}
    if gemma2:
        scale = torch.tensor(cfg["hidden_size"] ** 0.5, dtype=torch.float32).item()
        xs = [x * scale for x in xs]
    for i in range(c["layers"]):
        if gemma2:
            xs = gemma2_layer(xs, w, i, cfg)
        elif c["model"] == "karupel":
            xs = karupel_layer(xs, w, i, cfg, first)
        else:
            xs = kerolorn_layer(xs, w, i, cfg)
    x = torch.stack([x[-1] for x in xs])
    if gemma2:
        y = unit(x, cfg["rms_norm_eps"]) * (1 + w("model.norm.weight"))
        cap = cfg["final_logit_softcapping"]
        return cap * torch.tanh(y @ w(table).T / cap)
    if c["model"] == "karupel":
        return unit(x, cfg["norm"]["eps"]) * (1 + w("final.norm")) @ w("embed").T
    return (unit(x, cfg["norm"]["eps"]) * w("final.norm")) @ w("head").T * cfg["logit_scale"]


def exact(c, seed):
    rows = sum(lengths_of(c))
    if c["call"] == "decode" and work(dict(c, call="prompt"))["flops"] > 2.5e14:
        return None                     # (the whole context in 64 bits: over 20 seconds)
    if c["model"] == "karupel" and c["longest"] * c["layers"] > 40000 or rows > 200000:
        return None
    cfg, stored, ids = config_of(c), weights_of(c, seed), tokens_of(c, seed)
    extra = 1 if c["call"] == "decode" else 0
    sequences = [t[:n + extra] for t, n in zip(ids, lengths_of(c))]
    if c["call"] != "generate":
        return {"logits": last_logits(c, cfg, stored, sequences)}
    chosen = [[] for _ in sequences]
    for _ in range(c["new"]):
        logits = last_logits(c, cfg, stored, sequences)
        for s, t, row in zip(sequences, chosen, logits.argmax(-1).tolist()):
            s.append(row)
            t.append(row)
    return {"tokens": torch.tensor(chosen), "logits": logits}
