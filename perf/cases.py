"""The work whose speed counts: prompts and single-token steps of this library's decoders at the sizes its own configurations name.

A case is a plain dict.  ``part`` says which entry points it goes through:

* ``"prompt"``: a whole Qwen2 model takes a prompt through ``Stepper.step`` (as ``Engine.generate`` does) and returns the last token's logits;
* ``"decode"``: a whole Qwen2 model takes one token a sequence through ``DecoderModel.forward`` in a captured graph and returns the logits;
* ``"layers"``: a run of layers (``Layer.run``) over a step's residual stream, in a captured graph, as the engine's steps run them;
* ``"mixers"``: the mixers (``Mixer.apply``) of layers of the other designs on normed rows, in a captured graph, from empty states.

``new`` and ``before`` list, per sequence, the tokens the step brings and those the cache holds already ("a,b,c").
"""
from __future__ import annotations

import hashlib
import math

import torch

DEVICE = "cuda"
EPS = 1e-6
THETA = 1000000.0
PAGE = 64
# (width, heads, key/value heads, head size, feed-forward width): the widths of qwen2.5-0.5b, of design_compare's middle size, of qwen2.5-7b
SMALL, MIDDLE, LARGE = (896, 14, 2, 64, 4864), (2048, 16, 4, 128, 8192), (3584, 28, 4, 128, 18944)
VOCAB = 151936


def _case(part, design, size, layers, new, before, dtype="bfloat16", **more):
    width, heads, kv_heads, dim, ff = size
    text = lambda v: ",".join(str(int(n)) for n in v)          # noqa: E731
    return dict(part=part, design=design, width=width, heads=heads, kv_heads=kv_heads, dim=dim, ff=ff, layers=layers, dtype=dtype,
                new=text(new), before=text(before), **more)


def _spread(n, low, high):
    """n lengths between low and high, unequal, as live sequences of a batch have."""
    return [low + (high - low) * ((i * 37 + 11) % n) // max(n - 1, 1) for i in range(n)]


def listed():
    return [
        # one user, one token: a run of layers of the small model, nothing but latency and launches
        dict(_case("layers", "qwen2", SMALL, 6, [1], [600]), name="decode_1"),
        # the benchmark's workload: a whole step of 8 sequences at context 4,096, embedding to logits
        dict(_case("decode", "qwen2", SMALL, 24, [1] * 8, [4095] * 8), name="decode_8_whole"),
        # a full batch of unequal sequences
        dict(_case("layers", "qwen2", SMALL, 6, [1] * 64, _spread(64, 300, 4000)), name="decode_64"),
        # the larger model: a few users
        dict(_case("layers", "qwen2", LARGE, 2, [1] * 8, _spread(8, 500, 2000)), name="decode_8_large"),
        # one prompt of 2,048 tokens through the step function, as generate() starts a request
        dict(_case("prompt", "qwen2", SMALL, 24, [2048], [0]), name="prompt_2048_whole"),
        # unequal prompts of a batch, among them a long one, at the larger model's widths
        dict(_case("layers", "qwen2", LARGE, 1, [5001, 1807, 700, 33], [0] * 4), name="prompt_large"),
        # the 32-bit engine on a short batch of prompts
        dict(_case("layers", "qwen2", SMALL, 2, [301, 207], [0, 0], "float32"), name="prompt_float32"),
        # linear attention with a fixed and with a learned decay: a prompt
        dict(_case("mixers", "kevelorn", MIDDLE, 2, [2048], [0]), name="linear_attention"),
        # the state-space mixer: two unequal prompts
        dict(_case("mixers", "pupidra_ssm", MIDDLE, 1, [1400, 647], [0, 0]), name="state_space"),
        # attention over latent rows: a prompt
        dict(_case("mixers", "pupidra_latent", MIDDLE, 1, [2048], [0]), name="latent_attention"),
        # attention whose weights are mixed across heads: a prompt
        dict(_case("mixers", "mebalorn", MIDDLE, 1, [1024], [0]), name="mixed_heads"),
        # a layer with differential attention beside its feed-forward: prompts
        dict(_case("layers", "razelorn", MIDDLE, 1, [1500, 500], [0, 0], window=1024), name="differential"),
    ]


def draw(rng):
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))      # noqa: E731
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "float32", "mixer", "mixer"])
    if kind == "decode":                                       # 1 to 64 sequences, contexts of 64 to 8,192 tokens
        size = rng.choice([SMALL, MIDDLE, LARGE])
        rows = log(1, 64)
        top = log(64, 8192 if rows <= 16 else 4096)
        return _case("layers", "qwen2", size, {SMALL: 6, MIDDLE: 4, LARGE: 2}[size], [1] * rows, [rng.randint(top // 3, top) for _ in range(rows)])
    if kind == "float32":
        return _float32(rng)
    if kind == "prompt":
        size = rng.choice([SMALL, MIDDLE, LARGE])
        rows = rng.choice([1, 1, 2, 4])
        total = log(160, 7000)
        return _case("layers", "qwen2", size, {SMALL: 3, MIDDLE: 2, LARGE: 1}[size], _parts(rng, total, rows), [0] * rows)
    design = rng.choice(["kevelorn", "pupidra_ssm", "pupidra_latent", "mebalorn", "razelorn"])
    size = rng.choice([SMALL, MIDDLE])
    rows = rng.choice([1, 1, 2, 3])
    total = log(200, 1500 if design == "mebalorn" else 3000)
    new = _parts(rng, total, rows)
    if design == "razelorn":
        return _case("layers", design, size, 1, new, [0] * rows, window=rng.choice([256, 1024]))
    return _case("mixers", design, size, 2 if design == "kevelorn" else 1, new, [0] * rows)


def _parts(rng, total, rows):
    cut = sorted(rng.randint(1, total - 1) for _ in range(rows - 1))
    return [max(17, b - a) for a, b in zip([0] + cut, cut + [total])]


def _float32(rng):
    if rng.random() < 0.5:                                     # single tokens
        rows = rng.randint(1, 12)
        return _case("layers", "qwen2", SMALL, 2, [1] * rows, [rng.randint(50, 1500) for _ in range(rows)], "float32")
    rows = rng.choice([1, 2, 3])
    return _case("layers", "qwen2", SMALL, 2, _parts(rng, rng.randint(60, 520), rows), [0] * rows, "float32")


# ---------------------------------------------------------------------------- sizes and configurations

def _ints(text):
    return [int(n) for n in text.split(",")]


def _mixer_sizes(case):
    """The mixer's config.json object."""
    W, H, G, D = (case[k] for k in ("width", "heads", "kv_heads", "dim"))
    design = case["design"]
    if design == "mebalorn":
        return {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "scale": D ** -0.5}
    if design == "pupidra_latent":
        rot = D // 2
        return {"heads": H, "dim": D, "rot_dim": rot, "vdim": D, "kv_rank": min(2 * D, 256 - rot), "scale": (D + rot) ** -0.5,
                "rot": {"base": 100000.0, "dims": rot}}
    if design == "pupidra_ssm":
        return {"heads": 2 * W // 64, "vdim": 64, "state": 128, "groups": 2, "conv": 4, "norm_groups": 2}
    if design == "razelorn":
        H, G = H * D // 128, G * D // 128
        return {"heads": H, "kv_heads": G, "dim": 64, "vdim": 128, "scale": 64 ** -0.5, "diff": 0.5, "mask": {"size": case["window"]},
                "rot": {"base": 500000.0, "dims": 48, "scaling": {"factor": 8.0, "high": 4.0, "low": 1.0, "original": 8192}}}
    raise ValueError(design)


def _decays(heads):
    return [1.0 - 2.0 ** -(3 + h % 6) for h in range(heads)]


def _vocab(case):
    return VOCAB if case["part"] in ("prompt", "decode") else 256


def _config(case):
    W, H, G, D, F, L = (case[k] for k in ("width", "heads", "kv_heads", "dim", "ff", "layers"))
    design = case["design"]
    if design == "qwen2":
        return {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "hidden_act": "silu", "torch_dtype": "bfloat16",
                "num_hidden_layers": L, "hidden_size": W, "num_attention_heads": H, "num_key_value_heads": G, "head_dim": D,
                "intermediate_size": F, "vocab_size": _vocab(case), "rope_theta": THETA, "rms_norm_eps": EPS,
                "max_position_embeddings": 32768, "tie_word_embeddings": True, "use_sliding_window": False}
    d = {"vocab": _vocab(case), "width": W, "norm": {"eps": EPS}}
    if design == "kevelorn":
        return dict(d, architecture="Kevelorn", layers=[
            {"type": "lightning", "mixer": {"heads": H, "dim": D, "vdim": D, "decay": _decays(H)}, "mlp": None},
            {"type": "gla", "mixer": {"heads": H, "dim": D, "vdim": D, "tau": 16.0}, "mlp": None}])
    if design == "mebalorn":
        return dict(d, architecture="Mebalorn", canon={"taps": 4}, layers=[{"type": "attention", "mixer": _mixer_sizes(case), "mlp": None}])
    if design == "razelorn":
        return dict(d, architecture="Razelorn", embedding={"scale": float(W) ** 0.5},
                    layers=[{"type": "attention", "mixer": _mixer_sizes(case), "mlp": {"kind": "dense", "ff": F}}])
    kind = "mamba2" if design == "pupidra_ssm" else "latent_attention"
    return dict(d, architecture="Pupidra", layers=[{"type": kind, "mixer": _mixer_sizes(case), "mlp": None}])


def _shapes(case):
    """Tensor name -> (shape, how it is drawn)."""
    W, H, G, D, F, L = (case[k] for k in ("width", "heads", "kv_heads", "dim", "ff", "layers"))
    design, V = case["design"], _vocab(case)
    out = {}
    if design == "qwen2":
        out["model.embed_tokens.weight"], out["model.norm.weight"] = ((V, W), "table"), ((W,), "one")
        for i in range(L):
            p = f"model.layers.{i}."
            for n, r in (("q", H * D), ("k", G * D), ("v", G * D)):
                out[p + f"self_attn.{n}_proj.weight"], out[p + f"self_attn.{n}_proj.bias"] = ((r, W), "matrix"), ((r,), "little")
            out[p + "self_attn.o_proj.weight"] = ((W, H * D), "matrix")
            out[p + "mlp.gate_proj.weight"] = out[p + "mlp.up_proj.weight"] = ((F, W), "matrix")
            out[p + "mlp.down_proj.weight"] = ((W, F), "matrix")
            out[p + "input_layernorm.weight"] = out[p + "post_attention_layernorm.weight"] = ((W,), "one")
        return out
    out.update({"embed": ((V, W), "table"), "final.norm": ((W,), "one"), "head": ((V, W), "matrix"), "l0.norm1": ((W,), "one")})
    m = None if design == "kevelorn" else _mixer_sizes(case)
    p = "l0.mix."
    if design in ("mebalorn", "razelorn"):
        out.update({"final.norm.b": ((W,), "little"), "l0.norm1.b": ((W,), "little")})
    if design == "kevelorn":
        out["l1.norm1"] = ((W,), "one")
        for i in (0, 1):
            out.update({f"l{i}.mix.{n}": ((H * D, W), "matrix") for n in "qkvg"})
            out[f"l{i}.mix.o"] = ((W, H * D), "matrix")
        out.update({"l0.mix.norm": ((H * D,), "one"), "l1.mix.norm": ((D,), "one"), "l1.mix.a1": ((16, W), "matrix"),
                    "l1.mix.a2": ((H * D, 16), "matrix"), "l1.mix.a2.b": ((H * D,), "little")})
    elif design == "pupidra_ssm":
        n, P, N, g = m["heads"], m["vdim"], m["state"], m["groups"]
        inner, conv = n * P, n * P + 2 * g * N
        out.update({p + "in": ((inner + conv + n, W), "matrix"), p + "conv": ((conv, 4), "taps"), p + "conv.b": ((conv,), "little"),
                    p + "dt_bias": ((n,), "dt_bias"), p + "A_log": ((n,), "a_log"), p + "D": ((n,), "one"), p + "norm": ((inner,), "one"),
                    p + "o": ((W, inner), "matrix"), "l0.ls1": ((W,), "one")})
    elif design == "pupidra_latent":
        rot, rank = m["rot_dim"], m["kv_rank"]
        out.update({p + "q": ((H * (D + rot), W), "matrix"), p + "dkv": ((rank + rot, W), "matrix"), p + "dkv.norm": ((rank,), "one"),
                    p + "uk": ((H * D, rank), "matrix"), p + "uv": ((H * D, rank), "matrix"), p + "o": ((W, H * D), "matrix"),
                    p + "g": ((H, W), "matrix"), "l0.ls1": ((W,), "one")})
    elif design == "mebalorn":
        for n, r in (("q", H * D), ("k", G * D), ("v", G * D)):
            out[p + n], out[p + n + ".b"] = ((r, W), "matrix"), ((r,), "little")
        out.update({p + "o": ((W, H * D), "matrix"), p + "q.norm": ((D,), "one"), p + "k.norm": ((D,), "one"), p + "sink": ((H,), "little"),
                    p + "talk": ((H, H), "identity"), "l0.canon1": ((W, 4), "taps")})
    else:
        n, g, d, v = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        out.update({p + "q": ((2 * n * d, W), "matrix"), p + "k": ((2 * g * d, W), "matrix"), p + "v": ((g * v, W), "matrix"),
                    p + "o": ((W, n * v), "matrix"), p + "q.norm": ((d,), "one"), p + "k.norm": ((d,), "one"),
                    "l0.mlp.up": ((F, W), "matrix"), "l0.mlp.down": ((W, F), "matrix")})
        out.update({p + "l" + n: ((d,), "little") for n in ("q1", "k1", "q2", "k2")})
    return out


# ---------------------------------------------------------------------------- inputs, from the seed alone

def _generator(seed, name):
    digest = hashlib.sha256(f"{seed}:{name}".encode("utf-8")).digest()
    return torch.Generator(DEVICE).manual_seed(int.from_bytes(digest[:7], "little"))


def _tensor(seed, name, shape, kind, dtype=torch.bfloat16):
    """One weight: of a size that keeps activations near one, as trained weights do."""
    g = _generator(seed, name)
    if kind in ("a_log", "dt_bias"):                           # decay rates of 1 to 16, time steps of 0.001 to 0.1
        u = torch.rand(shape, generator=g, device=DEVICE)
        if kind == "a_log":
            return torch.log(1 + 15 * u).to(dtype)
        dt = torch.exp(u * math.log(100.0) + math.log(0.001))
        return (dt + torch.log(-torch.expm1(-dt))).to(dtype)
    t = torch.randn(shape, generator=g, device=DEVICE)
    if kind == "matrix":
        t.mul_(shape[-1] ** -0.5)
    elif kind == "taps":
        t.mul_(0.5)
    elif kind == "identity":
        t = torch.eye(shape[0], device=DEVICE) + 0.05 * t
    elif kind == "table":
        t.mul_(0.5)
    else:
        t = 0.05 * t + (1.0 if kind == "one" else 0.0)
    return t.to(dtype)


def _rows(case, seed):
    """What enters: the residual stream, or the normed rows of a mixer."""
    T = sum(_ints(case["new"]))
    t = torch.randn(T, case["width"], generator=_generator(seed, "rows"), device=DEVICE)
    return t if case["part"] == "layers" else t.to(getattr(torch, case["dtype"]))


def _tokens(case, seed):
    g = torch.Generator().manual_seed(seed * 7919 + 13)
    return [torch.randint(0, _vocab(case), (n,), generator=g).tolist() for n in _ints(case["new"])]


def _cached(case, seed, layer):
    """Keys and values [rows, longest, heads, dim] that the cache holds before the step."""
    shape = (len(_ints(case["before"])), max(_ints(case["before"])), case["kv_heads"], case["dim"])
    dtype = getattr(torch, case["dtype"])
    return tuple(torch.randn(shape, generator=_generator(seed, f"{n}{layer}"), device=DEVICE, dtype=dtype) for n in "kv")


# ---------------------------------------------------------------------------- the library's side

def prepare(case, seed):
    from pico_engine.cache import Cache
    from pico_engine.config import config_from_dict
    from pico_engine.config.registry import architecture
    from pico_engine.engine.step import Stepper
    from pico_engine.ops.library import core, require_cuda
    from pico_engine.weights.loader import load_into
    device = require_cuda(f"{DEVICE}:{torch.cuda.current_device()}")
    core()
    dtype = getattr(torch, case["dtype"])
    with torch.inference_mode():
        config = config_from_dict(_config(case))
        model = architecture(config.ARCHITECTURE).build_model(config, dtype, device)
        shapes = _shapes(case)
        load_into(model, lambda n: _tensor(seed, n, *shapes[n]), {n: s for n, (s, _) in shapes.items()}, "the case's weights")
        new, before = _ints(case["new"]), _ints(case["before"])
        longest = max(n + b for n, b in zip(new, before))
        pages = sum(-(-(n + b) // PAGE) for n, b in zip(new, before))
        cache = Cache(model.cache_needs(), pages * PAGE, len(new), dtype, device)
        model.prepare(longest)
        stepper = Stepper(model, cache, longest)
        state = {"stepper": stepper, "cache": cache, "model": model, "tokens": _tokens(case, seed)}
        if case["part"] == "prompt":
            state["run"] = lambda: _prompt(state)
            return state
        slots = [cache.open() for _ in new]
        for s, n in zip(slots, before):
            if n:
                cache.reserve(s, n)
                cache.advance(s, n)
        if max(before):
            table = cache.page_table(0, slots)
            for e in range(case["layers"]):
                for pool, dense in zip(cache.pools(e), _cached(case, seed, e)):
                    for r, n in enumerate(before):
                        full = -(-n // PAGE)
                        rows = torch.zeros(full * PAGE, *dense.shape[2:], dtype=dtype, device=device)
                        rows[:n] = dense[r, :n]
                        at = torch.from_numpy(table[r, :full].astype("int64")).to(device)
                        pool[at] = rows.view(full, PAGE, *dense.shape[2:]).transpose(1, 2)
        layout, host, starts = stepper.describe(slots, new, None, state["tokens"])
        buffer = stepper.upload(host)
        ctx = stepper.context(layout, buffer, new, starts, slots)
        state.update(buffer=buffer, layout=layout, rows=_rows(case, seed))
        if case["part"] == "decode":
            body = lambda: model.forward(buffer[layout.ids: layout.ids + layout.T], ctx, buffer[layout.want: layout.want + layout.W])   # noqa: E731
        elif case["part"] == "layers":
            x = torch.empty_like(state["rows"])

            def body():
                x.copy_(state["rows"])
                for e, layer in enumerate(model.layers):
                    layer.run(x, ctx, e, e, True)
                ctx.settle(x)
                return x
        else:
            def body():
                out = []
                for e, layer in enumerate(model.layers):
                    if cache.state_of(e) is not None:          # as Cache.open does: a sequence starts from an empty state
                        cache.state_of(e).zero_()
                    out.append(layer.mixer.apply(state["rows"], ctx, e, e, True))
                return out
        state["out"], state["graph"] = _captured(body)
    return state


def _captured(body):
    """The step as the engine keeps it: run until everything lazy is set up, then captured."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            body()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = body()
    return out, graph


def _prompt(state):
    cache = state["cache"]
    slots = [cache.open() for _ in state["tokens"]]
    logits = state["stepper"].step(slots, state["tokens"], use_graph=True)
    for s in slots:
        cache.close(s)
    return logits


def run(state):
    if "graph" not in state:
        return state["run"]()
    state["graph"].replay()
    return state["out"]


# ---------------------------------------------------------------------------- what a pass cannot do without

def _seen(case, window=None):
    """Query and key pairs of the step."""
    total = 0
    for n, b in zip(_ints(case["new"]), _ints(case["before"])):
        if window is None:
            total += n * b + n * (n + 1) // 2
        else:
            total += sum(min(b + i + 1, window) for i in range(n))
    return total


def work(case):
    shapes, size = _shapes(case), 2 if case["dtype"] == "bfloat16" else 4
    new, before = _ints(case["new"]), _ints(case["before"])
    T, W, L = sum(new), case["width"], case["layers"]
    used = {n: s for n, (s, _) in shapes.items() if n.startswith(("l0.", "l1.", "model.layers."))}
    if case["part"] == "mixers":
        used = {n: s for n, s in used.items() if ".mix." in n}
    count = sum(math.prod(s) for s in used.values())
    matrices = sum(math.prod(s) for s in used.values() if len(s) == 2 and s[1] > 4)
    flops, nbytes = 2.0 * T * matrices, float(size * count)
    if case["part"] in ("prompt", "decode"):
        nbytes += size * VOCAB * W + 4.0 * len(new) * VOCAB + T * (4 + size * W)
        flops += 2.0 * len(new) * VOCAB * W
    elif case["part"] == "layers":
        nbytes += 8.0 * T * W
    else:
        nbytes += (1 + L) * float(size) * T * W
    design = case["design"]
    if design == "qwen2":
        kv = 2 * case["kv_heads"] * case["dim"] * size
        nbytes += L * kv * float(sum(before) + T)
        flops += 4.0 * L * case["heads"] * case["dim"] * _seen(case)
    elif design == "kevelorn":
        flops += 2 * 4.0 * T * case["heads"] * case["dim"] ** 2
        nbytes += 2 * 4.0 * len(new) * case["heads"] * case["dim"] ** 2
    elif design == "pupidra_ssm":
        m = _mixer_sizes(case)
        flops += 4.0 * T * m["heads"] * m["vdim"] * m["state"]
        nbytes += 4.0 * len(new) * m["heads"] * m["vdim"] * m["state"]
    elif design == "pupidra_latent":
        m = _mixer_sizes(case)                                 # scores over plain and rotated parts, then values: no carrying into the row
        flops += 2.0 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]) * _seen(case)
        nbytes += float(size) * T * (m["kv_rank"] + m["rot_dim"])
    elif design == "mebalorn":
        flops += 4.0 * case["heads"] * case["dim"] * _seen(case)
        nbytes += 2.0 * size * T * case["kv_heads"] * case["dim"]
    else:
        m = _mixer_sizes(case)
        flops += 2.0 * m["heads"] * (2 * m["dim"] + m["vdim"]) * _seen(case, case["window"])
        nbytes += float(size) * T * m["kv_heads"] * (2 * m["dim"] + m["vdim"])
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    if case["part"] in ("prompt", "decode"):                   # 24 layers of bfloat16 between the inputs and the logits
        return {"rel": 3e-2, "max": 0.5}
    return {"rel": 1e-2, "max": 0.3}


# ---------------------------------------------------------------------------- the same in 64 bits, written out plainly

def _unit(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _silu(z):
    return z * torch.sigmoid(z)


def _layer_norm(x, weight, bias):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + EPS) * weight + bias


def _turned_halves(u, positions, freqs):
    """u [n, heads, D]: entry i pairs with entry i + len(freqs); the entries behind stay."""
    half = len(freqs)
    angle = positions[:, None] * torch.tensor(freqs, dtype=torch.float64, device=u.device)
    c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    a, b = u[..., :half], u[..., half: 2 * half]
    return torch.cat([a * c - b * s, b * c + a * s, u[..., 2 * half:]], -1)


def _turned_pairs(u, positions, freqs):
    angle = positions[:, None] * torch.tensor(freqs, dtype=torch.float64, device=u.device)
    c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    a, b = u[..., 0::2], u[..., 1::2]
    return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)


def _seen_mask(first, n, window=None):
    """[n, first + n] bool: the keys a query at position first + i sees."""
    d = (first + torch.arange(n, device=DEVICE))[:, None] - torch.arange(first + n, device=DEVICE)[None]
    return (d >= 0) if window is None else (d >= 0) & (d < window)


def _softmax(scores, seen):
    return torch.softmax(scores.masked_fill(~seen, -math.inf), -1)


def _attention(q, k, v, scale, first, window=None):
    """q [n, H, D] of positions first.., k and v [first + n, G, D]."""
    n, H = q.shape[:2]
    per, seen = H // k.shape[1], _seen_mask(first, n, window)
    return torch.stack([_softmax(q[:, h] @ k[:, h // per].T * scale, seen) @ v[:, h // per] for h in range(H)], 1)


def _qwen2_layer(x, w, p, case, spans, cached):
    H, G, D = case["heads"], case["kv_heads"], case["dim"]
    freqs = [THETA ** (-2.0 * i / D) for i in range(D // 2)]
    h = _unit(x) * w(p + "input_layernorm.weight")
    q, k, v = (h @ w(p + f"self_attn.{n}_proj.weight").T + w(p + f"self_attn.{n}_proj.bias") for n in "qkv")
    rows = []
    for r, (at, n, b) in enumerate(spans):
        pos = torch.arange(b, b + n, dtype=torch.float64, device=x.device)
        qr = _turned_halves(q[at: at + n].view(n, H, D), pos, freqs)
        kr = _turned_halves(k[at: at + n].view(n, G, D), pos, freqs)
        vr = v[at: at + n].view(n, G, D)
        if b:
            kr, vr = torch.cat([cached[0][r, :b].double(), kr]), torch.cat([cached[1][r, :b].double(), vr])
        rows.append(_attention(qr, kr, vr, D ** -0.5, b).reshape(n, H * D))
    x = x + torch.cat(rows) @ w(p + "self_attn.o_proj.weight").T
    h = _unit(x) * w(p + "post_attention_layernorm.weight")
    return x + (_silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)) @ w(p + "mlp.down_proj.weight").T


def _recurrence(q, k, v, decay):
    """S_t = diag(decay_t) S_(t-1) + k_t v_t^T, o_t = S_t^T q_t; decay [n, H, D]."""
    n, H, D = q.shape
    S, out = torch.zeros(H, D, v.shape[2], dtype=q.dtype, device=q.device), torch.empty_like(v)
    for t in range(n):
        S = decay[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
        out[t] = torch.matmul(q[t][:, None, :], S)[:, 0]
    return out


def _linear_mixers(h, w, case):
    n, H, D = h.shape[0], case["heads"], case["dim"]
    heads = lambda name: (h @ w(name).T).view(n, H, D)         # noqa: E731
    q, k, v = (_silu(heads(f"l0.mix.{c}")) for c in "qkv")
    decay = torch.tensor(_decays(H), dtype=h.dtype, device=h.device).view(1, H, 1).expand(n, H, D)
    o = _unit(_recurrence(q, k, v, decay).reshape(n, H * D)) * w("l0.mix.norm")
    first = (o * torch.sigmoid(h @ w("l0.mix.g").T)) @ w("l0.mix.o").T
    q, k, v = heads("l1.mix.q") * D ** -0.5, heads("l1.mix.k"), heads("l1.mix.v")
    z = (h @ w("l1.mix.a1").T) @ w("l1.mix.a2").T + w("l1.mix.a2.b")
    o = _unit(_recurrence(q, k, v, (torch.sigmoid(z) ** (1.0 / 16.0)).view(n, H, D))) * w("l1.mix.norm")
    return [first, (o.reshape(n, H * D) * _silu(h @ w("l1.mix.g").T)) @ w("l1.mix.o").T]


def _state_space_mixer(h, w, case):
    m, n, p = _mixer_sizes(case), h.shape[0], "l0.mix."
    H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * P
    proj = h @ w(p + "in").T
    z, u, dt = proj[:, :inner], proj[:, inner: 2 * inner + 2 * G * N], proj[:, 2 * inner + 2 * G * N:]
    y = torch.zeros_like(u) + w(p + "conv.b")
    for j in range(4):
        shift = 3 - j
        y[shift:] += u[: n - shift] * w(p + "conv")[:, j]
    u = _silu(y)
    x = u[:, :inner].reshape(n, H, P)
    B, C = (u[:, inner + i * G * N: inner + (i + 1) * G * N].reshape(n, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    dt = torch.nn.functional.softplus(dt + w(p + "dt_bias"), threshold=100.0)
    decay = torch.exp(-torch.exp(w(p + "A_log")) * dt)[:, :, None].expand(n, H, N)
    y = _recurrence(C, dt[:, :, None] * B, x, decay) + w(p + "D")[:, None] * x
    y = y.reshape(n, inner) * _silu(z)
    y = _unit(y.view(n, m["norm_groups"], -1)).reshape(n, inner) * w(p + "norm")
    return y @ w(p + "o").T


def _latent_mixer(h, w, case):
    m, n, p = _mixer_sizes(case), h.shape[0], "l0.mix."
    H, D, R, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
    pos = torch.arange(n, dtype=torch.float64, device=h.device)
    freqs = [m["rot"]["base"] ** (-2.0 * i / R) for i in range(R // 2)]
    q = (h @ w(p + "q").T).view(n, H, D + R)
    down = h @ w(p + "dkv").T
    c = _unit(down[:, :rank]) * w(p + "dkv.norm")
    q_rot, k_rot = _turned_pairs(q[..., D:], pos, freqs), _turned_pairs(down[:, None, rank:], pos, freqs)[:, 0]
    k, v = ((c @ w(p + n2).T).view(n, H, D) for n2 in ("uk", "uv"))
    seen = _seen_mask(0, n)
    o = torch.stack([_softmax((q[:, a, :D] @ k[:, a].T + q_rot[:, a] @ k_rot.T) * m["scale"], seen) @ v[:, a] for a in range(H)], 1)
    return (o * torch.sigmoid(h @ w(p + "g").T)[:, :, None]).reshape(n, H * D) @ w(p + "o").T


def _mixed_heads_mixer(h, w, case):
    m, n, p = _mixer_sizes(case), h.shape[0], "l0.mix."
    H, G, D = m["heads"], m["kv_heads"], m["dim"]
    q, k, v = ((h @ w(p + c).T + w(p + c + ".b")).view(n, -1, D) for c in "qkv")
    q, k = _unit(q) * w(p + "q.norm"), _unit(k) * w(p + "k.norm")
    k, v = k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1)
    s = (torch.einsum("ihd,jhd->hij", q, k) * m["scale"]).masked_fill(~_seen_mask(0, n), -math.inf)
    s = torch.softmax(torch.cat([s, w(p + "sink").view(H, 1, 1).expand(H, n, 1)], -1), -1)[..., :n]
    o = torch.einsum("hij,jhd->ihd", torch.einsum("hg,gij->hij", w(p + "talk"), s), v)
    return o.reshape(n, H * D) @ w(p + "o").T


def _razelorn_layer(x, w, case, spans):
    m, p = _mixer_sizes(case), "l0.mix."
    H, G, D, V = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    sc, freqs = m["rot"]["scaling"], []
    for i in range(m["rot"]["dims"] // 2):
        f = m["rot"]["base"] ** (-2.0 * i / m["rot"]["dims"])
        s = min(max((sc["original"] * f / (2 * math.pi) - sc["low"]) / (sc["high"] - sc["low"]), 0.0), 1.0)
        freqs.append((1 - s) * f / sc["factor"] + s * f)
    lam = torch.exp((w(p + "lq1") * w(p + "lk1")).sum()) - torch.exp((w(p + "lq2") * w(p + "lk2")).sum()) + m["diff"]
    h = _layer_norm(x, w("l0.norm1"), w("l0.norm1.b"))
    rows = []
    for at, n, _ in spans:
        hr, pos = h[at: at + n], torch.arange(n, dtype=torch.float64, device=x.device)
        q = _turned_halves((_unit((hr @ w(p + "q").T).view(n, 2 * H, D)) * w(p + "q.norm")), pos, freqs).view(n, H, 2, D)
        k = _turned_halves((_unit((hr @ w(p + "k").T).view(n, 2 * G, D)) * w(p + "k.norm")), pos, freqs).view(n, G, 2, D)
        v = (hr @ w(p + "v").T).view(n, G, V)
        a1, a2 = (_attention(q[:, :, t], k[:, :, t], v, m["scale"], 0, case["window"]) for t in (0, 1))
        rows.append((_unit(a1 - lam * a2) * (1 - m["diff"])).reshape(n, H * V))
    return x + torch.cat(rows) @ w(p + "o").T + (torch.relu(h @ w("l0.mlp.up").T) ** 2) @ w("l0.mlp.down").T


def exact(case, seed):
    shapes = _shapes(case)
    dtype = getattr(torch, case["dtype"])
    w = lambda n: _tensor(seed, n, *shapes[n]).to(dtype).double()     # noqa: E731
    new, before = _ints(case["new"]), _ints(case["before"])
    spans, at = [], 0
    for n, b in zip(new, before):
        spans.append((at, n, b))
        at += n
    with torch.inference_mode():
        if case["part"] in ("prompt", "decode"):
            ids = torch.tensor([t for row in _tokens(case, seed) for t in row], device=DEVICE)
            x = w("model.embed_tokens.weight")[ids]
        else:
            x = _rows(case, seed).double()
        if case["design"] == "qwen2":
            for i in range(case["layers"]):
                cached = _cached(case, seed, i) if max(before) else None
                x = _qwen2_layer(x, w, f"model.layers.{i}.", case, spans, cached)
            if case["part"] == "layers":
                return x
            last = torch.tensor([a + n - 1 for a, n, _ in spans], device=DEVICE)
            return (_unit(x[last]) * w("model.norm.weight")) @ w("model.embed_tokens.weight").T
        if case["design"] == "razelorn":
            return _razelorn_layer(x, w, case, spans)
        mixer = {"kevelorn": _linear_mixers, "pupidra_ssm": lambda *a: [_state_space_mixer(*a)], "pupidra_latent": lambda *a: [_latent_mixer(*a)],
                 "mebalorn": lambda *a: [_mixed_heads_mixer(*a)]}[case["design"]]
        kept = {n: w(n) for n in shapes if ".mix." in n}
        parts = [mixer(x[a: a + n], kept.__getitem__, case) for a, n, _ in spans]
        return [torch.cat([p[i] for p in parts]) for i in range(len(parts[0]))]
