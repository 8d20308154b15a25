"""Timed cases of the framework's public entry points: packed linears, groups of matvecs, the exporter's quantise-and-pack
with its inverse, and generation with the three model families (a prompt, then decode steps over given tokens).

`listed()` names the cases, `draw(rng)` gives more of the same ranges, `prepare(case, seed)` makes what a user's program
holds before the call, `run(state)` is one pass, `work(case)` what the pass cannot do without, `exact(case, seed)` the same
outputs in 64 bits from plain torch, `tolerance(case)` how far two correct implementations may be apart."""
import math
import zlib

import torch

from nativebit_b200 import MatvecGroup, PackedLinear, nabalix, nerulorn
from nativebit_b200 import generate as G
from nativebit_b200 import pack as P

DEV = "cuda"
TYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
VOCAB = 32000


# ---------------------------------------------------------------------- the cases
def _linear(n, k, rows, bits, dtype):
    return {"op": "linear", "n": n, "k": k, "rows": rows, "bits": bits, "dtype": dtype}


def _generate(family, width, ff, layers, heads, bits, dtype, batch, prompt, steps, context):
    return {"op": "generate", "family": family, "width": width, "ff": ff, "layers": layers, "heads": heads, "bits": bits, "dtype": dtype,
            "batch": batch, "prompt": prompt, "steps": steps, "context": context}


def listed():
    def named(name, case):
        return dict(case, name=name)
    return [
        # one activation row through one attention-sized linear: the smallest call, what a token by token caller makes
        named("linear 1 row", _linear(2560, 2560, 1, 3, "bf16")),
        # the down projection of a batch of 16 sequences
        named("linear 16 rows", _linear(2560, 6912, 16, 3, "bf16")),
        # a short prompt of an odd length through a fused q|k|v, fp32 activations as the packed decoder has them
        named("linear 129 rows f32", _linear(7680, 2560, 129, 3, "f32")),
        # a long prompt through gate (or up)
        named("linear 2048 rows", _linear(6912, 2560, 2048, 3, "bf16")),
        # all feed-forward matvecs of a 26-layer model, one row each, as one group: weights stream from memory
        named("group of 78", {"op": "group", "width": 2560, "ff": 6912, "layers": 26, "rows": 1, "bits": 3}),
        # exporter and loader of one feed-forward matrix: nearest entry, packing, dense weight back
        named("convert", {"op": "convert", "n": 6912, "k": 2560, "bits": 3, "block": 128}),
        # a small packed model answering a short question: latency
        named("packed small", _generate("packed", 1024, 2816, 4, 8, 3, "f32", 1, 17, 8, 512)),
        # the 2.2B packed model, one sequence: a prompt and a run of single-token steps
        named("packed 2.2B one sequence", _generate("packed", 2560, 6912, 26, 32, 3, "f32", 1, 128, 48, 1024)),
        # the same at 2 bits serving eight sequences whose prompts fill half the context
        named("packed 2.2B batch 8", _generate("packed", 2560, 6912, 26, 32, 2, "f32", 8, 512, 12, 1024)),
        # a batch past the few-row kernels, 12 layers
        named("packed batch 32", _generate("packed", 2560, 6912, 12, 32, 3, "f32", 32, 100, 12, 512)),
        # layered decoders: a long prompt, then single-token steps
        named("nerulorn", _generate("nerulorn", 2560, 6912, 12, 20, 16, "bf16", 1, 2048, 16, 4096)),
        named("nabalix", _generate("nabalix", 2048, 5632, 4, 16, 16, "bf16", 1, 1000, 16, 4096)),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.random()
    if kind < 0.4:
        n = _log(rng, 256, 13824)
        if rng.random() < 0.6:
            n = max(256, n // 16 * 16)
        return _linear(n, 128 * _log(rng, 4, 54), _log(rng, 1, 2048), rng.choice([3, 3, 3, 2, 4]), rng.choice(["bf16", "bf16", "f32", "f32", "f16"]))
    if kind < 0.5:
        width = 128 * rng.randint(8, 20)
        return {"op": "group", "width": width, "ff": 128 * rng.randint(20, 54), "layers": rng.randint(2, 26),
                **rng.choice([{"rows": 1, "bits": 3}, {"rows": 4, "bits": 3}, {"rows": 2, "bits": 2}, {"rows": 1, "bits": 4}])}
    if kind < 0.6:
        return {"op": "convert", "n": _log(rng, 100, 6912), "k": _log(rng, 100, 2560), "bits": rng.choice([3, 3, 2, 4]), "block": rng.choice([128, 128, 64, 8])}
    width = rng.choice([1024, 2048, 2560])
    ff = {1024: 2816, 2048: 5632, 2560: 6912}[width]
    if kind < 0.85:
        batch = rng.choice([1, 1, 1, 2, 4, 8, 16, 24, 32])
        prompt = _log(rng, 5, 480) if batch > 1 else _log(rng, 5, 960)
        return _generate("packed", width, ff, rng.randint(2, 12), {1024: 8, 2048: 16, 2560: 32}[width], rng.choice([3, 3, 2, 4]), "f32", batch, prompt,
                         rng.randint(4, 24), 512 if batch > 1 else 1024)
    family = rng.choice(["nerulorn", "nabalix"])
    layers = rng.randint(1, 2) * (4 if family == "nerulorn" else 2)
    dtype = rng.choice(["bf16", "bf16", "bf16", "f32"])
    return _generate(family, width, ff, layers, width // 128, 16, dtype, 1, _log(rng, 16, 2048 if dtype == "bf16" else 512), rng.randint(4, 16), 4096)


# ---------------------------------------------------------------------- inputs
def _gen(seed, tag):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + zlib.crc32(tag.encode())) % (1 << 62))


def _quantised(n, k, bits, seed, tag):
    """Uniform indices and a sorted codebook per 128 weights with a scale of its own: (indices (n * k), codebook fp16)."""
    g = _gen(seed, tag)
    idx = torch.randint(0, 1 << bits, (n * k,), dtype=torch.uint8, device=DEV, generator=g)
    blocks = n * k // 128
    cb = torch.randn(blocks, 1 << bits, device=DEV, generator=g).sort(dim=1).values
    cb = cb * torch.empty(blocks, 1, device=DEV).uniform_(0.01, 0.05, generator=g)
    return idx, cb.half()


def _dense(idx, cb, n, k):
    """The weight of `_quantised` in 64 bits."""
    return torch.gather(cb.double(), 1, idx.view(-1, 128).long()).view(n, k)


def _rows(rows, k, seed, tag, dtype=torch.float32):
    return torch.randn(rows, k, device=DEV, generator=_gen(seed, tag)).to(dtype)


def _near_one(n, seed, tag):
    return 1.0 + 0.1 * torch.randn(n, device=DEV, generator=_gen(seed, tag))


def _tokens(case, seed):
    """(prompt (batch, prompt), the tokens of the steps (batch, steps))"""
    t = torch.randint(0, VOCAB, (case["batch"], case["prompt"] + case["steps"]), device=DEV, generator=_gen(seed, "tokens"))
    return t[:, :case["prompt"]].contiguous(), t[:, case["prompt"]:].contiguous()


GROUP = (("gate", 0), ("up", 0), ("down", 1))


def _group_shape(case, down):
    return (case["width"], case["ff"]) if down else (case["ff"], case["width"])


PACKED = ("qkv", "out_proj", "gate", "up", "down")


def _packed_shape(case, name):
    c, f = case["width"], case["ff"]
    return {"qkv": (3 * c, c), "out_proj": (c, c), "gate": (f, c), "up": (f, c), "down": (c, f)}[name]


def _packed_model(case, seed):
    c = case["width"]
    cfg = G.ModelConfig(vocab_size=VOCAB, n_layers=case["layers"], n_embd=c, n_head=case["heads"], ffn_hidden=case["ff"], context_len=case["context"],
                        bits=case["bits"])
    blocks = []
    for i in range(case["layers"]):
        full = {}
        for name in PACKED:
            idx, cb = _quantised(*_packed_shape(case, name), case["bits"], seed, f"{i}.{name}")
            full[name] = (P.pack_nbits(idx, case["bits"]), cb)
        blocks.append(G.shard_block(cfg, full, _near_one(c, seed, f"{i}.ln1"), _near_one(c, seed, f"{i}.ln2"), 0, 1))
    emb = (0.02 * _rows(VOCAB, c, seed, "embedding")).bfloat16()
    return G.PackedGPT(cfg, emb, blocks, _near_one(c, seed, "ln_f"))


def _nerulorn_config(case):
    """Gated linear attention and latent attention in turn, a feed-forward behind the latter; every second latent layer
    reads the cache of the one before."""
    c, h = case["width"], case["heads"]
    rot = {"dims": 64, "base": 500000.0, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
    layers = []
    for i in range(case["layers"]):
        if i % 2 == 0:
            layers.append({"type": "gla", "mlp": None, "mixer": {"heads": h, "dim": 128, "vdim": 128, "tau": 16.0}})
            continue
        mix = {"heads": h, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": c * 3 // 8, "mask": {"size": 1024}, "rot": rot,
               "scale": 192 ** -0.5}
        if i % 4 == 3:
            mix["kv_from"] = i - 2
        layers.append({"type": "latent_attention", "mlp": {"kind": "dense", "ff": case["ff"]}, "mixer": mix})
    return {"architecture": "Nerulorn", "vocab": VOCAB, "width": c, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0}, "layers": layers}


def _nabalix_config(case):
    """Attention with mixed heads beside the forget-gate recurrence in every layer, two residual streams."""
    h = case["heads"]
    mixer = {"left": {"heads": h, "kv_heads": h // 4, "dim": 128, "vdim": 128, "mask": {"size": 1024}, "scale": 128 ** -0.5, "softcap": 30.0},
             "right": {"heads": h, "dim": 128, "vdim": 128}}
    return {"architecture": "Nabalix", "vocab": VOCAB, "width": case["width"], "streams": 2, "norm": {"eps": 1e-6},
            "layers": [{"type": "parallel", "mixer": mixer, "mlp": {"kind": "dense", "ff": case["ff"], "limit": 7.0}} for _ in range(case["layers"])]}


#: mean and spread of the vectors of a checkpoint, by the end of their names; everything else is a matrix ~ N(0, 1 / fan-in)
_VECTORS = {
    "nerulorn": {"norm": (1, 0.1), "norm1": (1, 0.1), "norm1b": (1, 0.1), "norm2": (1, 0.1), "norm2b": (1, 0.1), "a2.b": (1, 1), "b": (0, 0.1)},
    "nabalix": {"norm1": (0, 0.1), "norm2": (0, 0.1), "final.norm": (0, 0.1), "right.norm": (1, 0.1), "out": (1, 0.1), "f.b": (1.5, 1.5),
                "ls1": (0.5, 0.1), "ls2": (0.5, 0.1), "hc1.in": (0.5, 0.2), "hc2.in": (0.5, 0.2), "hc1.out": (1, 0.2), "hc2.out": (1, 0.2)},
}
_UNIFORM = {"r1": (0.0, 2.0), "r2": (0.05, 0.5), "lower": (0.0, 0.9)}


def _weights(case, seed):
    """tensor(name, shape) -> a seeded bf16 weight of a layered model."""
    vectors = _VECTORS[case["family"]]

    def tensor(name, shape):
        shape = tuple(16 if s is None else s for s in shape)
        g = _gen(seed, name)
        z = torch.randn(shape, device=DEV, generator=g)
        last = name.rsplit(".", 1)[-1]
        if last in _UNIFORM:
            lo, hi = _UNIFORM[last]
            return torch.empty(shape, device=DEV).uniform_(lo, hi, generator=g).bfloat16()
        if last in ("talk", "mix"):
            return (torch.eye(shape[0], device=DEV) + (0.3 if last == "talk" else 0.15) * z).bfloat16()
        if len(shape) == 1:
            ends = [e for e in vectors if name == e or name.endswith("." + e)]
            mean, std = vectors[max(ends, key=len)]
            return (mean + std * z).bfloat16()
        return (z if name == "embed" else z * shape[1] ** -0.5).bfloat16()
    return tensor


def prepare(case, seed):
    op = case["op"]
    if op == "linear":
        idx, cb = _quantised(case["n"], case["k"], case["bits"], seed, "w")
        lin = PackedLinear(P.pack_nbits(idx, case["bits"]), cb, case["n"], case["k"], bits=case["bits"])
        return {"op": op, "lin": lin, "x": _rows(case["rows"], case["k"], seed, "x", TYPES[case["dtype"]])}
    if op == "group":
        m, c, f = case["rows"], case["width"], case["ff"]
        x = [_rows(m, c, seed, "x", torch.bfloat16), _rows(m, f, seed, "h", torch.bfloat16)]     # a group takes a few distinct inputs
        out = torch.zeros(case["layers"], m * (2 * f + c), dtype=torch.bfloat16, device=DEV)
        items = []
        for i in range(case["layers"]):
            at = 0
            for name, down in GROUP:
                n, k = _group_shape(case, down)
                idx, cb = _quantised(n, k, case["bits"], seed, f"{i}.{name}")
                items.append((PackedLinear(P.pack_nbits(idx, case["bits"]), cb, n, k, bits=case["bits"]), x[down], out[i, at:at + m * n].view(m, n)))
                at += m * n
        return {"op": op, "group": MatvecGroup(items), "out": out}
    if op == "convert":
        n, k = case["n"], case["k"]
        blocks = -(-n * k // case["block"])
        cb = 0.02 * _rows(blocks, 1 << case["bits"], seed, "cb").sort(dim=1).values
        return {"op": op, "w": 0.02 * _rows(n, k, seed, "w"), "cb": cb, "block": case["block"]}
    if case["family"] == "packed":
        session = _packed_model(case, seed).session(case["batch"])
    else:
        family, config = (nerulorn, _nerulorn_config(case)) if case["family"] == "nerulorn" else (nabalix, _nabalix_config(case))
        model = family.build(config, _weights(case, seed), TYPES[case["dtype"]], case["context"])
        torch.cuda.synchronize()             # as the loader does: decode kernels request weights ahead of the stream's order
        session = model.session(case["batch"])
    prompt, steps = _tokens(case, seed)
    out = torch.zeros(case["steps"] + 1, case["batch"], VOCAB, device=DEV)
    return {"op": op, "session": session, "prompt": prompt, "steps": [steps[:, i:i + 1].contiguous() for i in range(case["steps"])], "out": out}


# ---------------------------------------------------------------------- one pass
def run(state):
    op = state["op"]
    if op == "linear":
        return state["lin"](state["x"])
    if op == "group":
        state["group"].run()
        return state["out"]
    if op == "convert":
        lin = P.pack_linear(state["w"], state["cb"], state["block"])
        return {"packed": lin.packed_indices, "codebook": lin.codebook, "dense": lin.dequantized_weight()}
    # the tokens of the steps are given, as a sampler would give them: logits of every step come back
    session, out = state["session"], state["out"]
    out[0].copy_(session.prefill(state["prompt"]))
    for i, token in enumerate(state["steps"]):
        out[i + 1].copy_(session.extend(token)[:, -1])
    return out


def _packed_bytes(n, k, bits):
    return n * k * bits / 8 + n * k / 128 * (1 << bits) * 2


def _bytes_of(dtype):
    return 4 if dtype == "f32" else 2


def work(case):
    """Weights once per pass of the path over them (a prompt, a decode step), activations in and out, cached keys and values
    once per step that reads them; two operations per weight and row."""
    op = case["op"]
    if op == "linear":
        n, k, m = case["n"], case["k"], case["rows"]
        return {"bytes": _packed_bytes(n, k, case["bits"]) + m * (n + k) * _bytes_of(case["dtype"]), "flops": 2.0 * m * n * k}
    if op == "group":
        c, f, m = case["width"], case["ff"], case["rows"]
        return {"bytes": case["layers"] * (3 * _packed_bytes(f, c, case["bits"]) + m * (2 * f + c) * 2), "flops": case["layers"] * 6.0 * m * c * f}
    if op == "convert":
        n, k, e = case["n"], case["k"], 1 << case["bits"]
        # weight and codebook in, packed indices and fp16 codebook out and in again, dense weight out
        return {"bytes": n * k * (8 + 2 * case["bits"] / 8) + n * k / case["block"] * e * 8, "flops": 3.0 * n * k * e}
    c, f, t, b, s = case["width"], case["ff"], case["prompt"], case["batch"], case["steps"]
    head = VOCAB * c
    seen = sum(t + i + 1 for i in range(s))                      # keys that the steps read
    if case["family"] == "packed":
        weights = case["layers"] * (4 * c * c + 3 * c * f)
        nbytes = (s + 1) * (_packed_bytes(weights, 1, case["bits"]) + 2 * head)
        cache = case["layers"] * b * c * 2 * 4
        pairs = case["layers"] * b * c * (t * (t + 1) / 2 + seen)
    elif case["family"] == "nerulorn":
        h, pair = case["heads"] * 128, (case["layers"] + 1) // 2
        q = c * 3 // 8
        att = c * (q + 576 + case["heads"]) + q * case["heads"] * 192 + 512 * 2 * h + h * c + 3 * c * f
        weights = pair * (c * (4 * h + 16) + 16 * h + h * c) + (case["layers"] - pair) * att
        nbytes = (s + 1) * 2 * (weights + head) + pair * (s + 1) * 2 * h * 128 * 4
        cache = (case["layers"] - pair) * 576 * _bytes_of(case["dtype"])
        near = sum(min(i + 1, 1024) for i in range(t))
        pairs = (case["layers"] - pair) * h * 1.25 * near + pair * h * 128 * 2 * t
    else:
        h = case["heads"] * 128
        weights = case["layers"] * (c * (2 * h + h // 2) + c * 3 * h + 2 * h * c + 3 * c * f)
        nbytes = (s + 1) * 2 * (weights + head) + case["layers"] * (s + 1) * 2 * h * 128 * 4
        cache = case["layers"] * (h // 2) * _bytes_of(case["dtype"])
        near = sum(min(i + 1, 1024) for i in range(t))
        pairs = case["layers"] * h * (near + 128 * 2 * t)
    nbytes += cache * (t + (seen if case["family"] == "packed" else min(t, 1024) * s))
    nbytes += (s + 1) * b * VOCAB * 4
    return {"bytes": float(nbytes), "flops": 2.0 * b * ((t + s) * weights + (s + 1) * head) + 4.0 * pairs}


def tolerance(case):
    op = case["op"]
    if op == "convert":
        return "exact"                        # nearest entries, bytes and a gather: nothing is summed
    if op in ("linear", "group"):
        return {"rel": {"bf16": 6e-3, "f16": 1e-3, "f32": 1e-5}[case.get("dtype", "bf16")]}
    if case["family"] == "packed":
        return {"rel": 2e-4}                  # fp32 activations through up to 26 layers: 5e-5 from 64 bits
    return {"rel": 2e-2} if case["dtype"] == "bf16" else {"rel": 1e-4}


# ---------------------------------------------------------------------- the same in 64 bits
def _rms(x, w, eps=1e-6):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _layer_norm(x, w, eps):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w


def _turn(x, cos, sin):
    """x (..., T, D): pairs (2i, 2i + 1) turned; cos, sin (T, D / 2)."""
    u, v = x[..., ::2], x[..., 1::2]
    return torch.stack((u * cos - v * sin, v * cos + u * sin), -1).reshape(x.shape)


def _attend(q, k, v, scale, window):
    """(B, H, T, .): causal, the last `window` keys."""
    t = q.shape[2]
    d = torch.arange(t, device=DEV)[:, None] - torch.arange(t, device=DEV)[None, :]
    s = (q @ k.transpose(-1, -2)) * scale
    return torch.softmax(s.masked_fill((d < 0) | (d >= window), float("-inf")), -1) @ v


def _recur(q, k, v, decay):
    """(B, T, H, D): S <- diag(decay) S + k v^T, o = S^T q."""
    b, t, h, dim = q.shape
    s = torch.zeros(b, h, dim, v.shape[-1], dtype=torch.float64, device=DEV)
    out = torch.empty(b, t, h, v.shape[-1], dtype=torch.float64, device=DEV)
    for i in range(t):
        s = torch.addcmul(k[:, i, :, :, None] * v[:, i, :, None, :], decay[:, i, :, :, None], s)
        out[:, i] = (q[:, i, :, None, :] @ s)[:, :, 0]
    return out


def _exact_packed(case, seed, tokens, places):
    c, h = case["width"], case["heads"]
    hd, (b, t) = c // h, tokens.shape
    emb = (0.02 * _rows(VOCAB, c, seed, "embedding")).bfloat16()
    # the model's rotary tables are fp32 by definition
    f = 1.0 / (10000.0 ** (torch.arange(0, hd, 2, dtype=torch.float32, device=DEV) / hd))
    a = torch.outer(torch.arange(t, dtype=torch.float32, device=DEV), f)
    cos, sin = torch.cos(a).double(), torch.sin(a).double()
    x = emb[tokens].double()

    def w(i, name):
        shape = _packed_shape(case, name)
        return _dense(*_quantised(*shape, case["bits"], seed, f"{i}.{name}"), *shape).T
    for i in range(case["layers"]):
        q, k, v = ((_rms(x, _near_one(c, seed, f"{i}.ln1").double()) @ w(i, "qkv")).view(b, t, 3, h, hd).permute(2, 0, 3, 1, 4))
        o = _attend(_turn(q, cos, sin), _turn(k, cos, sin), v, hd ** -0.5, t)
        x = x + o.transpose(1, 2).reshape(b, t, c) @ w(i, "out_proj")
        y = _rms(x, _near_one(c, seed, f"{i}.ln2").double())
        x = x + (torch.nn.functional.silu(y @ w(i, "gate")) * (y @ w(i, "up"))) @ w(i, "down")
    z = _rms(x[:, places], _near_one(c, seed, "ln_f").double()) @ emb.double().T
    return 30.0 * torch.tanh(z / 30.0)


def _yarn(rot, t):
    """cos and sin of the rotated part, tables in fp32 as the model keeps them."""
    d, base, s = rot["dims"], rot["base"], rot["scaling"]
    f = [base ** (-2.0 * i / d) for i in range(d // 2)]

    def at(turns):
        return d * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(at(s["fast"])), 0), min(math.ceil(at(s["slow"])), d - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(d // 2)]
    f = torch.tensor([x / s["factor"] * r + x * (1.0 - r) for x, r in zip(f, ramp)], dtype=torch.float64, device=DEV)
    m = 0.1 * math.log(s["factor"]) + 1.0
    a = torch.outer(torch.arange(t, dtype=torch.float64, device=DEV), f)
    return (a.cos() * m).float().double(), (a.sin() * m).float().double()


def _exact_nerulorn(case, seed, tokens, places):
    cfg, tensor = _nerulorn_config(case), _weights(case, seed)
    c, eps, (b, t) = case["width"], 1e-6, tokens.shape
    x = tensor("embed", (VOCAB, c))[tokens].double()
    kept = {}
    for i, spec in enumerate(cfg["layers"]):
        m = spec["mixer"]
        h, dim, vd = m["heads"], m["dim"], m["vdim"]

        def w(name, *shape):
            return tensor(f"l{i}.{name}", shape).double()
        u = _layer_norm(x, w("norm1", c), eps)
        if spec["type"] == "gla":
            q = (u @ w("mix.q", h * dim, c).T).view(b, t, h, dim) * dim ** -0.5
            k, v = (u @ w("mix.k", h * dim, c).T).view(b, t, h, dim), (u @ w("mix.v", h * vd, c).T).view(b, t, h, vd)
            z = u @ w("mix.a1", 16, c).T @ w("mix.a2", h * dim, 16).T + w("mix.a2.b", h * dim)
            o = _rms(_recur(q, k, v, torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).view(b, t, h, dim)), w("mix.norm", vd))
            o = o.reshape(b, t, -1) * torch.nn.functional.silu(u @ w("mix.g", h * vd, c).T)
        else:
            rank, rd, qr = m["kv_rank"], m["rot_dim"], m["q_rank"]
            cos, sin = _yarn(m["rot"], t)
            q = (_rms(u @ w("mix.dq", qr, c).T, w("mix.dq.norm", qr)) @ w("mix.uq", h * (dim + rd), qr).T).view(b, t, h, -1).transpose(1, 2)
            if m.get("kv_from") is None:
                kv = u @ w("mix.dkv", rank + rd, c).T
                kept[i] = (_rms(kv[..., :rank], w("mix.dkv.norm", rank)), _turn(kv[..., rank:], cos, sin))
            lat, kr = kept[m.get("kv_from", i)]
            k = (lat @ w("mix.uk", h * dim, rank).T).view(b, t, h, dim).transpose(1, 2)
            v = (lat @ w("mix.uv", h * vd, rank).T).view(b, t, h, vd).transpose(1, 2)
            q = torch.cat((q[..., :dim], _turn(q[..., dim:], cos, sin)), -1)
            k = torch.cat((k, kr[:, None].expand(b, h, t, rd)), -1)
            o = _attend(q, k, v, m["scale"], m["mask"]["size"]).transpose(1, 2)
            o = (o * torch.sigmoid(u @ w("mix.g", h, c).T)[..., None]).reshape(b, t, -1)
        x = x + _layer_norm(o @ w("mix.o", c, h * vd).T, w("norm1b", c), eps)
        if spec["mlp"] is not None:
            f = spec["mlp"]["ff"]
            u = _layer_norm(x, w("norm2", c), eps)
            a = torch.nn.functional.silu(u @ w("mlp.gate", f, c).T + w("mlp.gate.b", f)) * (u @ w("mlp.up", f, c).T + w("mlp.up.b", f))
            x = x + _layer_norm(a @ w("mlp.down", c, f).T + w("mlp.down.b", c), w("norm2b", c), eps)
    return _layer_norm(x[:, places], tensor("final.norm", (c,)).double(), eps) @ tensor("head", (VOCAB, c)).double().T


def _exact_nabalix(case, seed, tokens, places):
    cfg, tensor = _nabalix_config(case), _weights(case, seed)
    c, n, (b, t) = case["width"], cfg["streams"], tokens.shape
    x = tensor("embed", (VOCAB, c))[tokens].double().expand(n, b, t, c)
    d = torch.arange(t, device=DEV)[:, None] - torch.arange(t, device=DEV)[None, :]
    for i, spec in enumerate(cfg["layers"]):
        def w(name, *shape):
            return tensor(f"l{i}.{name}", shape).double()

        def attention(u, m):
            h, g, dim, vd = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            q = (u @ w("mix.left.q", h * dim, c).T).view(b, t, h, dim).transpose(1, 2)
            k = (u @ w("mix.left.k", g * dim, c).T).view(b, t, g, dim).transpose(1, 2).repeat_interleave(h // g, 1)
            v = (u @ w("mix.left.v", g * vd, c).T).view(b, t, g, vd).transpose(1, 2).repeat_interleave(h // g, 1)
            s = m["softcap"] * torch.tanh((q @ k.transpose(-1, -2)) * (m["scale"] / m["softcap"]))
            s = s - w("mix.left.r1", h)[:, None, None] * torch.log1p(w("mix.left.r2", h)[:, None, None] * d.clamp(min=0))
            s = torch.einsum("hg,bgij->bhij", w("mix.left.talk", h, h), s)
            o = torch.softmax(s.masked_fill_((d < 0) | (d >= m["mask"]["size"]), float("-inf")), -1) @ v
            o = o.transpose(1, 2).reshape(b, t, -1) * torch.sigmoid(u @ w("mix.left.g", h * vd, c).T)
            return o @ w("mix.left.o", c, h * vd).T

        def recurrence(u, m):
            h, dim, vd = m["heads"], m["dim"], m["vdim"]
            q = torch.nn.functional.silu(u @ w("mix.right.q", h * dim, c).T).view(b, t, h, dim)
            v = (u @ w("mix.right.v", h * vd, c).T).view(b, t, h, vd)
            z, low = u @ w("mix.right.f", h * dim, c).T + w("mix.right.f.b", h * dim), w("mix.right.lower", h * dim)
            f, write = low + (1 - low) * torch.sigmoid(z), (1 - low) * torch.sigmoid(-z)
            o = _rms(_recur(q, write.view(b, t, h, dim), v, f.view(b, t, h, dim)), w("mix.right.norm", vd))
            return o.reshape(b, t, -1) @ w("mix.right.o", c, h * vd).T

        def mixer(u):
            left = _rms(attention(u, spec["mixer"]["left"]), w("mix.left.out", c))
            return w("ls1", c) * (left + _rms(recurrence(u, spec["mixer"]["right"]), w("mix.right.out", c))) / 2

        def feed_forward(u):
            f, lim = spec["mlp"]["ff"], spec["mlp"]["limit"]
            gate = (u @ w("mlp.gate", f, c).T).clamp(max=lim)
            up = (u @ w("mlp.up", f, c).T).clamp(-lim, lim)
            return w("ls2", c) * ((gate * torch.sigmoid(1.702 * gate) * (up + 1)) @ w("mlp.down", c, f).T)
        for j, sublayer in ((1, mixer), (2, feed_forward)):
            u = torch.tensordot(w(f"hc{j}.in", n), x, 1)
            y = sublayer(_rms(u, 1 + w(f"norm{j}", c)))
            x = torch.tensordot(w(f"hc{j}.mix", n, n).T, x, 1) + w(f"hc{j}.out", n)[:, None, None, None] * y
    return _rms(x.sum(0)[:, places], 1 + tensor("final.norm", (c,)).double()) @ tensor("head", (VOCAB, c)).double().T


@torch.no_grad()
def exact(case, seed):
    op = case["op"]
    if op == "linear":
        n, k = case["n"], case["k"]
        w = _dense(*_quantised(n, k, case["bits"], seed, "w"), n, k)
        return _rows(case["rows"], k, seed, "x", TYPES[case["dtype"]]).double() @ w.T
    if op == "group":
        m, c, f = case["rows"], case["width"], case["ff"]
        out = torch.empty(case["layers"], m * (2 * f + c), dtype=torch.float64, device=DEV)
        for i in range(case["layers"]):
            ys = []
            for name, down in GROUP:
                n, k = _group_shape(case, down)
                x = _rows(m, k, seed, "h" if down else "x", torch.bfloat16).double()
                ys.append((x @ _dense(*_quantised(n, k, case["bits"], seed, f"{i}.{name}"), n, k).T).reshape(-1))
            out[i] = torch.cat(ys)
        return out
    if op == "convert":
        n, k, block = case["n"], case["k"], case["block"]
        blocks = -(-n * k // block)
        cb = 0.02 * _rows(blocks, 1 << case["bits"], seed, "cb").sort(dim=1).values
        w = torch.zeros(blocks * block, device=DEV)
        w[:n * k] = (0.02 * _rows(n, k, seed, "w")).view(-1)
        near = torch.empty(blocks, block, dtype=torch.long, device=DEV)
        for a in range(0, blocks, 1 << 16):
            near[a:a + (1 << 16)] = (w.view(blocks, block)[a:a + (1 << 16), :, None].double() - cb[a:a + (1 << 16), None, :].double()).abs().argmin(-1)
        dense = torch.gather(cb.half().double(), 1, near).view(-1)[:n * k].view(n, k)
        return {"packed": None, "codebook": cb.half().double(), "dense": dense}
    tokens = torch.cat(_tokens(case, seed), 1)
    places = list(range(case["prompt"] - 1, case["prompt"] + case["steps"]))
    of = {"packed": _exact_packed, "nerulorn": _exact_nerulorn, "nabalix": _exact_nabalix}[case["family"]]
    return of(case, seed, tokens, places).transpose(0, 1).contiguous()
