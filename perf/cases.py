"""The work that users of this framework have it do, as a list of measurable cases.

A case is one call sequence of a program that holds a plan (``B200MasterPlan``): a decode step that returns the logits of one token, or a
prompt that goes through the batched prefill and ends in logits.  Models are synthetic and have the layer geometries that this
repository's configurations, tests and benchmark use, with two layers (GGUF plans) or one to four layer runs (layered plans) and small
vocabularies: the layers of a deep model repeat the same launches.

Kinds
  gguf_decode     a GGUF plan (Q8_0 or FP16): ``forward_decode`` at a position of a sequence that is already in the cache
  gguf_prompt     a GGUF plan: all but the last prompt token through ``forward_batch_prefill`` in chunks, then ``forward_decode``
  layered_decode  a layered plan (BF16 weights): ``forward_decode`` at a position
  layered_prompt  a layered plan: a prompt through ``forward_batch_logits`` that wants the logits of a few rows

``draw`` gives cases of the same ranges: every geometry below, positions up to 3000, prompts of 2 to 513 tokens.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch


def _package():
    """The package's folder has a dot in its name: it is registered under the alias the framework documents."""
    name = "gpullama3_java_b200"
    if name not in sys.modules:
        root = os.path.join(os.getcwd(), "gpullama3.java_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(root, "__init__.py"), submodule_search_locations=[root])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# Layered geometries: the sizes of the framework's own model comparisons.
PIBIDRA = {  # width, ff, heads, kv_heads, head size, window, layers, loop (start, stop, times)
    "small": (1024, 4096, 16, 4, 64, 512, 2, None),
    "1b-like": (2048, 8192, 32, 8, 64, 1024, 3, (1, 2, 2)),
    "8b-like": (4096, 14336, 32, 8, 128, 2048, 2, None),
}
LATUSUN = {  # width, heads, unrotated, rotated, value, latent, experts, top, expert ff
    "small": (1024, 8, 48, 16, 64, 256, 8, 2, 1024),
    "lite-like": (2048, 16, 128, 64, 128, 512, 16, 4, 1408),
}
LEROSUN = {  # width, ff, attention heads, key heads, head size, window, delta value heads, q/k heads, key size, value size, taps
    "small": (1024, 4096, 16, 2, 64, 1024, 8, 4, 64, 128, 4),
    "1b-like": (2048, 8192, 16, 2, 128, 1024, 16, 8, 128, 128, 4),
}
LAYERED = {"pibidra": PIBIDRA, "latusun": LATUSUN, "lerosun": LEROSUN}
VOCAB = 32768
GGUF_SHAPES = ("tiny-llama", "tiny-qwen3", "tiny-phi3-gqa", "small-llama", "mid-llama-1b", "mid-qwen3-4b", "mid-phi3-mini", "mid-llama")
BATCH = 512  # tokens of one prefill call, as in the framework's benchmark


def listed():
    return [
        # the smallest call: one token of a toy model, where launches and the host path are all there is
        {"name": "tiny_q8_decode", "kind": "gguf_decode", "shape": "tiny-llama", "quant": "q8_0", "position": 20},
        # the headline: single-stream decode of an 8B Q8_0 model early in a chat
        {"name": "8b_q8_decode", "kind": "gguf_decode", "shape": "mid-llama", "quant": "q8_0", "position": 100},
        # the same late in a long conversation
        {"name": "8b_q8_decode_deep", "kind": "gguf_decode", "shape": "mid-llama", "quant": "q8_0", "position": 3000},
        # decode of a 1B FP16 model in the middle of an answer
        {"name": "1b_f16_decode", "kind": "gguf_decode", "shape": "mid-llama-1b", "quant": "f16", "position": 600},
        # a short question to a Q8_0 model, until its first logits
        {"name": "4b_q8_prompt", "kind": "gguf_prompt", "shape": "mid-qwen3-4b", "quant": "q8_0", "tokens": 37},
        # a long prompt to a Q8_0 model (one full prefill chunk and the first decode step)
        {"name": "8b_q8_prompt", "kind": "gguf_prompt", "shape": "mid-llama", "quant": "q8_0", "tokens": 513},
        # the same to an FP16 model
        {"name": "8b_f16_prompt", "kind": "gguf_prompt", "shape": "mid-llama", "quant": "f16", "tokens": 513},
        # layered plans: windowed attention with a loop block, decode in the middle of the window
        {"name": "pibidra_decode", "kind": "layered_decode", "design": "pibidra", "size": "1b-like", "compute": "bfloat16", "position": 900},
        # its prompt at the larger geometry
        {"name": "pibidra_prompt", "kind": "layered_prompt", "design": "pibidra", "size": "8b-like", "compute": "bfloat16", "tokens": 512},
        # latent attention and a mixture of experts: decode and prompt of one layer
        {"name": "latusun_decode", "kind": "layered_decode", "design": "latusun", "size": "lite-like", "compute": "bfloat16", "position": 511},
        {"name": "latusun_prompt", "kind": "layered_prompt", "design": "latusun", "size": "lite-like", "compute": "bfloat16", "tokens": 512},
        # a delta-rule layer and a head-mixed attention layer: prompt
        {"name": "lerosun_prompt", "kind": "layered_prompt", "design": "lerosun", "size": "1b-like", "compute": "bfloat16", "tokens": 512},
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("gguf_decode", "gguf_decode", "gguf_prompt", "gguf_prompt", "layered_decode", "layered_prompt"))
    if kind == "gguf_decode":
        return {"kind": kind, "shape": rng.choice(GGUF_SHAPES), "quant": rng.choice(("q8_0", "f16")), "position": _spread(rng, 1, 3000)}
    if kind == "gguf_prompt":
        return {"kind": kind, "shape": rng.choice(GGUF_SHAPES), "quant": rng.choice(("q8_0", "f16")), "tokens": _spread(rng, 3, 513)}
    design = rng.choice(("pibidra", "latusun", "lerosun")) if kind == "layered_prompt" else rng.choice(("pibidra", "latusun"))
    size = rng.choice(sorted(LAYERED[design]))
    compute = "float32" if size == "small" and rng.random() < 0.3 else "bfloat16"  # the runner's two modes
    case = {"kind": kind, "design": design, "size": size, "compute": compute}
    if kind == "layered_decode":
        return dict(case, position=_spread(rng, 1, 2000))
    return dict(case, tokens=_spread(rng, 2, 512))


# ---- models ---------------------------------------------------------------------------------------------------------------------
def _gguf(case, seed):
    """(shape, ggml type, {name: (type, dims, bytes)})"""
    pkg = _package()
    shape = pkg.synth.SHAPES[case["shape"]]
    quant = pkg.gguf.GGMLType.Q8_0 if case["quant"] == "q8_0" else pkg.gguf.GGMLType.F16
    return shape, quant, pkg.synth.build_tensors_fast(shape, quant, seed=seed, device="cuda")


def _tokens(vocab, n, seed):
    return np.random.default_rng(seed).integers(0, vocab, n).astype(np.int32)


class _Weights:
    """BF16 weights by name, made on the GPU from one seeded stream."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.w = {}

    def normal(self, name, shape, std=1.0, mean=0.0):
        self.w[name] = (torch.randn(shape, device="cuda", generator=self.gen) * std + mean).bfloat16()

    def mat(self, name, rows, cols, gain=1.0):
        self.normal(name, (rows, cols), gain / math.sqrt(cols))


def _pibidra(case, seed):
    E, F, H, G, hs, window, layers, loop = PIBIDRA[case["size"]]
    S = _package().synth
    cfg = S.pibidra_config(E, VOCAB, [S.pibidra_layer(H, G, hs, hs, window, F, bias_max=float(window)) for _ in range(layers)], loop=loop)
    b = _Weights(seed)
    b.normal("embed", (VOCAB, E), 0.1)
    b.mat("head", VOCAB, E)
    b.normal("final.norm", (E,), 0.2)
    if loop:
        b.normal("loop.step", (loop[2], E), 0.3)
    for i in range(layers):
        p = "l%d." % i
        for n in ("norm1", "norm1b", "norm2", "norm2b"):
            b.normal(p + n, (E,), 0.2)
        for n, rows, gain in (("q", H * hs, 2.0), ("k", G * hs, 2.0), ("v", G * hs, 1.0)):
            b.mat(p + "mix." + n, rows, E, gain)
            b.normal(p + "mix." + n + ".b", (rows,), 0.2)
        b.normal(p + "mix.q.norm", (H * hs,), 0.3, 1.0)
        b.normal(p + "mix.k.norm", (G * hs,), 0.3, 1.0)
        b.normal(p + "mix.rel", (32, H))
        b.mat(p + "mix.g", H * hs, E)
        b.mat(p + "mix.o", E, H * hs)
        b.mat(p + "mlp.gate", F, E)
        b.mat(p + "mlp.up", F, E)
        b.mat(p + "mlp.down", E, F)
    return cfg, b.w


def _latusun(case, seed):
    E, H, dk, dr, dv, R, X, top, F = LATUSUN[case["size"]]
    S = _package().synth
    blend = {"factor": 8.0, "original": 1024, "fast": 32.0, "slow": 1.0}
    cfg = S.latusun_config(E, VOCAB, [S.latusun_layer("latent_attention", H, dk, dr, dv, R, experts=X, top=top, ff=F, scaling=blend)])
    b = _Weights(seed)
    b.normal("embed", (VOCAB, E))
    b.mat("head", VOCAB, E, 3.0)
    for n in ("final.norm", "l0.norm1", "l0.norm2"):
        b.normal(n, (E,), 0.2, 1.0)
        b.normal(n + ".b", (E,), 0.1)
    p = "l0.mix."
    b.mat(p + "q", H * (dk + dr), E, 2.0)
    b.mat(p + "dkv", R + dr, E, 2.0)
    b.normal(p + "dkv.norm", (R,), 0.3, 1.0)
    b.mat(p + "uk", H * dk, R, 2.0)
    b.mat(p + "uv", H * dv, R)
    b.mat(p + "g", H * dv, E, 2.0)
    b.mat(p + "o", E, H * dv)
    b.mat("l0.mlp.router", X, E, 2.0)
    for e in range(X):
        b.mat("l0.mlp.e%d.gate" % e, F, E, 2.0)
        b.mat("l0.mlp.e%d.up" % e, F, E)
        b.mat("l0.mlp.e%d.down" % e, E, F, 2.0)
    return cfg, b.w


def _lerosun(case, seed):
    E, F, H, G, hs, window, DH, DG, dd, dv, taps = LEROSUN[case["size"]]
    S = _package().synth
    cfg = S.lerosun_config(E, VOCAB, [S.lerosun_delta(DH, DG, dd, dv, taps, F), S.lerosun_attention(H, G, hs, window, F, rot_dims=hs // 2)])
    b = _Weights(seed)
    b.normal("embed", (VOCAB, E), 0.1)
    b.mat("head", VOCAB, E)
    for n in ("embed.norm", "final.norm", "l0.norm1", "l0.norm2", "l1.norm1", "l1.norm2"):
        b.normal(n, (), 0.2, 1.0)
    for p in ("l0.", "l1."):
        b.normal(p + "ls1", (E,), 0.2, 0.5)
        b.normal(p + "ls2", (E,), 0.2, 0.5)
        b.mat(p + "mlp.gate", F, E)
        b.mat(p + "mlp.up", F, E)
        b.mat(p + "mlp.down", E, F)
    p = "l0.mix."
    for n, rows in (("q", DG * dd), ("k", DG * dd), ("v", DH * dv)):
        b.mat(p + n, rows, E, 2.0)
        b.normal(p + n + ".conv", (rows, taps), 0.6)
    b.mat(p + "b", DH, E, 2.0)
    b.mat(p + "a", DH, E, 2.0)
    b.normal(p + "A_log", (DH,), 0.7, -1.0)
    b.normal(p + "dt_bias", (DH,), 0.7)
    b.normal(p + "norm", (dv,), 0.2, 1.0)
    b.mat(p + "g", DH * dv, E, 2.0)
    b.mat(p + "o", E, DH * dv)
    p = "l1.mix."
    for n, rows in (("q", H * hs), ("k", G * hs)):
        b.mat(p + n, rows, E, 1.5)
        b.normal(p + n + ".b", (rows,), 0.2)
    b.normal(p + "talk", (H, H), 0.3)
    b.w[p + "talk"] = (b.w[p + "talk"].float() + torch.eye(H, device="cuda")).bfloat16()
    b.normal(p + "temp", (H,), 0.3, 1.0)
    b.normal(p + "sink", (H,))
    b.mat(p + "g", H, E, 2.0)
    b.mat(p + "o", E, H * hs)
    return cfg, b.w


def _layered(case, seed):
    return {"pibidra": _pibidra, "latusun": _latusun, "lerosun": _lerosun}[case["design"]](case, seed)


def _layered_model(case, cfg, w, context):
    L = _package().loader
    configuration = {"pibidra": L.pibidra_configuration, "latusun": L.latusun_configuration, "lerosun": L.lerosun_configuration}[case["design"]]
    tensors = {k: (L.GGML_BF16, tuple(reversed(v.shape)), v.contiguous().reshape(-1).view(torch.uint8).cpu().numpy()) for k, v in w.items()}
    return L.Model(None, configuration(cfg, {k: tuple(v.shape) for k, v in w.items()}, context), case["design"].upper(), tensors)


def _rows(n):
    """The prompt rows whose logits are wanted: the last one and up to three on the way."""
    return sorted({max(0, (n * k) // 4 - 1) for k in (1, 2, 3)} | {n - 1})


# ---- the measured calls -----------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    """What the program holds: the plan with its weights, the tokens, and for a decode step the sequence in the plan's cache."""
    pkg = _package()
    kind = case["kind"]
    length = case["tokens"] if kind.endswith("prompt") else case["position"] + 1
    context = length + 32
    if kind.startswith("gguf"):
        shape, quant, tensors = _gguf(case, seed)
        model = pkg.loader.model_from_tensors(shape, quant, tensors, context)
        del tensors
        # FP16 decode follows the default program, token by token; the others use the batched prefill
        batch = 1 if kind == "gguf_decode" and case["quant"] == "f16" else BATCH
        plan = pkg.B200MasterPlan(model, prefill_batch_size=batch)
        vocab = shape.vocab
    else:
        cfg, w = _layered(case, seed)
        model = _layered_model(case, cfg, w, context)
        del w
        batch = BATCH
        plan = pkg.B200MasterPlan(model, prefill_batch_size=batch, compute=case["compute"])
        vocab = VOCAB
    model.tensors = {}  # the plan keeps its own copy on the device
    tokens = _tokens(vocab, length, seed)
    if kind.endswith("decode"):
        if batch == 1:
            for p in range(length - 1):
                plan.forward_prefill(int(tokens[p]), p)
        else:
            for p in range(0, length - 1, batch):
                plan.forward_batch_prefill(tokens[p:min(p + batch, length - 1)], p)
    return {"kind": kind, "plan": plan, "tokens": tokens, "last": int(tokens[-1]), "rows": _rows(length)}


def run(state):
    plan, tokens, n = state["plan"], state["tokens"], len(state["tokens"])
    if state["kind"] == "layered_prompt":
        return plan.forward_batch_logits(tokens, 0, state["rows"])[0]
    if state["kind"] == "gguf_prompt":
        for p in range(0, n - 1, BATCH):
            plan.forward_batch_prefill(tokens[p:min(p + BATCH, n - 1)], p)
    return plan.forward_decode(state["last"], n - 1)[0]


def work(case):
    kind = case["kind"]
    n = case["tokens"] if kind.endswith("prompt") else 1
    first = 0 if kind.endswith("prompt") else case["position"]
    pairs = sum(first + i + 1 for i in range(n))
    if kind.startswith("gguf"):
        s = _package().synth.SHAPES[case["shape"]]
        per = 34 / 32 if case["quant"] == "q8_0" else 2.0
        cache = 8.0 * s.n_layers * s.kv_dim * (first + n)
        return {"bytes": per * s.matmul_elements() + cache + 4.0 * s.vocab,
                "flops": 2.0 * (n * s.matmul_elements_no_head() + s.vocab * s.dim) + 4.0 * s.n_layers * s.q_dim * pairs}
    rows = len(_rows(n)) if kind.endswith("prompt") else 1
    if case["design"] == "pibidra":
        E, F, H, G, hs, window, layers, loop = PIBIDRA[case["size"]]
        runs = layers + ((loop[1] - loop[0]) * (loop[2] - 1) if loop else 0)
        per_run = (2 * H * hs + 2 * G * hs) * E + H * hs * E + 3 * F * E
        seen = sum(min(first + i + 1, window) for i in range(n))
        stored, used = layers * per_run, runs * per_run
        pair_flops = 4.0 * runs * H * hs * seen
        cache = 8.0 * runs * G * hs * min(first + n, window)
    elif case["design"] == "latusun":
        E, H, dk, dr, dv, R, X, top, F = LATUSUN[case["size"]]
        mixer = H * (dk + dr) * E + (R + dr) * E + H * dv * E + H * dk * R + H * dv * R + E * H * dv + X * E
        stored = mixer + min(X, n * top) * 3 * F * E
        used = mixer + top * 3 * F * E
        pair_flops = 2.0 * H * (dk + dr + dv) * pairs
        cache = 4.0 * (R + dr) * (first + n)
    else:
        E, F, H, G, hs, window, DH, DG, dd, dv, taps = LEROSUN[case["size"]]
        stored = (2 * DG * dd + 2 * DH * dv + 2 * DH) * E + E * DH * dv + (H * hs + G * hs + H) * E + E * H * hs + 6 * F * E
        used = stored
        pair_flops = 4.0 * H * hs * pairs + 6.0 * DH * dd * dv * n
        cache = 8.0 * G * hs * n + 4.0 * DH * dd * dv
    return {"bytes": 2.0 * (stored + VOCAB * E) + cache + 4.0 * rows * VOCAB, "flops": 2.0 * (n * used + rows * VOCAB * E) + pair_flops}


def tolerance(case):
    if case["kind"] == "gguf_decode" or (case["kind"] == "gguf_prompt" and case["quant"] == "q8_0"):
        return "exact"  # the framework's contract: every float in the order of the CPU path
    if case["kind"] == "gguf_prompt":
        return {"rel": 4e-3}  # FP16 operands, FP32 sums (measured: 7e-4 from 64 bits)
    if case["compute"] == "float32":
        return {"rel": 2e-5}
    # BF16 operands in the prefill, FP32 sums; a decode step is FP32 on a cache that the prefill left (measured: 4e-3 and 9e-4 from 64 bits)
    return {"rel": 4e-3 if case["kind"] == "layered_decode" else 2e-2}


# ---- the same results in 64 bits -----------------------------------------------------------------------------------------------------
def _rms(v, eps):
    return v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, heads, kv_heads, bias=None, scale=1.0, cap=None, window=None, sink=None, rows=None):
    """q [T, heads, d], k [T, kv_heads, d], v [T, kv_heads, dv] in one head at a time; ``rows``: only these query rows are needed."""
    T = k.shape[0]
    at = torch.arange(T, device="cuda") if rows is None else rows
    gap = at[:, None] - torch.arange(T, device="cuda")[None, :]
    hidden = (gap < 0) if window is None else (gap < 0) | (gap >= window)
    out = []
    for h in range(heads):
        g = h // (heads // kv_heads)
        e = (q[at, h] @ k[:, g].T) * scale
        if cap is not None:
            e = cap * torch.tanh(e / cap)
        if bias is not None:
            e = e + bias[gap.clamp(min=0), h]
        e = e.masked_fill(hidden, float("-inf"))
        if sink is not None:
            e = torch.cat((e, sink[h].expand(e.shape[0], 1)), 1)
        p = torch.softmax(e, -1)
        out.append(p[:, :T] @ v[:, g])
    return torch.stack(out, 1)


def _rotate(x, positions, freq, pairs="half", magnitude=1.0):
    """x [T, ..., d]; the first 2 * len(freq) entries turn."""
    n = freq.numel()
    a = positions.double()[:, None] * freq[None, :]
    a = a.reshape(a.shape[0], *([1] * (x.dim() - 2)), n)
    cos, sin = torch.cos(a) * magnitude, torch.sin(a) * magnitude
    y = x.clone()
    if pairs == "half":
        u, v = x[..., :n], x[..., n:2 * n]
        y[..., :n], y[..., n:2 * n] = u * cos - v * sin, v * cos + u * sin
    else:
        u, v = x[..., 0:2 * n:2], x[..., 1:2 * n:2]
        y[..., 0:2 * n:2], y[..., 1:2 * n:2] = u * cos - v * sin, v * cos + u * sin
    return y


def _frequencies(base, dims):
    return torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64, device="cuda")


def _gguf_exact(case, seed):
    shape, quant, tensors = _gguf(case, seed)
    q8 = case["quant"] == "q8_0"
    length = case["tokens"] if case["kind"] == "gguf_prompt" else case["position"] + 1
    tokens = torch.from_numpy(_tokens(shape.vocab, length, seed)).long().cuda()

    def get(name):
        kind, dims, raw = tensors[name]
        t = torch.from_numpy(raw).cuda()
        if len(dims) == 1:
            return t.view(torch.float32).double()
        if q8:
            blocks = t.view(-1, 34)
            t = blocks[:, 2:].view(torch.int8).double() * blocks[:, :2].contiguous().view(torch.float16).double()
        else:
            t = t.view(torch.float16).double()
        return t.view(dims[1], dims[0])

    def times(x, *names):
        if q8:  # Q8_0 multiplies quantised activations: blocks of 32 with an FP16 scale
            b = x.reshape(-1, 32)
            d = b.abs().amax(-1, keepdim=True) / 127.0
            s = b * torch.where(d != 0, 1.0 / d, torch.zeros_like(d))
            x = (torch.trunc(s + torch.copysign(torch.full_like(s, 0.5), s)) * d.half().double()).view(x.shape)
        return [x @ get(n).T for n in names]

    T, hs, H, G = length, shape.head_size, shape.n_heads, shape.n_kv_heads
    at = torch.arange(T, device="cuda")
    freq = _frequencies(shape.rope_theta, hs)
    x = get("token_embd.weight")[tokens]
    for i in range(shape.n_layers):
        p = "blk.%d." % i
        a = _rms(x, shape.eps) * get(p + "attn_norm.weight")
        if shape.arch == "phi3":
            q, k, v = times(a, p + "attn_qkv.weight")[0].split((H * hs, G * hs, G * hs), -1)
        else:
            q, k, v = times(a, p + "attn_q.weight", p + "attn_k.weight", p + "attn_v.weight")
        q, k, v = q.reshape(T, H, hs), k.reshape(T, G, hs), v.reshape(T, G, hs)
        if shape.arch == "qwen3":
            q, k = _rms(q, shape.eps) * get(p + "attn_q_norm.weight"), _rms(k, shape.eps) * get(p + "attn_k_norm.weight")
        pairs = "interleaved" if shape.arch == "llama" else "half"
        q, k = _rotate(q, at, freq, pairs), _rotate(k, at, freq, pairs)
        last = i == shape.n_layers - 1  # behind the last layer only the last row is needed
        o = _attend(q, k, v, H, G, scale=hs ** -0.5, rows=at[-1:] if last else None)
        x = x[-1:] if last else x
        x = x + times(o.reshape(x.shape[0], H * hs), p + "attn_output.weight")[0]
        a = _rms(x, shape.eps) * get(p + "ffn_norm.weight")
        if shape.arch == "phi3":
            gate, up = times(a, p + "ffn_up.weight")[0].split(shape.hidden, -1)
        else:
            gate, up = times(a, p + "ffn_gate.weight", p + "ffn_up.weight")
        x = x + times(torch.nn.functional.silu(gate) * up, p + "ffn_down.weight")[0]
    x = _rms(x, shape.eps) * get("output_norm.weight")
    return times(x, "token_embd.weight" if shape.tied else "output.weight")[0][-1]


def _pibidra_exact(cfg, W, tokens):
    eps, T = cfg["norm"]["eps"], len(tokens)

    def norm(v, w):
        return _rms(v, eps) * (1.0 + W(w))

    x = start = W("embed")[tokens] * cfg["embedding"]["scale"]
    n, loop = len(cfg["layers"]), cfg.get("loop")
    runs = [(i, None) for i in range(n)]
    if loop:
        runs = runs[:loop["start"]] + [(i, t if i == loop["start"] else None) for t in range(loop["times"]) for i in range(loop["start"], loop["stop"])] + runs[loop["stop"]:]
    for i, turn in runs:
        if turn is not None:
            x = x + (start if turn > 0 else 0.0) + W("loop.step")[turn]
        m, p = cfg["layers"][i]["mixer"], "l%d." % i
        H, G, dk = m["heads"], m["kv_heads"], m["dim"]
        a = norm(x, p + "norm1")
        q, k, v = (a @ W(p + "mix." + c).T + W(p + "mix." + c + ".b") for c in "qkv")
        q, k = _rms(q, eps) * W(p + "mix.q.norm"), _rms(k, eps) * W(p + "mix.k.norm")
        rel, far = W(p + "mix.rel"), m["bias_max"]
        rows, half = rel.shape[0], rel.shape[0] // 2
        bucket = [d if d < half else min(rows - 1, half + int(math.floor(math.log(d / half) / math.log(far / half) * (rows - half)))) for d in range(T)]
        o = _attend(q.view(T, H, dk), k.view(T, G, dk), v.view(T, G, -1), H, G, bias=rel[torch.tensor(bucket, device="cuda")], scale=m["scale"], cap=m["softcap"],
                    window=m["mask"]["size"], sink=torch.zeros(H, dtype=torch.float64, device="cuda"))
        o = o.reshape(T, -1) * torch.sigmoid(a @ W(p + "mix.g").T)
        x = x + norm(o @ W(p + "mix.o").T, p + "norm1b")
        a = norm(x, p + "norm2")
        f = torch.nn.functional.gelu(a @ W(p + "mlp.gate").T, approximate="tanh") * (a @ W(p + "mlp.up").T)
        x = x + norm(f @ W(p + "mlp.down").T, p + "norm2b")
    return lambda rows: norm(x[rows], "final.norm") @ W("head").T


def _latusun_exact(cfg, W, tokens):
    eps, T = cfg["norm"]["eps"], len(tokens)

    def norm(v, w):
        d = v - v.mean(-1, keepdim=True)
        return _rms(d, eps) * W(w) + W(w + ".b")

    x = W("embed")[tokens]
    at = torch.arange(T, device="cuda")
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], "l%d." % i
        H, dk, dr, dv, R = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        rot, sc = m["rot"], m["rot"]["scaling"]
        dims, base = rot["dims"], rot["base"]

        def turn(t):
            return dims * math.log(sc["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(base))

        low, high = max(math.floor(turn(sc["fast"])), 0), min(math.ceil(turn(sc["slow"])), dims - 1)
        ramp = ((torch.arange(dims // 2, dtype=torch.float64, device="cuda") - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
        f = _frequencies(base, dims)
        f, mag = f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
        a = norm(x, p + "norm1")
        q = (a @ W(p + "mix.q").T).view(T, H, dk + dr)
        q = torch.cat((q[..., :dk], _rotate(q[..., dk:], at, f, magnitude=mag)), -1)
        d = a @ W(p + "mix.dkv").T
        c = _rms(d[:, :R], eps) * W(p + "mix.dkv.norm")
        shared = _rotate(d[:, R:], at, f, magnitude=mag)
        k = torch.cat(((c @ W(p + "mix.uk").T).view(T, H, dk), shared[:, None].expand(T, H, dr)), -1)
        o = _attend(q, k, (c @ W(p + "mix.uv").T).view(T, H, dv), H, H, scale=m["scale"])
        y = (o.reshape(T, -1) * torch.sigmoid(a @ W(p + "mix.g").T)) @ W(p + "mix.o").T
        a = norm(x, p + "norm2")
        scores = torch.sigmoid(a @ W(p + "mlp.router").T)
        best, chosen = scores.topk(layer["mlp"]["router"]["top"], -1)
        for e in range(scores.shape[1]):
            row, slot = torch.nonzero(chosen == e, as_tuple=True)
            if row.numel():
                h = a[row] * best[row, slot][:, None]
                q8 = p + "mlp.e%d." % e
                y[row] += (torch.nn.functional.silu(h @ W(q8 + "gate").T) * (h @ W(q8 + "up").T)) @ W(q8 + "down").T
        x = x + cfg["residual_mult"] * y
    cap = cfg["logit_softcap"]
    return lambda rows: cap * torch.tanh(norm(x[rows], "final.norm") @ W("head").T / cap)


def _lerosun_exact(cfg, W, tokens):
    eps, T = cfg["norm"]["eps"], len(tokens)
    silu = torch.nn.functional.silu

    def norm(v, w):
        return _rms(v, eps) * W(w)

    def conv(u, w):
        taps = w.shape[1]
        padded = torch.cat((u.new_zeros(taps - 1, u.shape[1]), u))
        return silu(sum(w[:, k] * padded[k:k + T] for k in range(taps)))

    x = norm(W("embed")[tokens], "embed.norm")
    at = torch.arange(T, device="cuda")
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], "l%d." % i
        H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        a = norm(x, p + "norm1")
        if layer["type"] == "attention":
            q, k = ((a @ W(p + "mix." + c).T + W(p + "mix." + c + ".b")).view(T, n, d) for c, n in (("q", H), ("k", G)))
            v = k
            f = _frequencies(m["rot"]["base"], m["rot"]["dims"])
            q, k = _rotate(q, at, f), _rotate(k, at, f)
            # scores mixed over the heads are scores of mixed queries against all key heads
            talk = W(p + "mix.talk") * W(p + "mix.temp")[None, :]
            wide = torch.stack([torch.einsum("hm,tmd->thd", talk[:, g * (H // G):(g + 1) * (H // G)], q[:, g * (H // G):(g + 1) * (H // G)]) for g in range(G)], 2)
            o = _attend(wide.reshape(T, H, G * d), k.reshape(T, 1, G * d).expand(T, G, G * d), v, H, G, scale=m["scale"], window=m["mask"]["size"], sink=W(p + "mix.sink"))
            y = (o * torch.sigmoid(a @ W(p + "mix.g").T)[:, :, None]).reshape(T, -1) @ W(p + "mix.o").T
        else:
            q, k, v = (conv(a @ W(p + "mix." + c).T, W(p + "mix." + c + ".conv")) for c in "qkv")
            q, k = (z.view(T, G, d) / torch.sqrt((z.view(T, G, d) ** 2).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
            q, k = (z.repeat_interleave(H // G, 1) for z in (q * d ** -0.5, k))
            v = v.view(T, H, dv)
            beta = torch.sigmoid(a @ W(p + "mix.b").T)
            decay = torch.exp(-torch.exp(W(p + "mix.A_log")) * torch.nn.functional.softplus(a @ W(p + "mix.a").T + W(p + "mix.dt_bias")))
            S, o = a.new_zeros(H, d, dv), []
            for t in range(T):
                S = S * decay[t][:, None, None]
                u = beta[t][:, None] * (v[t] - torch.einsum("hde,hd->he", S, k[t]))
                S = S + k[t][:, :, None] * u[:, None, :]
                o.append(torch.einsum("hde,hd->he", S, q[t]))
            o = _rms(torch.stack(o), eps) * W(p + "mix.norm")
            y = (o.reshape(T, -1) * silu(a @ W(p + "mix.g").T)) @ W(p + "mix.o").T
        x = x + W(p + "ls1") * y
        a = norm(x, p + "norm2")
        x = x + W(p + "ls2") * ((torch.relu(a @ W(p + "mlp.gate").T) * (a @ W(p + "mlp.up").T)) @ W(p + "mlp.down").T)
    return lambda rows: norm(x[rows], "final.norm") @ W("head").T


def exact(case, seed):
    if case["kind"].startswith("gguf"):
        return _gguf_exact(case, seed)
    cfg, w = _layered(case, seed)
    length = case["tokens"] if case["kind"] == "layered_prompt" else case["position"] + 1
    tokens = torch.from_numpy(_tokens(VOCAB, length, seed)).long().cuda()
    logits = {"pibidra": _pibidra_exact, "latusun": _latusun_exact, "lerosun": _lerosun_exact}[case["design"]](cfg, lambda n: w[n].double(), tokens)
    if case["kind"] == "layered_decode":
        return logits([length - 1])[0]
    return logits(_rows(length))
