"""The work that a host of this library has it do, as cases for timing: one EXL3 linear, a decode step of
transformer layers, the lm_head with its token drawn, a prefill chunk of a layer, and the mixture-of-experts layer.

Everything runs through the public callers (``berth_b200.engine``, ``berth_b200.kernels``, ``berth_b200.moe``).
Weights, scratch and outputs are made once, as a model loads them; a pass is what the host does per token or chunk.
A model's layers follow one another with weights that are not in the L2 cache, so a state whose one layer is small
holds several layers with weights of their own.

Values follow the benchmark's distributions: trellis words uniform, sign-scales a random sign times N(1, 0.05) with
1/sqrt(fan in) on the output side (as trained scales carry it), activations N(0, 1) with 0.1 % outliers of 20 times
that in prefill, router weights N(0, 0.02).
"""
from __future__ import annotations

import math

import torch

from berth_b200 import kernels, moe
from berth_b200.engine import Exl3Linear, Gpu, MlpLayer, RowScratch, SlicedMultiLinear
from berth_b200.kernels import Codebook, OutDtype, ops

INST3, MCG, MUL1 = 0, 1, 2


def listed() -> list:
    dense = {"hidden": 5120, "inter": 17408, "q": 6144, "kv": 1024}       # the 27B-shaped layer
    a3b = {"kind": "moe", "hidden": 2048, "inter": 512, "experts": 256, "top_k": 8, "bits": 4, "cb": MUL1, "skew": False}
    return [
        # one projection called on its own, the smallest call: launch and latency count
        {"name": "linear m1", "kind": "linear", "rows": 1, "k": 5120, "n": 6144, "bits": 4, "cb": MUL1, "layers": 8},
        # one user's decode, a token at a time
        {"name": "decode m1", "kind": "decode", "rows": 1, "bits": 4, "cb": MUL1, "layers": 2, **dense},
        # the same from a checkpoint in the MCG codebook
        {"name": "decode m1 mcg", "kind": "decode", "rows": 1, "bits": 4, "cb": MCG, "layers": 2, **dense},
        # a draft of three tokens verified at once
        {"name": "decode m3", "kind": "decode", "rows": 3, "bits": 4, "cb": MUL1, "layers": 2, **dense},
        # small and larger decode batches
        {"name": "decode m8", "kind": "decode", "rows": 8, "bits": 4, "cb": MUL1, "layers": 2, **dense},
        {"name": "decode m32", "kind": "decode", "rows": 32, "bits": 4, "cb": MUL1, "layers": 2, **dense},
        # logits of the vocabulary and the token drawn from them
        {"name": "lm_head m1", "kind": "lm_head", "rows": 1, "hidden": 5120, "vocab": 248320, "bits": 6, "cb": MUL1, "gumbel": True},
        # a short prompt's only chunk, of no round length, and a long prompt's full chunk (mixed 3/4/5 bits)
        {"name": "prefill 421", "kind": "prefill", "rows": 421, "bits": 4, "cb": MUL1, **dense},
        {"name": "prefill 4096", "kind": "prefill", "rows": 4096, "bits": 4, "cb": MUL1, **dense},
        # the A3B layer for one user, for a decode batch, and for a prefill chunk
        {"name": "moe 1", "tokens": 1, "layers": 8, **a3b},
        {"name": "moe 64", "tokens": 64, "layers": 2, **a3b},
        {"name": "moe 1024", "tokens": 1024, "layers": 1, **a3b},
    ]


def _log(rng, lo: float, hi: float, step: int = 1) -> int:
    """A multiple of ``step`` between lo and hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(int(lo), min(int(hi), int(round(v / step)) * step))


def _codebook(rng) -> int:
    return rng.choice([MUL1, MUL1, MUL1, MCG, INST3])


def _layers(nbytes: float, most: int) -> int:
    """As many layers as keep the weights of three states out of the L2 cache."""
    return max(1, min(most, math.ceil(100e6 / nbytes)))


def draw(rng) -> dict:
    """Sizes from those of a small dense model up to the 27B-shaped layer, multiples of the 128-wide rotation (256
    where several projections share a launch), 3 to 6 bits, all three codebooks."""
    kind = rng.choice(["linear", "decode", "decode", "decode", "lm_head", "prefill", "prefill", "moe", "moe", "moe"])
    if kind == "linear":
        k, n = _log(rng, 1024, 17408, 128), _log(rng, 1024, 17408, 128)
        bits = rng.choice([3, 4, 4, 5, 6])
        return {"kind": kind, "rows": _log(rng, 1, 32), "k": k, "n": n, "bits": bits, "cb": _codebook(rng),
                "layers": _layers(k * n * bits / 8, 16)}
    if kind == "lm_head":
        return {"kind": kind, "rows": _log(rng, 1, 32), "hidden": 128 * rng.randint(16, 40), "vocab": _log(rng, 32000, 248320, 256),
                "bits": rng.choice([4, 6, 6]), "cb": _codebook(rng), "gumbel": rng.random() < 0.5}
    if kind == "moe":
        tokens = _log(rng, 1, 4096)
        return {"kind": kind, "tokens": tokens, "hidden": 2048, "inter": rng.choice([512, 768]), "experts": rng.choice([128, 256]),
                "top_k": 8, "bits": rng.choice([3, 4, 4]), "cb": MUL1, "skew": rng.random() < 0.5,
                "layers": 8 if tokens <= 8 else 2 if tokens <= 128 else 1}
    hidden = 128 * rng.randint(16, 40)
    dims = {"hidden": hidden, "inter": 128 * int(hidden * rng.uniform(2.5, 3.4) / 128), "q": 256 * rng.randint(hidden // 256, hidden * 6 // 1280),
            "kv": 256 * rng.randint(1, 4)}
    if kind == "decode":
        bits = rng.choice([3, 4, 4, 4, 5])
        return {"kind": kind, "rows": _log(rng, 1, 32), "bits": bits, "cb": _codebook(rng),
                "layers": 1 + _layers(3.5 * hidden * dims["inter"] * bits / 8, 3), **dims}
    return {"kind": kind, "rows": _log(rng, 33, 4096), "bits": 4, "cb": _codebook(rng), **dims}


# ------------------------------------------------------------------ inputs

class Source:
    """Seeded tensors made on the GPU."""

    def __init__(self, seed: int):
        self.device = torch.device("cuda", torch.cuda.current_device())
        self.g = torch.Generator(device=self.device)
        self.g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 12345)

    def words(self, *shape) -> torch.Tensor:
        n = math.prod(shape)
        t = torch.randint(-2 ** 31, 2 ** 31, (n // 2,), dtype=torch.int32, device=self.device, generator=self.g)
        return t.view(torch.int16).view(*shape)

    def word(self) -> int:
        return int(torch.randint(0, 2 ** 31, (1,), device=self.device, generator=self.g))

    def normal(self, *shape, scale: float = 1.0, mean: float = 0.0) -> torch.Tensor:
        return torch.randn(*shape, device=self.device, generator=self.g) * scale + mean

    def sign_scale(self, *shape, gain: float = 1.0) -> torch.Tensor:
        sign = torch.randint(0, 2, shape, device=self.device, generator=self.g) * 2 - 1
        return (sign * self.normal(*shape, scale=0.05, mean=1.0) * gain).half()

    def activations(self, *shape, outliers: bool = False) -> torch.Tensor:
        x = self.normal(*shape)
        if outliers:
            x = torch.where(torch.rand(*shape, device=self.device, generator=self.g) < 0.001, x * 20.0, x)
        return x

    def linear(self, gpu: Gpu, name: str, k: int, n: int, bits: int, cb: int, rows: int) -> Exl3Linear:
        return Exl3Linear(gpu, name, self.words(k // 16, n // 16, 16 * bits), self.sign_scale(k), self.sign_scale(n, gain=k ** -0.5),
                          bits, Codebook(cb), max_rows=rows)


def prepare(case: dict, seed: int) -> dict:
    s = Source(seed)
    make = {"linear": _prepare_linear, "decode": _prepare_decode, "lm_head": _prepare_lm_head, "prefill": _prepare_prefill,
            "moe": _prepare_moe}[case["kind"]]
    return {"kind": case["kind"], **make(case, s)}


def run(state: dict):
    return {"linear": _run_linear, "decode": _run_decode, "lm_head": _run_lm_head, "prefill": _run_prefill, "moe": _run_moe}[state["kind"]](state)


# ------------------------------------------------------------------ one linear

def _prepare_linear(c, s):
    gpu = Gpu(s.device.index)
    f16 = torch.float16
    return {"gpu": gpu, "rows": c["rows"],
            "lin": [s.linear(gpu, f"layers.{i}.proj", c["k"], c["n"], c["bits"], c["cb"], c["rows"]) for i in range(c["layers"])],
            "x": s.activations(c["rows"], c["k"]).half(),
            "y": [torch.empty((c["rows"], c["n"]), dtype=f16, device=s.device) for _ in range(c["layers"])]}


def _run_linear(st):
    for lin, y in zip(st["lin"], st["y"]):
        lin.forward_n(st["gpu"], st["rows"], st["x"], y, OutDtype.F16)
    return st["y"]


# ------------------------------------------------------------------ a decode step

EPS, NORM_BIAS = 1e-6, 1.0      # the norms' weights are stored around zero


def _norm(s, dim):
    return s.normal(dim, scale=0.05).bfloat16()


def _prepare_decode(c, s):
    """The residual stream through ``layers`` layers: norm, q/k/v, o, norm, MLP.  Attention itself is the host's; q
    stands in for its output, so that o has an input of the real shape and scale."""
    gpu = Gpu(s.device.index)
    h, rows, bits, cb = c["hidden"], c["rows"], c["bits"], c["cb"]
    layers = []
    for i in range(c["layers"]):
        mk = lambda name, k, n: s.linear(gpu, f"layers.{i}.{name}", k, n, bits, cb, rows)
        mlp = MlpLayer(gpu, mk("gate_proj", h, c["inter"]), mk("up_proj", h, c["inter"]), mk("down_proj", c["inter"], h), max_rows=rows)
        qkv = SlicedMultiLinear(gpu, [mk("q_proj", h, c["q"]), mk("k_proj", h, c["kv"]), mk("v_proj", h, c["kv"])], OutDtype.F16, max_rows=rows)
        layers.append({"mlp": mlp, "qkv": qkv, "o": mk("o_proj", c["q"], h), "norm1": _norm(s, h), "norm2": _norm(s, h)})
    f32 = lambda: torch.zeros((rows, h), dtype=torch.float32, device=s.device)
    return {"gpu": gpu, "rows": rows, "hidden": h, "layers": layers, "embedding": s.activations(rows, h), "residual": f32(),
            "x": torch.empty((rows, h), dtype=torch.float16, device=s.device), "o": f32(), "mlp": f32()}


def _run_decode(st):
    gpu, rows, h, x, res = st["gpu"], st["rows"], st["hidden"], st["x"], st["residual"]
    stream = gpu.raw_stream()
    res.copy_(st["embedding"])
    for i, layer in enumerate(st["layers"]):
        if i == 0:
            ops.rms_norm(res, layer["norm1"], x, rows, h, EPS, NORM_BIAS, 1.0, True, stream)
        else:
            ops.rms_norm_res_in(st["mlp"], layer["norm1"], x, res, rows, h, EPS, NORM_BIAS, 1.0, True, stream)
        q, _, _ = layer["qkv"].forward_n(gpu, rows, x)
        layer["o"].forward_n(gpu, rows, q, st["o"], OutDtype.F32)
        ops.rms_norm_res_in(st["o"], layer["norm2"], x, res, rows, h, EPS, NORM_BIAS, 1.0, True, stream)
        layer["mlp"].forward_n(gpu, rows, x, st["mlp"])
    return {"residual": res, "mlp": st["mlp"], "qkv": [layer["qkv"].outputs for layer in st["layers"]]}


# ------------------------------------------------------------------ lm_head

def _prepare_lm_head(c, s):
    gpu = Gpu(s.device.index)
    rows = c["rows"]
    lin = s.linear(gpu, "lm_head", c["hidden"], c["vocab"], c["bits"], c["cb"], rows)
    return {"gpu": gpu, "rows": rows, "lin": lin, "mode": 1 if c["gumbel"] else 0, "random": s.word(),
            "x": s.activations(rows, c["hidden"]).half(), "best": torch.zeros(rows, dtype=torch.int64, device=s.device),
            "logits": torch.empty((rows, c["vocab"]), dtype=torch.float32, device=s.device)}


def _run_lm_head(st):
    lin = st["lin"]
    kernels.exl3_linear_sample(st["x"], lin.trellis, st["logits"], lin.suh, lin.a_had, lin.svh, st["best"], st["rows"], lin.size_k, lin.size_n,
                               lin.k_bits, lin.codebook, OutDtype.F32, 1.25, st["random"], st["mode"], st["gpu"].raw_stream())
    # a key's low word is the token (complemented), its high word the score; the host splits it when it reads it back
    return {"logits": st["logits"], "token": st["best"].view(torch.int32).view(-1, 2)[:, 0]}


# ------------------------------------------------------------------ a prefill chunk

def _prefill_bits(c):
    """Mixed rates as quantizers allot them: down a bit more than the rest, k and v a bit less."""
    return {"gate": c["bits"], "up": c["bits"], "down": c["bits"] + 1, "q": c["bits"], "k": c["bits"] - 1, "v": c["bits"] - 1, "o": c["bits"]}


def _prepare_prefill(c, s):
    gpu = Gpu(s.device.index)
    h, rows, b, cb = c["hidden"], c["rows"], _prefill_bits(c), c["cb"]
    mk = lambda name, k, n: s.linear(gpu, f"layers.0.{name}_proj", k, n, b[name], cb, 1)
    mlp = MlpLayer(gpu, mk("gate", h, c["inter"]), mk("up", h, c["inter"]), mk("down", c["inter"], h), max_rows=rows)
    e = lambda n, dt: torch.empty((rows, n), dtype=dt, device=s.device)
    return {"gpu": gpu, "rows": rows, "hidden": h, "mlp": mlp, "qkv": [mk("q", h, c["q"]), mk("k", h, c["kv"]), mk("v", h, c["kv"])],
            "o_proj": mk("o", c["q"], h), "norm1": _norm(s, h), "norm2": _norm(s, h), "embedding": s.activations(rows, h, outliers=True),
            "residual": e(h, torch.float32), "x": e(h, torch.float16), "o": e(h, torch.float32), "out": e(h, torch.float32),
            "outputs": [e(n, torch.float16) for n in (c["q"], c["kv"], c["kv"])],
            "scratch": RowScratch(gpu, rows, max(h, c["inter"], c["q"]), max(h, c["inter"], c["q"]))}


def _run_prefill(st):
    gpu, rows, h, x, res, sc = st["gpu"], st["rows"], st["hidden"], st["x"], st["residual"], st["scratch"]
    stream = gpu.raw_stream()
    res.copy_(st["embedding"])
    ops.rms_norm(res, st["norm1"], x, rows, h, EPS, NORM_BIAS, 1.0, True, stream)
    for lin, y in zip(st["qkv"], st["outputs"]):
        lin.forward_rows(gpu, rows, x, y, OutDtype.F16, sc)
    st["o_proj"].forward_rows(gpu, rows, st["outputs"][0], st["o"], OutDtype.F32, sc)
    ops.rms_norm_res_in(st["o"], st["norm2"], x, res, rows, h, EPS, NORM_BIAS, 1.0, True, stream)
    st["mlp"].prefill(gpu, rows, x, st["out"], sc)
    return {"residual": res, "out": st["out"], "qkv": st["outputs"]}


# ------------------------------------------------------------------ mixture of experts

def _prepare_moe(c, s):
    """``layers`` layers with expert stacks and inputs of their own (chained layers would let one rounding difference
    choose another expert further on)."""
    h, i, e, b, t = c["hidden"], c["inter"], c["experts"], c["bits"], c["tokens"]
    layers = []
    for _ in range(c["layers"]):
        w = {"hidden": h, "inter": i, "shared_inter": i, "n_experts": e, "top_k": c["top_k"], "bits": b, "cb": c["cb"],
             "w_router": s.normal(h, e, scale=0.02).half(), "router_bias": None}
        if c["skew"]:       # popularity falls off as rank^-1.1
            rank = torch.randperm(e, device=s.device, generator=s.g) + 1
            w["router_bias"] = (-1.1 * torch.log(rank.float())).contiguous()
        for name, k, n in (("gate", h, i), ("up", h, i), ("down", i, h)):
            w[f"{name}_trellis"], w[f"{name}_suh"], w[f"{name}_svh"] = s.words(e, k // 16, n // 16, 16 * b), s.sign_scale(e, k), s.sign_scale(e, n, gain=k ** -0.5)
            w[f"sh_{name}_trellis"], w[f"sh_{name}_suh"], w[f"sh_{name}_svh"] = s.words(k // 16, n // 16, 16 * b), s.sign_scale(k), s.sign_scale(n, gain=k ** -0.5)
        layer = moe.MoeLayer(s.device, w, t)
        layers.append({"layer": layer, "x": s.activations(t, h).half(), "out": torch.empty((t, h), dtype=torch.float32, device=s.device),
                       "idx": torch.empty((t, c["top_k"]), dtype=torch.int32, device=s.device),
                       "w": torch.empty((t, c["top_k"]), dtype=torch.float32, device=s.device)})
        del w
    return {"layers": layers}


def _run_moe(st):
    for l in st["layers"]:
        l["layer"].forward(l["x"], l["out"], l["idx"], l["w"])
    return [(l["out"], l["idx"], l["w"]) for l in st["layers"]]


# ------------------------------------------------------------------ the work of a pass

def _linear_work(rows, k, n, bits, out_bytes=2):
    """Trellis, sign-scales and rows read, outputs written; a multiply and an add per weight and row."""
    return k * n * bits / 8 + 2 * (k + n) + rows * (2 * k + out_bytes * n), 2.0 * rows * k * n


def work(case: dict) -> dict:
    c, kind = case, case["kind"]
    if kind == "linear":
        parts = [_linear_work(c["rows"], c["k"], c["n"], c["bits"])] * c["layers"]
    elif kind == "lm_head":
        parts = [_linear_work(c["rows"], c["hidden"], c["vocab"], c["bits"], 4)]
    elif kind in ("decode", "prefill"):
        h, r = c["hidden"], c["rows"]
        b = _prefill_bits(c) if kind == "prefill" else dict.fromkeys(("gate", "up", "down", "q", "k", "v", "o"), c["bits"])
        shapes = {"gate": (h, c["inter"]), "up": (h, c["inter"]), "down": (c["inter"], h), "q": (h, c["q"]), "k": (h, c["kv"]), "v": (h, c["kv"]),
                  "o": (c["q"], h)}
        # weights and scales once, the residual stream in and out, q/k/v out (the cache takes k and v); what lies
        # between two of the layer's own steps need not leave the chip
        per = [k * n * b[name] / 8 + 2 * (k + n) for name, (k, n) in shapes.items()]
        flops = sum(2.0 * r * k * n for k, n in shapes.values())
        parts = [(sum(per) + 4 * h + r * 2 * (c["q"] + 2 * c["kv"]), flops)] * c.get("layers", 1) + [(r * h * 12, 0)]
    else:
        t, h, i, e = c["tokens"], c["hidden"], c["inter"], c["experts"]
        hit = e * (1 - (1 - c["top_k"] / e) ** t) if not c["skew"] else min(e, c["top_k"] * t, e * (1 - (1 - c["top_k"] / e) ** (0.6 * t)) + c["top_k"])
        weights = (hit + 1) * (3 * h * i * c["bits"] / 8 + 6 * (h + i)) + 2 * h * e
        parts = [(weights + t * (2 * h + 4 * h + 8 * c["top_k"]), t * (2.0 * h * e + (c["top_k"] + 1) * 6.0 * h * i))] * c["layers"]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case: dict):
    """Activations between steps are fp16 (2.8e-4 of a value's magnitude per rounding), and a decoded weight is an
    fp16 value or the same value unrounded: about 5e-4 per linear, four linears deep in each layer."""
    if case["kind"] in ("linear", "lm_head"):
        return {"rel": 1e-3, "max": 0.02}
    if case["kind"] == "moe":
        return {"rel": 2e-3, "max": 0.04}
    return {"rel": 5e-3, "max": 0.1}
