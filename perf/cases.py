"""Performance cases of the W4A4 path: the calls a program makes of this package, from one decoded token to a 70B-shaped
layer and a whole prefill, each through its public entry point.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` makes what a program holds
before the call (activations, packed weights, a module or a model), ``run`` is one call, ``work`` the bytes and operations
that call cannot do without, ``tolerance`` how far two correct implementations of the same precision may be apart and
``exact`` what plain torch gives for the same inputs in 64 bits.

Kinds:
  layer     ``linear_forward(use_hadamard=True)``, no workspaces: the functional form of the W4A4 linear
  plain     the same without the Hadamard transform
  module    ``Linear4bit`` with a bias on a 3-D input
  prefill   the decoder body with every linear replaced and the quantisers fused into their producers
  prepare   ``preprocess_weight``: a bf16 weight into packed int4 codes, scales and offsets
  quantise  ``hadamard_quantize_int4`` alone, as in front of several layers that share their input
"""
from __future__ import annotations

import math

import torch

import quest_b200 as quest
from quest_b200.prefill import Decoder, DecoderConfig, swap_linears

DEV = "cuda"


# ------------------------------------------------------------------------------------------------ cases
def listed() -> list[dict]:
    return [
        # one sequence decoding: a 7B attention projection for a single token; launches and host time are the cost
        {"name": "decode_1", "kind": "layer", "m": 1, "k": 4096, "n": 4096, "dist": "student"},
        # a batch of 16 sequences decoding: the 7B gate / up projection, bound by the stream over the packed weights
        {"name": "decode_16", "kind": "layer", "m": 16, "k": 4096, "n": 11008, "dist": "student"},
        # a short prompt or a large decoding batch through the fused QKV projection
        {"name": "chunk_128", "kind": "layer", "m": 128, "k": 4096, "n": 12288, "dist": "student"},
        # three ragged prompts of 111 tokens through the module (bias, 3-D input): gate / up of the 800M model
        {"name": "module_333", "kind": "module", "m": 333, "k": 2048, "n": 5632, "dist": "student"},
        # a program that trained without the transform: 512 tokens, square projection
        {"name": "plain_512", "kind": "plain", "m": 512, "k": 4096, "n": 4096, "dist": "randn"},
        # an odd number of tokens through the 7B down projection (K = 11008 is 86 blocks of 128)
        {"name": "down_1000", "kind": "layer", "m": 1000, "k": 11008, "n": 4096, "dist": "student"},
        # the layer the benchmark reports
        {"name": "layer_2048", "kind": "layer", "m": 2048, "k": 4096, "n": 4096, "dist": "student"},
        # the largest call of the 7B sweep
        {"name": "layer_8192", "kind": "layer", "m": 8192, "k": 4096, "n": 12288, "dist": "student"},
        # the longest reduction: 70B down projection
        {"name": "down_70b", "kind": "layer", "m": 2048, "k": 28672, "n": 8192, "dist": "randn"},
        # four blocks of the 800M decoder on 16 prompts of 1024 tokens
        {"name": "prefill_16x1024", "kind": "prefill", "batch": 16, "seq": 1024, "layers": 4},
        # loading a model: one 7B gate / up weight
        {"name": "prepare_weight", "kind": "prepare", "k": 4096, "n": 11008},
        # the large end of the quantiser's bandwidth sweep, channel outliers included
        {"name": "quantise_65536", "kind": "quantise", "m": 65536, "k": 4096, "block": 128, "dist": "laplace"},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# (K, N) of the layers the repository's configurations and tests name: 800M, 7B and 70B shapes and their column shards
_SHAPES = [(2048, 2048), (2048, 6144), (2048, 5632), (5632, 2048), (4096, 4096), (4096, 12288), (4096, 11008), (4096, 22016),
           (11008, 4096), (8192, 10240), (8192, 28672), (8192, 3584), (8192, 1280), (28672, 8192), (28672, 1024)]
_MOST_MKN = 2048 * 28672 * 8192  # down_70b


def draw(rng) -> dict:
    kind = rng.choices(["layer", "plain", "module", "prefill", "prepare", "quantise"], [8, 2, 2, 1, 1, 2])[0]
    if kind == "prefill":
        return {"kind": kind, "batch": rng.randint(1, 16), "seq": rng.randint(16, 128) * 8 - rng.choice([0, 0, 1, 3]), "layers": rng.randint(1, 4)}
    if kind == "prepare":
        return {"kind": kind, "k": 128 * _log_int(rng, 4, 224), "n": _log_int(rng, 256, 8192)}
    if kind == "quantise":
        k = rng.choice([2048, 4096, 5632, 8192, 11008, 14336, 128 * rng.randint(8, 64)])
        block = rng.choice([64, 128, 256]) if k % 256 == 0 else 128
        return {"kind": kind, "m": _log_int(rng, 1, 65536 * 4096 // k), "k": k, "block": block, "dist": rng.choice(["laplace", "student", "randn"])}
    if rng.random() < 0.7:
        k, n = rng.choice(_SHAPES)
    else:  # a shape no configuration names: any number of blocks, any number of columns
        k, n = 128 * rng.randint(4, 96), rng.randint(200, 12000)
    m = _log_int(rng, 1, min(16384, _MOST_MKN // (k * n)))
    case = {"kind": kind, "m": m, "k": k, "n": n, "dist": rng.choice(["student", "randn", "outlier"])}
    return case


# ------------------------------------------------------------------------------------------------ inputs
def _activations(dist: str, m: int, k: int, g) -> torch.Tensor:
    """bf16 [m, k] with the distributions of the repository's tests, made on the GPU."""
    def randn(*s):
        return torch.randn(*s, generator=g, device=DEV)

    if dist == "randn":
        return randn(m, k).to(torch.bfloat16)
    if dist == "outlier":  # 0.5 % of the entries twenty times larger
        x = randn(m, k)
        return torch.where(torch.rand(m, k, generator=g, device=DEV) < 0.005, x * 20, x).to(torch.bfloat16)
    if dist == "student":  # Student-t with four degrees of freedom, unit RMS
        x, chi = randn(m, k), torch.zeros(m, k, device=DEV)
        for _ in range(4):
            chi += randn(m, k).square_()
        x /= (chi / 4).sqrt_()
        return (x / x.square().mean().sqrt()).to(torch.bfloat16)
    if dist == "laplace":  # Laplace(0, 1), 1 % of the columns fifty times larger
        u = torch.rand(m, k, generator=g, device=DEV) - 0.5
        x = (-u.sign() * torch.log1p(-2 * u.abs() * (1 - 1e-7))).to(torch.bfloat16)
        cols = torch.randperm(k, generator=g, device=DEV)[: max(1, k // 100)]
        x[:, cols] *= 50
        return x
    raise ValueError(dist)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    if kind == "prefill":
        cfg = DecoderConfig(n_layer=case["layers"], sequence_length=1024)
        with torch.random.fork_rng(devices=[torch.cuda.current_device()]):
            torch.manual_seed(seed)
            with torch.device(DEV):
                model = Decoder(cfg).to(torch.bfloat16).eval()
        swap_linears(model, "int4_fused", use_hadamard=True)
        idx = torch.randint(0, cfg.vocab_size, (case["batch"], case["seq"]), generator=g, device=DEV)
        return {"kind": kind, "model": model, "idx": idx}
    if kind == "quantise":
        return {"kind": kind, "x": _activations(case["dist"], case["m"], case["k"], g), "block": case["block"]}
    w = (0.02 * torch.randn(case["n"], case["k"], generator=g, device=DEV)).to(torch.bfloat16)
    if kind == "prepare":
        return {"kind": kind, "w": w}
    x = _activations(case["dist"], case["m"], case["k"], g)
    if kind == "module":
        lin = quest.Linear4bit(case["k"], case["n"], bias=True, device=DEV, dtype=torch.bfloat16, use_hadamard=True, weight=w)
        lin.bias.data.copy_(0.1 * torch.randn(case["n"], generator=g, device=DEV))
        rows = 3 if case["m"] % 3 == 0 else 1
        return {"kind": kind, "lin": lin.eval(), "x": x.view(rows, case["m"] // rows, case["k"])}
    wp, ws, wa, _ = quest.preprocess_weight(w, use_hadamard=kind == "layer")
    return {"kind": kind, "x": x, "wp": wp, "ws": ws, "wa": wa}


# ------------------------------------------------------------------------------------------------ the call
@torch.inference_mode()
def run(state: dict):
    kind = state["kind"]
    if kind in ("layer", "plain"):
        return quest.linear_forward(state["x"], state["wp"], state["ws"], state["wa"], use_hadamard=kind == "layer")
    if kind == "module":
        return state["lin"](state["x"])
    if kind == "prefill":
        return state["model"](state["idx"])
    if kind == "prepare":
        return quest.preprocess_weight(state["w"], use_hadamard=True)[:3]
    return quest.hadamard_quantize_int4(state["x"], state["block"])


# ------------------------------------------------------------------------------------------------ what it cannot do without
def work(case: dict) -> dict:
    """Each input read once, each output written once; multiply-adds of the contractions count two operations."""
    kind = case["kind"]
    if kind == "prefill":
        d, f, t = 2048, 5632, case["batch"] * case["seq"]
        weights = case["layers"] * (4 * d * d + 3 * d * f)
        attention = 2 * 2 * case["batch"] * case["seq"] * case["seq"] * d * case["layers"] / 2  # causal
        return {"bytes": 8 * t + 2 * t * d + weights / 2 + 2 * t * d, "flops": 2 * t * weights + attention}
    k = case["k"]
    if kind == "quantise":
        m = case["m"]
        return {"bytes": 2.5 * m * k + 6 * m, "flops": m * k * math.log2(case["block"])}
    n = case["n"]
    if kind == "prepare":
        return {"bytes": 2.5 * n * k + 6 * n, "flops": n * k * 7}
    m = case["m"]
    return {"bytes": 2 * m * k + n * k / 2 + 6 * n + 2 * m * n + (2 * n if kind == "module" else 0), "flops": 2 * m * n * k}


def tolerance(case: dict):
    """Against the same path with the transform and every sum in float64 (three seeds each, same bf16 rounding points):

    layer, plain, module   most seeds reproduce every bf16 output; where a transform output rounds the other way and moves a
                           code, or the scale of a row, the 2-norm moves by up to 2.1e-3 and a single value by up to 0.14
    prepare                no byte, scale or offset differs
    quantise               3.6e-7 of the packed bytes, 7.3e-4 of the row sums (one code in a row moves its sum), no scale

    Each is stated about four times as large.  The prefill is chaotic: an output of a block that rounds the other way moves
    int4 codes of the next one, and after four blocks two correct implementations (quantisers fused or not, another
    attention kernel) are 0.2 to 0.35 apart.  What is stated there holds for an implementation that reproduces the
    blocks' roundings and differs in the last norm at most."""
    kind = case["kind"]
    if kind == "prepare":
        return {"rel": 1e-4, "max": 1e-2, "differ": 1e-6}
    if kind == "quantise":
        return {"rel": 1e-3, "max": 1e-2, "differ": 3e-3}
    if kind == "prefill":
        return {"rel": 3e-2}
    return {"rel": 1e-2, "max": 0.5}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _transform64(x: torch.Tensor, block: int, scale: float) -> torch.Tensor:
    """The block transform of bf16 rows with sums in float64, rounded once to bf16 (a rounding point of the format)."""
    h = x.double().view(x.size(0), -1, block)
    half = 1
    while half < block:
        h = h.view(x.size(0), -1, 2, half)
        h = torch.stack((h[:, :, 0] + h[:, :, 1], h[:, :, 0] - h[:, :, 1]), dim=2)
        half *= 2
    return (h.reshape(x.shape) * scale).to(torch.bfloat16)


def _codes64(x: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    """(codes as float64 [rows, K], scale in float64 [rows, 1]); the codes are taken with the scale rounded to bf16."""
    x = x.double()
    s = x.square().mean(dim=1, keepdim=True).sqrt() * (2.513930578568423 * 2 / 15) + 1e-8
    return (x / s.to(torch.bfloat16).double()).floor().clamp(-8, 7), s


def _pack(codes: torch.Tensor) -> torch.Tensor:
    c = codes.to(torch.int16).bitwise_and_(15).to(torch.uint8)
    return c[:, ::2] | (c[:, 1::2] << 4)


@torch.inference_mode()
def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "prefill":
        return None
    g = torch.Generator(device=DEV).manual_seed(seed)
    if kind == "quantise":
        x = _activations(case["dist"], case["m"], case["k"], g)
        packed, scale, sums = [], [], []
        act = torch.tensor(case["block"] ** -0.5).to(torch.bfloat16).item()
        for rows in x.split(8192):
            q, s = _codes64(_transform64(rows, case["block"], act))
            packed.append(_pack(q)), scale.append(s), sums.append(q.sum(dim=1, keepdim=True).to(torch.int32))
        return torch.cat(packed), torch.cat(scale), torch.cat(sums)
    w = (0.02 * torch.randn(case["n"], case["k"], generator=g, device=DEV)).to(torch.bfloat16)
    x = None if kind == "prepare" else _activations(case["dist"], case["m"], case["k"], g)
    bias = 0.1 * torch.randn(case["n"], generator=g, device=DEV) if kind == "module" else None
    if kind != "plain":  # weights carry the fp32 constant, activations its bf16 rounding
        w = _transform64(w, 128, torch.tensor(128.0).rsqrt().item())
        x = None if x is None else _transform64(x, 128, torch.tensor(128.0).rsqrt().to(torch.bfloat16).item())
    qw, sw = _codes64(w)
    del w
    if kind == "prepare":
        return _pack(qw), sw, (qw.sum(dim=1, keepdim=True) + case["k"] // 2).to(torch.int32)
    qa, sa = _codes64(x)
    sa, sw = sa.to(torch.bfloat16).double(), sw.to(torch.bfloat16).double()
    y = torch.empty(case["m"], case["n"], dtype=torch.float64, device=DEV)
    for i in range(0, case["n"], 4096):  # (a + 1/2) . (w + 1/2) is what the offsets of the integer path add up to
        y[:, i:i + 4096] = (qa + 0.5) @ (qw[i:i + 4096] + 0.5).T
    y *= sa
    y *= sw.T
    if bias is not None:
        rows = 3 if case["m"] % 3 == 0 else 1
        y = (y + bias.to(torch.bfloat16)).view(rows, case["m"] // rows, case["n"])
    return y
