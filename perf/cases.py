"""What a user's program has this library do, as measurable cases.

Every case is one call pattern on BF16 tensors through the public entry points
(``operations``, ``LCTensor``, ``update_plan``, ``components``):

    roundtrip     compress, decompress and release one tensor (checkpoint and small-parameter traffic)
    compress      compress one tensor, after releasing the value of the pass before
    decompress    decompress one stored tensor
    decode_many   decompress the matrices of a model in one call (loading, weight streaming)
    update        one in-place update of one compressed optimizer state per call
    plan          the prepared in-place update of a list of optimizer states
    apply         dense result of  p + alpha * m  with m compressed (the weight update)
    sgdm          an optimizer step over compressed weights with compressed momentum
    activations   a layer's saved activations: store, compress as a group, load, release

The codec is lossless and its bytes are defined, so every output has to be the same to the bit.
"""
from __future__ import annotations

import math

import torch

from losslessly_compressed_tensors_b200.LCTensor import LCTTensor
from losslessly_compressed_tensors_b200.codec import pointwise
from losslessly_compressed_tensors_b200.codec.geometry import geometry
from losslessly_compressed_tensors_b200.comp_format import Distribution, DistType, NoiseLevel
from losslessly_compressed_tensors_b200.components.activations import ActivationCache
from losslessly_compressed_tensors_b200.components.sparse_utils import SparseSGDM
from losslessly_compressed_tensors_b200.kernels import dispatch
from losslessly_compressed_tensors_b200.operations import (
    a_compA_add_B, compress, decompress, decompress_many,
)
from losslessly_compressed_tensors_b200.tensor_buffer import TensorBuffer
from losslessly_compressed_tensors_b200.update_plan import UpdatePlan

# Codebook and values go together: a codebook is chosen for what a tensor holds.
_CODEBOOKS = {
    "gaussian": lambda: Distribution(DistType.GAUSSIAN),
    "weight": lambda: Distribution(DistType.LAPLACE, param=0.02),
    "activation": lambda: Distribution(DistType.LAPLACE, zero_prob=0.0),
    "relu": lambda: Distribution(DistType.LAPLACE, param=1.0, zero_prob=0.5,
                                 noise_level=NoiseLevel.SPARSE),
    "momentum": lambda: Distribution(DistType.GAUSSIAN, noise_level=NoiseLevel.MEDIUM),
    "noisy": lambda: Distribution(DistType.GAUSSIAN, noise_level=NoiseLevel.HIGH),
    "state": lambda: Distribution(DistType.EMPIRICAL, zero_prob=0.02),
    "model": lambda: Distribution(DistType.EMPIRICAL),
}


def listed() -> list[dict]:
    return [
        # A bias or normalisation vector of a model, through the arena: latency and launches only.
        dict(name="vector_roundtrip", op="roundtrip", values="model", rows=1, cols=2304, arena=True),
        # An ordinary matrix kept in private tensors (no arena): one host synchronisation inside.
        dict(name="matrix_private", op="roundtrip", values="gaussian", rows=1024, cols=1024, arena=False),
        # A large weight with rare outliers: both directions on their own.
        dict(name="weight_compress", op="compress", values="weight", rows=8192, cols=8192, arena=True),
        dict(name="weight_decompress", op="decompress", values="weight", rows=8192, cols=8192, arena=True),
        # Activations behind a ReLU: half zeros, many streams overflow their budget.
        dict(name="relu_compress", op="compress", values="relu", rows=16384, cols=4096, arena=True),
        # ... and read back at a size that fills neither its rows nor its last block.
        dict(name="relu_decompress_ragged", op="decompress", values="relu", rows=3001, cols=1537, arena=True),
        # The matrices of a 12-layer, 768-wide model decoded in one call.
        dict(name="model_decode", op="decode_many", layers=12, width=768, vocab=50304),
        # One momentum matrix advanced by one call: m <- 0.95 m + g.
        dict(name="momentum_update", op="update", values="momentum", rows=4096, cols=4096),
        # All momentum matrices of an optimizer advanced by one prepared call.
        dict(name="momentum_plan", op="plan", values="momentum", rows=4096, cols=4096, count=12, lerp=False),
        # The weight update that reads a compressed momentum.
        dict(name="weight_apply", op="apply", values="state", rows=3072, cols=4096),
        # An optimizer step over the matrices of two layers, weights and momentum compressed.
        dict(name="optimizer_step", op="sgdm", layers=2, width=768),
        # What a transformer layer saves between forward and backward.
        dict(name="layer_activations", op="activations", tokens=8192, width=768),
    ]


def _log_uniform(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _matrix(rng, low: int, high: int) -> dict:
    """A matrix of ``low`` to ``high`` elements; every other draw has sizes that are no multiples
    of anything."""
    numel = _log_uniform(rng, low, high)
    cols = min(numel, _log_uniform(rng, 33, 16384))
    rows = max(1, numel // cols)
    if rng.random() < 0.5:
        rows, cols = (-(-v // 64) * 64 if v > 64 else v for v in (rows, cols))
        while rows > 64 and rows * cols > high:
            rows -= 64
    return dict(rows=rows, cols=cols)


def draw(rng) -> dict:
    op = rng.choice(["roundtrip", "compress", "decompress", "decode_many", "update", "plan", "apply",
                     "sgdm", "activations"])
    if op == "decode_many":
        return dict(op=op, layers=rng.randint(1, 12), width=64 * rng.randint(2, 12),
                    vocab=_log_uniform(rng, 1000, 50304))
    if op == "sgdm":
        return dict(op=op, layers=rng.randint(1, 2), width=32 * rng.randint(4, 40))
    if op == "activations":
        return dict(op=op, tokens=_log_uniform(rng, 512, 8192), width=32 * rng.randint(8, 24))
    if op == "plan":
        return dict(op=op, values=rng.choice(["momentum", "state"]), count=rng.randint(2, 12),
                    lerp=rng.random() < 0.5, **_matrix(rng, 65536, 4096 * 4096))
    if op == "update":
        return dict(op=op, values=rng.choice(["momentum", "state", "gaussian", "noisy"]),
                    **_matrix(rng, 2048, 8192 * 4096))
    if op == "apply":
        return dict(op=op, values=rng.choice(["momentum", "state"]), **_matrix(rng, 2048, 8192 * 4096))
    return dict(op=op, values=rng.choice(["gaussian", "weight", "activation", "relu", "momentum",
                                          "noisy", "state", "model"]),
                arena=op == "compress" or rng.random() < 0.6, **_matrix(rng, 1024, 8192 * 8192))


def _values(kind: str, shape, generator, scale: float = 1.0) -> torch.Tensor:
    if kind in ("weight", "state"):
        u = torch.rand(shape, device="cuda", generator=generator).sub_(0.5)
        x = u.sign().mul_(u.abs_().mul_(-2.0).log1p_()).mul_(-0.02 if kind == "weight" else -1e-3)
        if kind == "weight":
            outliers = torch.rand(shape, device="cuda", generator=generator) < 1e-4
            x = torch.where(outliers, x * 100.0, x)
    else:
        x = torch.randn(shape, device="cuda", generator=generator)
        if kind == "relu":
            x.relu_()
        elif kind == "momentum":
            x.mul_(1e-3)
        elif kind == "model":
            x.mul_(0.02)
    return (x if scale == 1.0 else x.mul_(scale)).to(torch.bfloat16)


def _buffer(elements: int) -> TensorBuffer:
    return TensorBuffer(((1 << 20) + elements // 4) // 16 * 16)


def _layer_shapes(layers: int, width: int):
    return [s for _ in range(layers) for s in ((width, 3 * width), (width, width),
                                               (width, 4 * width), (4 * width, width))]


def _model_shapes(case):
    width = case["width"]
    return [(case["vocab"], width), (1024, width)] + _layer_shapes(case["layers"], width)


def _activation_columns(width: int):
    return (width, width, 3 * width, width, width, 4 * width, 4 * width)


def _scalar(value: float) -> torch.Tensor:
    return torch.tensor([value], dtype=torch.float32, device="cuda")


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda").manual_seed(seed)
    op = case["op"]
    state: dict = {"op": op}
    if op == "decode_many":
        shapes, dist = _model_shapes(case), _CODEBOOKS["model"]()
        state["buffer"] = _buffer(sum(r * c for r, c in shapes))
        state["items"] = [compress(_values("model", s, gen), dist, state["buffer"]) for s in shapes]
        return state
    if op == "sgdm":
        shapes = _layer_shapes(case["layers"], case["width"])
        buffer = state["buffer"] = _buffer(8 * sum(r * c for r, c in shapes))
        params = [LCTTensor(_values("weight", s, gen), buffer, _CODEBOOKS["weight"]()) for s in shapes]
        state["optimizer"] = SparseSGDM(params, lr=1e-4, momentum=0.9, buffer=buffer, compressed=True)
        for p, s in zip(params, shapes):
            p.grad = _values("state", s, gen)
        state["params"] = params
        state["optimizer"].step()      # the first step makes the momentums from the gradients
        return state
    if op == "activations":
        tokens, width = case["tokens"], case["width"]

        def normal(cols):
            return torch.randn(tokens, cols, device="cuda", generator=gen)

        x, attention, fc = normal(width), normal(width) * 0.5, normal(4 * width)
        ln1 = torch.nn.functional.layer_norm(x, (width,))
        ln2 = torch.nn.functional.layer_norm(x + attention, (width,))
        saved = (x, ln1, normal(3 * width), attention, ln2, fc, torch.nn.functional.gelu(fc))
        state["saved"] = [t.to(torch.bfloat16) for t in saved]
        state["buffer"] = _buffer(15 * tokens * width)
        state["cache"] = ActivationCache(state["buffer"], _CODEBOOKS["activation"](), batch=0)
        return state
    shape, dist = (case["rows"], case["cols"]), _CODEBOOKS[case["values"]]()
    numel = shape[0] * shape[1]
    if op == "plan":
        count, lerp = case["count"], case["lerp"]
        buffer = state["buffer"] = _buffer(2 * count * numel)
        state["states"] = [LCTTensor(_values(case["values"], shape, gen), buffer, dist) for _ in range(count)]
        state["grads"] = [_values(case["values"], shape, gen) for _ in range(count)]
        if lerp:       # momentum average and look-ahead direction, written beside the gradients
            state["outs"] = [torch.empty_like(g) for g in state["grads"]]
            state["plan"] = UpdatePlan(state["states"], _scalar(0.05), _scalar(0.95),
                                       operation=pointwise.LERP, emit=dispatch.EMIT_NESTEROV)
        else:
            state["plan"] = UpdatePlan(state["states"], _scalar(0.95))
        return state
    if op == "update":
        state["buffer"] = _buffer(2 * numel)
        state["state"] = LCTTensor(_values(case["values"], shape, gen), state["buffer"], dist)
        state["grad"] = _values(case["values"], shape, gen)
        state["alpha"] = _scalar(0.95)
        return state
    if op == "apply":
        state["buffer"] = _buffer(numel)
        state["momentum"] = compress(_values(case["values"], shape, gen), dist, state["buffer"])
        state["weight"] = _values("weight", shape, gen)
        state["alpha"] = _scalar(-0.1)
        return state
    state["buffer"] = _buffer(numel) if case["arena"] else None
    state["dist"] = dist
    x = _values(case["values"], shape, gen)
    if op == "decompress":
        state["item"] = compress(x, dist, state["buffer"])
    else:
        state["x"], state["held"] = x, None
    return state


def _parts(c) -> list:
    """What a compressed tensor stores, but for its overflow tails: those are in the shared arena,
    or in private tensors whose sizes depend on the data (the decoded tensor shows them)."""
    parts = [c.data, c.sign_mantissa, c.center, c.decode_table, c.fallback_count, c.fallback_used,
             c.fallback_blocks]
    return parts if c.fallback_descriptor is None else parts + [c.fallback_descriptor]


def run(state: dict):
    op = state["op"]
    if op == "roundtrip":
        c = compress(state["x"], state["dist"], state["buffer"])
        dense = decompress(c)
        out = [dense, *_parts(c)]
        c.free()
        return out
    if op == "compress":
        if state["held"] is not None:
            state["held"].free()
        c = state["held"] = compress(state["x"], state["dist"], state["buffer"])
        return _parts(c) + [state["buffer"].data]
    if op == "decompress":
        return decompress(state["item"])
    if op == "decode_many":
        return decompress_many(state["items"])
    if op == "update":
        state["state"].mul_add_(state["alpha"], state["grad"])
        return _parts(state["state"].x) + [state["buffer"].data]
    if op == "plan":
        state["plan"].step(state["grads"], state.get("outs"))
        values = [t.x for t in state["states"]]
        return {"payload": [v.data for v in values], "side": [v.sign_mantissa for v in values],
                "center": [v.center for v in values], "dense": state.get("outs", []),
                "arena": state["buffer"].data}
    if op == "apply":
        return a_compA_add_B(state["momentum"], state["alpha"], state["weight"])
    if op == "sgdm":
        state["optimizer"].step()
        values = [p.x for p in state["params"]] + [m.x for m in state["optimizer"].momentums]
        return {"payload": [v.data for v in values], "side": [v.sign_mantissa for v in values],
                "center": [v.center for v in values], "arena": state["buffer"].data}
    cache = state["cache"]
    handles = [cache.store(t) for t in state["saved"]]
    cache.flush()
    return [h.load() for h in handles]


def _stored(numel: int, dist: Distribution) -> int:
    """Bytes of the compressed form without overflow tails: side bytes and payload words."""
    block_symbols, lanes, _, fixed_words = geometry(dist)
    blocks = -(-numel // block_symbols)
    return blocks * (block_symbols + 4 * lanes * fixed_words)


def work(case: dict) -> dict:
    """Bytes a pass has to read and write: dense tensors at two bytes, compressed ones as stored."""
    op = case["op"]
    if op == "decode_many":
        dist = _CODEBOOKS["model"]()
        return {"bytes": sum(2 * r * c + _stored(r * c, dist) for r, c in _model_shapes(case)), "flops": 0}
    if op == "sgdm":
        weight = _CODEBOOKS["weight"]()
        shapes = _layer_shapes(case["layers"], case["width"])
        # momentum and weight are each read and written once, the gradient is read
        return {"bytes": sum(2 * r * c + 4 * _stored(r * c, weight) for r, c in shapes), "flops": 0}
    if op == "activations":
        dist = _CODEBOOKS["activation"]()
        numels = [case["tokens"] * c for c in _activation_columns(case["width"])]
        return {"bytes": sum(4 * n + 2 * _stored(n, dist) for n in numels), "flops": 0}
    numel = case["rows"] * case["cols"]
    stored = _stored(numel, _CODEBOOKS[case["values"]]())
    if op == "plan":
        return {"bytes": case["count"] * (2 * stored + (4 if case["lerp"] else 2) * numel), "flops": 0}
    total = {"roundtrip": 4 * numel + 2 * stored, "update": 2 * numel + 2 * stored,
             "apply": 4 * numel + stored}.get(op, 2 * numel + stored)
    return {"bytes": total, "flops": 0}


def tolerance(case: dict):
    return "exact"
