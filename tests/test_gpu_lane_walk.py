"""The walk of the bit streams at the edges of its chunks (16 rows of 256 columns), of a row, of a
block, and where lanes overflow: bit-exact against the input and the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_helpers import assert_same_components, bits_of, to_dev
from helpers import oracle_compress
from losslessly_compressed_tensors_b200 import config
from losslessly_compressed_tensors_b200.LCTensor import LCTTensor
from losslessly_compressed_tensors_b200.codec import pointwise
from losslessly_compressed_tensors_b200.codec.decode import operand_of
from losslessly_compressed_tensors_b200.codec.geometry import geometry
from losslessly_compressed_tensors_b200.comp_format import Distribution, DistType, NoiseLevel
from losslessly_compressed_tensors_b200.compression.huffman_tables import get_distribution_tables
from losslessly_compressed_tensors_b200.kernels import dispatch
from losslessly_compressed_tensors_b200.operations import (
    a_compA_add_B, a_compA_add_compB, compress, decompress, decompress_many,
)
from losslessly_compressed_tensors_b200.tensor_buffer import TensorBuffer
from losslessly_compressed_tensors_b200.update_plan import UpdatePlan
from synth import synth_bf16

pytestmark = pytest.mark.gpu

CHUNK = 16 * 256
SIZES = [1, 2, 255, 257, 511, CHUNK - 1, CHUNK, CHUNK + 1, 3 * CHUNK + 257, 32768 - 1, 32768 + 1,
         65536 + 7 * CHUNK + 513]
CODEBOOKS = {
    "short": Distribution(DistType.GAUSSIAN),                                    # 128 steps
    "long": Distribution(DistType.LAPLACE, zero_prob=0.0),                       # 256 steps
    "loose": Distribution(DistType.GAUSSIAN, noise_level=NoiseLevel.HIGH),       # budget never met
}


KINDS = ["normal", "outliers", "wide", "staggered"]


def values(n, seed, kind, base_exponent=0):
    """``staggered``: every lane holds codable values up to a row of its own and incompressible
    ones behind it, so the lanes of a warp leave their streams all over the block, and their tails
    start at every alignment."""
    if kind != "staggered":
        return synth_bf16(n, seed, kind, base_exponent)
    row, column = np.divmod(np.arange(n), 256)
    lane = column ^ (row & 254)
    wide = row % 128 >= (lane * 37 + seed) % 128
    return np.where(wide, synth_bf16(n, seed, "wide"), synth_bf16(n, seed, "normal", base_exponent))


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("codebook", sorted(CODEBOOKS))
@pytest.mark.parametrize("kind", KINDS)
def test_walk(oracle, n, codebook, kind):
    dist = CODEBOOKS[codebook]
    bits, right, third = values(n, 5, kind), synth_bf16(n + 1, 6, "normal", -2), values(n, 7, kind)
    buffer = TensorBuffer(1 << 20)
    a, b = compress(to_dev(bits), dist, buffer), compress(to_dev(third), dist, buffer)
    assert np.array_equal(bits_of(decompress(a)), bits)
    for got, want in zip(decompress_many([b, a]), (third, bits)):
        assert np.array_equal(bits_of(got), want)
    want_a = oracle_compress(oracle, bits, dist, oracle.new_arena(1 << 20))
    assert_same_components(a, want_a)
    alpha = torch.tensor([0.95], dtype=torch.float32, device="cuda")
    wide = to_dev(right)
    for offset in (0, 1):  # the dense operand at 16 and at 2 bytes alignment
        result = a_compA_add_B(a, alpha, wide[offset:offset + n])
        expect = oracle.pointwise(want_a, right[offset:offset + n], oracle.OP_SCALED, 0.95,
                                  alpha_is_one=False)
        assert np.array_equal(bits_of(result).view(np.uint16), expect)
    dual = a_compA_add_compB(a, alpha, b)
    expect = oracle.pointwise(want_a, third, oracle.OP_SCALED, 0.95, alpha_is_one=False)
    assert np.array_equal(bits_of(dual).view(np.uint16), expect)


@pytest.mark.parametrize("n", [CHUNK + 1, 65536 + 7 * CHUNK + 513])
@pytest.mark.parametrize("op", ["LERP", "EMA_SQUARE"])
@pytest.mark.parametrize("offset", [0, 1])  # the dense operand at 16 and at 2 bytes alignment
def test_averages_of_one_compressed_operand(oracle, n, op, offset):
    """The two operations that the functional interface reaches through updates only, with dense
    and with compressed results."""
    dist, alpha, beta = CODEBOOKS["short"], 0.25, 0.125
    bits, wide = values(n, 5, "staggered"), synth_bf16(n + 1, 6, "normal", -2)
    right, other = wide[offset:offset + n], to_dev(wide)[offset:offset + n]
    a = compress(to_dev(bits), dist, TensorBuffer(1 << 20))
    want_a = oracle_compress(oracle, bits, dist, oracle.new_arena(1 << 20))
    scalars = [torch.tensor([v], dtype=torch.float32, device="cuda") for v in (alpha, beta)]
    block_symbols, lanes, steps, fixed_words = geometry(dist)
    _, _, rare_length = get_distribution_tables(dist, a.data.device)
    for dense in (True, False):
        out = torch.empty(n if dense else a.size, dtype=torch.bfloat16 if dense else torch.uint8, device="cuda")
        exponents = torch.zeros(a.size, dtype=torch.uint8, device="cuda")
        dispatch.pointwise_dense(operand_of(a), other, out, exponents, a.size, *scalars,
                                 op=getattr(dispatch, "OP_" + op), alpha_is_one=False,
                                 beta_is_one=False, compressed_output=not dense, logical_numel=n,
                                 block_symbols=block_symbols, lanes=lanes, steps=steps,
                                 fixed_words=fixed_words, rare_length=rare_length)
        want = oracle.pointwise(want_a, right, getattr(oracle, "OP_" + op), alpha, beta,
                                alpha_is_one=False, beta_is_one=False, dense=dense)
        if dense:
            assert np.array_equal(bits_of(out).view(np.uint16), want)
        else:
            assert np.array_equal(out.cpu().numpy(), want[0])
            assert np.array_equal(exponents[:n].cpu().numpy(), want[1][:n])


def test_storage_with_more_than_2_31_elements_of_padding():
    """Blocks of pure padding write nothing, also where their distance from the end of the tensor
    does not fit 32 bits."""
    n, guard, dist = 1000, 4096, CODEBOOKS["short"]
    block_symbols, lanes, steps, fixed_words = geometry(dist)
    blocks = (1 << 31) // block_symbols + 2
    size = blocks * block_symbols
    bits = synth_bf16(n, 11, "normal")
    one = compress(to_dev(bits), dist, TensorBuffer(1 << 20))
    encoded = torch.zeros(fixed_words * blocks * lanes + 4, dtype=torch.int32, device="cuda")
    encoded[:-4].view(fixed_words, blocks * lanes)[:, :lanes] = one.data[:-4].view(fixed_words, lanes)
    side = torch.zeros(size, dtype=torch.uint8, device="cuda")
    side[:block_symbols] = one.sign_mantissa
    operand = dispatch.make_operand(encoded, side, one.decode_table, one.center,
                                    dispatch.pair_table_for(dist, encoded.device),
                                    dispatch.fallback_tail_args(None))
    _, _, rare_length = get_distribution_tables(dist, encoded.device)
    shape = dict(logical_numel=n, block_symbols=block_symbols, lanes=lanes, steps=steps,
                 fixed_words=fixed_words, rare_length=rare_length)
    out = torch.full((n + guard,), 77, dtype=torch.int16, device="cuda")
    dispatch.decode_kernel(operand, out, size, **shape)
    assert np.array_equal(out[:n].cpu().numpy(), bits) and bool((out[n:] == 77).all())
    zeros = torch.zeros(n, dtype=torch.bfloat16, device="cuda")
    out = torch.full((n + guard,), 77, dtype=torch.int16, device="cuda")
    dispatch.pointwise_dense(operand, zeros, out, None, size, None, None, op=pointwise.ADD.code,
                             alpha_is_one=True, beta_is_one=True, compressed_output=False, **shape)
    assert np.array_equal(out[:n].cpu().numpy(), bits) and bool((out[n:] == 77).all())


@pytest.fixture(params=["swizzle", "linear"])
def lane_mapping(request, monkeypatch):
    monkeypatch.setattr(config, "lane_mapping", request.param)
    yield request.param
    monkeypatch.undo()
    # hand the default mapping back to the library before any other test launches
    x = torch.zeros(256, dtype=torch.bfloat16, device="cuda")
    assert torch.equal(decompress(compress(x, CODEBOOKS["short"])), x)


NONE, RESULT, NESTEROV = dispatch.EMIT_NONE, dispatch.EMIT_RESULT, dispatch.EMIT_NESTEROV
# name: operation, its arguments, by-product
FORMS = {
    "scaled": (pointwise.SCALAR_MUL_ADD, dict(alpha=0.95), NONE),
    "both scaled": (pointwise.SCALAR_MUL_ADD, dict(alpha=0.95, beta=0.3), RESULT),
    "sum": (pointwise.SCALAR_MUL_ADD, dict(alpha=7.0, alpha_is_one=True), NONE),
    "right scaled": (pointwise.SCALAR_MUL_ADD, dict(alpha=7.0, beta=0.3, alpha_is_one=True), NONE),
    "add": (pointwise.ADD, dict(alpha=7.0), NONE),
    "multiply": (pointwise.MULTIPLY, dict(alpha=7.0), RESULT),
    "lerp": (pointwise.LERP, dict(alpha=0.05), RESULT),
    "lerp, direction": (pointwise.LERP, dict(alpha=0.05, beta=0.95), NESTEROV),
    "average of squares": (pointwise.EMA_SQUARE, dict(alpha=0.95, beta=0.05), RESULT),
}


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("codebook", ["short", "long"])
@pytest.mark.parametrize("offset", [0, 1])
def test_batched_update_forms_equal_single_updates(lane_mapping, form, codebook, offset):
    """Every arithmetic form and by-product of the batched update, in both lane mappings, against
    the single update: same payload, same result, same by-product (written over the update itself
    where that is aligned)."""
    operation, arguments, emit = FORMS[form]
    arguments = {k: torch.tensor([v], dtype=torch.float32, device="cuda") if isinstance(v, float) else v
                 for k, v in arguments.items()}
    dist, sizes = CODEBOOKS[codebook], SIZES[2:]
    buffer, reference = TensorBuffer(1 << 22), TensorBuffer(1 << 22)
    bits = [values(n, 20 + i, "staggered") for i, n in enumerate(sizes)]
    together = [LCTTensor(to_dev(b), buffer, dist) for b in bits]
    alone = [LCTTensor(to_dev(b), reference, dist) for b in bits]
    plan = UpdatePlan(together, operation=operation, emit=emit, **arguments)
    for step in range(2):
        wide = [to_dev(values(n + 1, 40 + 20 * step + i, "staggered", step - 1)) for i, n in enumerate(sizes)]
        grads = [w[offset:offset + n] for w, n in zip(wide, sizes)]
        expected = [torch.zeros(n, dtype=torch.bfloat16, device="cuda") for n in sizes]
        for b, g, out in zip(alone, grads, expected):
            new = pointwise.recycled_update(b.x, g, operation, emit=emit,
                                            dense_out=out if emit != NONE else None, **arguments)
            assert new is not None
            b.x = new
        outs = grads if offset == 0 else [torch.zeros_like(out) for out in expected]
        plan.step(grads, outs if emit != NONE else None)
        for a, b, out, want in zip(together, alone, outs, expected):
            for part in ("data", "sign_mantissa", "center", "fallback_count"):
                assert torch.equal(getattr(a.x, part), getattr(b.x, part)), (part, out.numel(), step)
            assert torch.equal(decompress(a.x).view(torch.int16), decompress(b.x).view(torch.int16))
            if emit != NONE:
                assert torch.equal(out.view(torch.int16), want.view(torch.int16)), (out.numel(), step)


@pytest.mark.parametrize("codebook", sorted(CODEBOOKS))
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("offset", [0, 1])
def test_batched_update_equals_single_updates(codebook, kind, offset):
    """The batched update walks lanes, the single one works on tiles: same payload, same result."""
    dist = CODEBOOKS[codebook]
    alpha = torch.tensor([0.95], dtype=torch.float32, device="cuda")
    buffer, reference = TensorBuffer(1 << 22), TensorBuffer(1 << 22)
    bits = [values(n, 20 + i, kind) for i, n in enumerate(SIZES)]
    together = [LCTTensor(to_dev(b), buffer, dist) for b in bits]
    alone = [LCTTensor(to_dev(b), reference, dist) for b in bits]
    plan = UpdatePlan(together, alpha)
    for step in range(3):
        grads = [to_dev(values(n + 1, 40 + 20 * step + i, kind, step - 1))[offset:offset + n]
                 for i, n in enumerate(SIZES)]
        plan.step(grads)
        for a, b, g in zip(together, alone, grads):
            b.mul_add_(alpha, g)
            for part in ("data", "sign_mantissa", "center", "fallback_count"):
                assert torch.equal(getattr(a.x, part), getattr(b.x, part)), (part, g.numel(), step)
            assert torch.equal(decompress(a.x).view(torch.int16), decompress(b.x).view(torch.int16))
