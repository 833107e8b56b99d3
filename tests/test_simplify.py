"""Graph rewrites of simplify.clean against the interpreter: a rewritten graph gives the same bits."""

import numpy as np
import pytest

from lumen_b200 import prims, tracer
from lumen_b200.simplify import clean
from tests.helpers import bf16, run_oracle


def ops(g):
    return [n.op for n in g.nodes]


def same_bits(g, inputs):
    cleaned = clean(g)
    for a, b in zip(run_oracle(g, inputs), run_oracle(cleaned, inputs), strict=True):
        assert a.dtype == b.dtype and a.shape == b.shape
        assert np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))
    return cleaned


def normal(*shape, seed=0):
    return bf16(np.random.default_rng(seed).standard_normal(shape))


MATRICES = (((1,), (0,)), ((), ()))
BOTH_LAST = (((1,), (1,)), ((), ()))


@pytest.mark.parametrize("dims,rhs", [(MATRICES, (24, 8)), (BOTH_LAST, (8, 24))])
@pytest.mark.parametrize("after", ["output", "cast", "add"])
def test_the_transpose_of_a_16_bit_product_is_the_swapped_product(dims, rhs, after):
    def program(a, b):
        t = prims.transpose(prims.dot_general(a, b, dims, "float32", "float32" if after == "cast" else "bfloat16"), (1, 0))
        return t.to("bfloat16") if after == "cast" else t + t if after == "add" else t

    g = tracer.trace(program, ("bfloat16", (16, 24)), ("bfloat16", rhs))
    assert "transpose" not in ops(same_bits(g, [normal(16, 24), normal(*rhs, seed=1)]))


def test_a_product_read_twice_or_of_float32_keeps_its_transpose():
    def twice(a, b):
        y = prims.dot_general(a, b, MATRICES, "float32", "bfloat16")
        return y, prims.transpose(y, (1, 0))

    g = tracer.trace(twice, ("bfloat16", (16, 24)), ("bfloat16", (24, 8)))
    assert ops(same_bits(g, [normal(16, 24), normal(24, 8, seed=1)])).count("dot_general") == 1
    f = tracer.trace(lambda a, b: prims.transpose(prims.dot_general(a, b, MATRICES, "float32"), (1, 0)), ("float32", (16, 24)), ("float32", (24, 8)))
    rng = np.random.default_rng(0)
    assert "transpose" in ops(same_bits(f, [rng.standard_normal((16, 24), dtype=np.float32), rng.standard_normal((24, 8), dtype=np.float32)]))


@pytest.mark.parametrize("lhs,rhs,dims", [
    ((3, 5, 24), (24,), (((2,), (0,)), ((), ()))),          # both free axes on one side
    ((24,), (24, 3, 5), (((0,), (0,)), ((), ()))),
    ((3, 5, 24), (3, 24), (((2,), (1,)), ((0,), (0,)))),    # a batch axis
    ((3, 5, 24), (3, 5, 24), (((2,), (2,)), ((0, 1), (0, 1)))),
    ((4, 6, 3), (6, 4, 5), (((0, 1), (1, 0)), ((), ()))),   # several contracted axes
])
def test_products_that_are_not_of_two_matrices_keep_their_transpose(lhs, rhs, dims):
    """Swapping the operands of a product transposes its result only where each side gives one of the two axes."""
    g = tracer.trace(lambda a, b: prims.transpose(prims.dot_general(a, b, dims, "float32", "bfloat16"), (1, 0)), ("bfloat16", lhs), ("bfloat16", rhs))
    same_bits(g, [normal(*lhs), normal(*rhs, seed=1)])
