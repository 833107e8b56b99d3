"""The fusion pass on graphs of bare prims: what it groups, and that grouping changes no value (the oracle evaluates
fusion bodies primitive by primitive, so the fused graph must give bit-identical results)."""

import numpy as np
import pytest

from lumen_b200 import functional as F
from lumen_b200 import prims, tracer
from lumen_b200.compiler import compile_graph
from lumen_b200.fusion_pass import fuse
from tests.helpers import bf16, run_oracle


def fusions(g):
    return [n for n in g.nodes if n.op == "fusion"]


def bare(g):
    return [n.op for n in g.nodes if n.op not in ("fusion", "fusion_output", "reshape", "slice", "dot_general", "concatenate")]


def same_values(g, fused, inputs):
    want, got = run_oracle(g, inputs), run_oracle(fused, inputs)
    assert len(want) == len(got)
    for a, b in zip(want, got):
        assert a.dtype == b.dtype and a.shape == b.shape
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))


def test_chain_with_a_row_sum_becomes_one_fusion():
    def chain(x, gg, b):
        y = F.relu(x * gg + b)
        return y, prims.reduce_sum(y * y, (1,), "float32")

    g = tracer.trace(chain, ("float32", (64, 256)), ("float32", (256,)), ("float32", (256,)))
    fused = fuse(g)
    assert len(fusions(fused)) == 1 and not bare(fused)
    f = fusions(fused)[0]
    assert f.params["name"] == "row" and len(f.params["body"].outputs) == 2  # y and the row sums: a multi-output fusion
    rng = np.random.default_rng(0)
    same_values(g, fused, [rng.standard_normal((64, 256), dtype=np.float32), rng.standard_normal(256, dtype=np.float32),
                           rng.standard_normal(256, dtype=np.float32)])
    assert compile_graph(g).labels == ["row"]


def test_softmax_row_is_one_fusion_and_a_reduction_keeps_its_epilogue():
    def program(x, w):
        p = F.softmax(x, -1)  # two reductions over the row and the elementwise work between and after them
        s = F.sum(p * w, -1) * 0.5  # a reduction with a prologue and an epilogue
        return p, s

    g = tracer.trace(program, ("float32", (32, 128)), ("float32", (32, 128)))
    fused = fuse(g)
    assert not bare(fused)
    assert len(fusions(fused)) <= 2
    rng = np.random.default_rng(1)
    same_values(g, fused, [rng.standard_normal((32, 128), dtype=np.float32), rng.standard_normal((32, 128), dtype=np.float32)])


def test_small_column_and_row_reductions_do_not_share_a_kernel():
    def program(x):
        return F.sum(x, 0), F.sum(x, 1)

    g = tracer.trace(program, ("float32", (128, 64)))
    fused = fuse(g)
    assert len(fusions(fused)) == 2 and not bare(fused)
    same_values(g, fused, [np.random.default_rng(2).standard_normal((128, 64), dtype=np.float32)])


def test_small_norms_and_their_column_sums_share_a_kernel():
    """Two row sums and more, which the column sums' operands depend on: one kernel whatever the size."""
    def program(x, g):
        c = x - prims.reduce_sum(x, (1,), "float32").reshape(24, 1) * (1.0 / 832)
        r = prims.rsqrt(prims.reduce_sum(c * c, (1,), "float32").reshape(24, 1) * (1.0 / 832) + 1e-5)
        return c * r, prims.reduce_sum(c * r * g, (0,), "float32"), prims.reduce_sum(g, (0,), "float32")

    g = tracer.trace(program, ("float32", (24, 832)), ("float32", (24, 832)))
    fused = fuse(g)
    assert len(fusions(fused)) == 1 and not bare(fused)
    rng = np.random.default_rng(5)
    same_values(g, fused, [rng.standard_normal((24, 832), dtype=np.float32) for _ in range(2)])


def test_gemm_takes_its_elementwise_tail_as_an_epilogue():
    dims = (((1,), (0,)), ((), ()))

    def program(a, w, r, u):
        y = prims.dot_general(a, w, dims, "float32", "bfloat16")
        z = F.relu(prims.dot_general(y + r, w, dims, "float32", "bfloat16"))  # y + r feeds only this product's operand
        m = F.where(F.gt(u, 0), prims.dot_general(z, w, dims, "float32", "bfloat16"), 0)
        return m

    t = ("bfloat16", (128, 128))
    g = tracer.trace(program, t, t, t, t)
    fused = fuse(g)
    names = [f.params["name"] for f in fusions(fused)]
    assert names.count("dot_general") == 3 and not bare(fused)
    labels = compile_graph(g).labels
    assert labels == ["dot_general_add", "dot_general_relu", "dot_general_relu_backward"]
    rng = np.random.default_rng(3)
    same_values(g, fused, [bf16(rng.standard_normal((128, 128)) / 12) for _ in range(4)])


def test_traced_fusions_pass_through_and_constants_of_unfusible_readers_stay_plain():
    from lumen_b200 import transformer as T

    cfg = T.Config(vocab=32, d_model=32, heads=2, hidden=64, layers=1, seq=16, dtype="float32")
    g, _, _ = T.trace_train_step(cfg, 2)
    fused = fuse(g)
    assert [n.op for n in fused.nodes] == [n.op for n in g.nodes]


@pytest.mark.parametrize("shape", [(1000003,), (3, 300007), (2, 2, 600014), (4, 1000000), (4096, 1536), (131072,)])
def test_long_reductions_are_split_without_changing_their_values(shape):
    """`simplify.split_long_reductions` (the last step of `clean`): sums and maxima over more elements than one block
    takes as a row - whole tensors and rows, lengths with and without useful divisors (1,000,003 and 300,007 are prime,
    600,014 is twice a prime) - evaluated by the oracle before and after the pass: maxima equal, sums within the
    rounding of a float32 sum; a reduction that fits one block is left as it is."""
    from lumen_b200.simplify import LONGEST_ROW, clean

    whole = len(shape) == 1 or shape == (4096, 1536)

    def program(x):
        return (F.sum(x), F.amax(x * x)) if whole else (F.sum(x, -1), F.amax(x * x, -1))

    g = tracer.trace(program, ("float32", shape))
    cleaned = clean(g)
    x = np.random.default_rng(len(shape)).standard_normal(shape).astype(np.float32)
    before, after = run_oracle(g, [x]), run_oracle(cleaned, [x])
    row = shape[-1] if not whole else int(np.prod(shape))
    assert (sum(n.op in ("reduce_sum", "reduce_max") for n in cleaned.nodes) > 2) == (row > LONGEST_ROW)
    exact = x.astype(np.float64).sum() if whole else x.astype(np.float64).sum(-1)
    magnitude = np.abs(x.astype(np.float64)).sum() if whole else np.abs(x.astype(np.float64)).sum(-1)
    assert after[0].shape == before[0].shape and after[1].shape == before[1].shape
    assert (np.abs(after[0] - exact) <= 1e-6 * magnitude).all()
    np.testing.assert_array_equal(after[1], before[1])


@pytest.mark.parametrize("count,dtype,beside", [(6, "float32", False), (7, "float32", False), (16, "float32", False), (4, "float64", False), (7, "bfloat16", False),
                                                (8, "float32", True), (5, "float64", True)])
def test_any_number_of_column_reductions_of_one_operand_compiles(count, dtype, beside):
    """Statistics per feature (column sums of `count` functions of one operand), alone and beside a row-wise output: the
    groups that read the operand are merged, and every kernel of the result is built (generation alone does not see limits
    of the hardware such as 48 KB of static shared memory)."""
    from lumen_b200.runtime import Fusion

    accum = "float64" if dtype == "float64" else "float32"

    def program(x):
        powers = [x]
        for _ in range(count - 1):
            powers.append(powers[-1] * x)
        sums = tuple(prims.reduce_sum(p, (0,), accum) for p in powers)
        return (F.relu(x), *sums) if beside else sums

    rows = 8192 if not beside else 70000  # narrow rows beside: several to a block, whose sums meet in shared memory
    g = tracer.trace(program, (dtype, (rows, 1024 if not beside else 64)))
    fused = fuse(g)
    assert not bare(fused)
    for f in fusions(fused):
        Fusion(f.params["body"])


def row_and_column_sums(x):
    return F.sum(x, 0), F.sum(x, 1)


def relu_and_column_sums(x):
    return F.relu(x), prims.reduce_sum(x, (0,), "float32")


def norm_gradients(x, dy):
    w, g = x.to("float32"), dy.to("float32")
    m = F.sum(w, 1, keepdim=True) * (1.0 / x.shape[1])
    r = F.rsqrt(F.sum((w - m) * (w - m), 1, keepdim=True) * (1.0 / x.shape[1]))
    h = (w - m) * r
    dx = r * (g - F.sum(g, 1, keepdim=True) * (1.0 / x.shape[1]) - h * (F.sum(g * h, 1, keepdim=True) * (1.0 / x.shape[1])))
    return dx.to(x.dtype), F.sum(g * h, 0).to(x.dtype), F.sum(g, 0).to(x.dtype)


@pytest.mark.parametrize("program,dtype,shape,together", [
    (relu_and_column_sums, "float32", (4096, 4096), True),
    (relu_and_column_sums, "float32", (256, 16384), False),   # 9 us apart, 13 together
    (relu_and_column_sums, "float32", (2048, 16384), True),   # 68 and 52
    (relu_and_column_sums, "float32", (256, 40000), False),   # 15 and 31
    (relu_and_column_sums, "bfloat16", (256, 1024), True),
    (relu_and_column_sums, "bfloat16", (1024, 1024), False),  # 5.6 and 7.9
    (relu_and_column_sums, "bfloat16", (256, 40000), False),  # 11 and 39
    (relu_and_column_sums, "bfloat16", (8192, 8192), True),   # 70 and 56: larger than the L2
    (relu_and_column_sums, "bfloat16", (4096, 3001), True),   # 18 and 14
    (norm_gradients, "float32", (8192, 1024), True),
    (norm_gradients, "float32", (256, 32768), False),         # 167 and 187 (with its forward)
    (norm_gradients, "bfloat16", (8192, 1024), True),
    (norm_gradients, "bfloat16", (256, 16384), False),        # 49 and 61
    (norm_gradients, "bfloat16", (1024, 16384), True),        # 166 and 124
])
def test_rows_and_columns_share_a_kernel_where_that_is_faster(program, dtype, shape, together):
    from lumen_b200.runtime import Fusion

    g = tracer.trace(program, *[(dtype, shape)] * program.__code__.co_argcount)
    fused = fuse(g)
    assert (len(fusions(fused)) == 1) == together and not bare(fused)
    for f in fusions(fused):
        Fusion(f.params["body"])


@pytest.mark.parametrize("program", [row_and_column_sums, relu_and_column_sums, norm_gradients])
def test_groups_joined_by_an_operand_give_the_same_values(program):
    g = tracer.trace(program, *[("float32", (300, 260))] * program.__code__.co_argcount)
    fused = fuse(g)
    assert len(fusions(fused)) == 1
    rng = np.random.default_rng(7)
    same_values(g, fused, [rng.standard_normal((300, 260), dtype=np.float32) for _ in range(program.__code__.co_argcount)])


@pytest.mark.parametrize("shape,threads", [
    ((5000, 3001), 256), ((20000, 513), 64), ((100000, 257), 32),            # 16 elements a thread: many long rows
    ((100000, 129), 32), ((100000, 65), 16),                                 # eight
    ((64, 3001), 1024), ((1000, 511), 128), ((20000, 127), 32), ((100000, 31), 8), ((1000, 15), 4), ((20000, 1022), 128),  # four
])
def test_threads_of_a_row_of_narrow_vectors(shape, threads):
    """Measured on 390 shapes: never more than 4 % slower than four vectors a thread, up to 3.2 times as 16 everywhere was (1000 x 15: 1.6 us
    with four elements a thread, 3.9 with 16)."""
    import re

    from lumen_b200.runtime import Fusion

    def chain(x, gg, b):
        y = F.relu(x * gg + b)
        return y, prims.reduce_sum(y * y, (1,), "float32")

    g = tracer.trace(chain, ("float32", shape), ("float32", shape[1:]), ("float32", shape[1:]))
    assert int(re.search(r"(\d+) threads per row", Fusion(g).source).group(1)) == threads
