"""Parity of the generated fused kernels with the CPU oracle, through the C ABI, on a B200."""

import numpy as np
import pytest
import torch

import lumen_b200
from lumen_b200 import functional as F
from lumen_b200 import prims, tracer
from lumen_b200.runtime import Fusion, desc
from tests.helpers import BF16, bf16, run_oracle, to_numpy, to_torch

pytestmark = pytest.mark.gpu


def chain(x, g, b):
    y = F.relu(x * g + b)
    return y, prims.reduce_sum(y * y, (1,), "float32")


def chain_inputs(rows, cols, dtype, seed=1):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((rows, cols)).astype(np.float32)
    g = rng.uniform(0.5, 1.5, cols).astype(np.float32)
    b = (0.1 * rng.standard_normal(cols)).astype(np.float32)
    if dtype == "bfloat16":
        x, g, b = bf16(x), bf16(g), bf16(b)
    return x, g, b


def device_run(graph, inputs, cuda):
    outs = Fusion(graph)(*[to_torch(a, cuda) for a in inputs])
    torch.cuda.synchronize()
    return [to_numpy(o) for o in outs]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("shape", [(64, 4096), (7, 1000), (33, 36), (1, 8), (5, 3)])
def test_chain_matches_oracle(cuda, dtype, shape):
    """y = relu(x*g+b) is bit-exact (one rounding per primitive); the row sum of squares differs from the
    sequential sum only by its order (rtol 1e-5, the reference's own tolerance for device reductions,
    tests/graph_compiler/test_elementwise_fusion.py:112-120)."""
    rows, cols = shape
    g = tracer.trace(chain, (dtype, shape), (dtype, (cols,)), (dtype, (cols,)))
    inputs = chain_inputs(rows, cols, dtype)
    y, s = device_run(g, inputs, cuda)
    want_y, want_s = run_oracle(g, inputs)
    assert y.dtype == want_y.dtype
    np.testing.assert_array_equal(y.view(np.uint16 if dtype == "bfloat16" else np.uint32), want_y.view(np.uint16 if dtype == "bfloat16" else np.uint32))
    np.testing.assert_allclose(s, want_s, rtol=1e-5, atol=1e-6)


def test_chain_sum_only(cuda):
    def f(x, g, b):
        return chain(x, g, b)[1]

    g = tracer.trace(f, ("float32", (128, 512)), ("float32", (512,)), ("float32", (512,)))
    inputs = chain_inputs(128, 512, "float32")
    (s,) = device_run(g, inputs, cuda)
    (want,) = run_oracle(g, inputs)
    np.testing.assert_allclose(s, want, rtol=1e-5)


def test_full_size_chain_properties(cuda):
    """At the benchmark's full size ([16384, 4096]) the oracle is too slow to run whole: check rows sampled against
    it, and size-independent properties: y >= 0, s == sum(y*y) recomputed in float64 from the device's y."""
    rows, cols = 16384, 4096
    g = tracer.trace(chain, ("float32", (rows, cols)), ("float32", (cols,)), ("float32", (cols,)))
    x, gg, b = chain_inputs(rows, cols, "float32")
    y, s = device_run(g, (x, gg, b), cuda)
    assert (y >= 0).all()
    np.testing.assert_allclose(s, (y.astype(np.float64) ** 2).sum(1), rtol=1e-5)
    sample = np.arange(0, rows, 1021)
    small = tracer.trace(chain, ("float32", (len(sample), cols)), ("float32", (cols,)), ("float32", (cols,)))
    want_y, want_s = run_oracle(small, (x[sample], gg, b))
    np.testing.assert_array_equal(y[sample], want_y)
    np.testing.assert_allclose(s[sample], want_s, rtol=1e-5)


def test_layer_norm_rows(cuda):
    """Layer norm spelled from prims (tests/graph_compiler/test_normalizations.py:103-106) as one row kernel; the
    bfloat16 variant widens to float32 for the statistics and narrows the result, as a bfloat16 model does
    (a sum accumulated in bfloat16 itself depends on the order of its 1024 terms far beyond any tolerance)."""
    def ln16(a, w, b):
        return F.layer_norm(a.float(), w.float(), b.float()).bfloat16()

    for dtype, f, tol in (("float32", F.layer_norm, 1e-5), ("bfloat16", ln16, 2**-7)):
        g = tracer.trace(f, (dtype, (96, 1024)), (dtype, (1024,)), (dtype, (1024,)))
        rng = np.random.default_rng(5)
        a = rng.standard_normal((96, 1024)).astype(np.float32) * 2 + 0.5
        w = rng.uniform(0.5, 1.5, 1024).astype(np.float32)
        b = rng.standard_normal(1024).astype(np.float32)
        inputs = (a, w, b) if dtype == "float32" else (bf16(a), bf16(w), bf16(b))
        (y,) = device_run(g, inputs, cuda)
        (want,) = run_oracle(g, inputs)
        np.testing.assert_allclose(y.astype(np.float32), want.astype(np.float32), rtol=tol, atol=tol)


def test_bfloat16_accumulated_sum(cuda):
    """A sum accumulated in bfloat16 (F.sum of a bfloat16 tensor): within the reference's 2e-1 for
    bf16-accumulated reductions (tests/graph_compiler/test_elementwise_fusion.py:112-120) on short rows."""
    g = tracer.trace(lambda x: F.sum(x, -1), ("bfloat16", (64, 32)))
    x = bf16(np.random.default_rng(8).standard_normal((64, 32)))
    (s,) = device_run(g, (x,), cuda)
    (want,) = run_oracle(g, (x,))
    np.testing.assert_allclose(s.astype(np.float32), want.astype(np.float32), rtol=2e-1, atol=2e-1)


def test_softmax_rows(cuda):
    g = tracer.trace(lambda x: F.softmax(x, -1), ("float32", (50, 300)))
    x = np.random.default_rng(6).standard_normal((50, 300)).astype(np.float32) * 3
    (y,) = device_run(g, (x,), cuda)
    (want,) = run_oracle(g, (x,))
    np.testing.assert_allclose(y, want, rtol=1e-5, atol=1e-7)


def test_embedding_gather_is_exact(cuda):
    """tokens[ids] + positions: indices clamped (lumen/reference/mod.rs:414-423), result bit-exact."""
    def f(tok, pos, ids):
        return (tok[ids] + pos).reshape(8 * 64, 128)

    g = tracer.trace(f, ("float32", (256, 128)), ("float32", (64, 128)), ("int64", (8, 64)))
    rng = np.random.default_rng(0)
    tok = rng.standard_normal((256, 128)).astype(np.float32)
    pos = rng.standard_normal((64, 128)).astype(np.float32)
    ids = rng.integers(-3, 260, (8, 64))  # some out of range: clamped
    (y,) = device_run(g, (tok, pos, ids), cuda)
    (want,) = run_oracle(g, (tok, pos, ids))
    np.testing.assert_array_equal(y, want)


def test_integer_rules_are_exact(cuda):
    """Integer division by zero is -1, overflow wraps, casts saturate (lumen/reference/mod.rs:448-468,203-220)."""
    def f(a, b, x):
        q = prims.div(a, b)
        return q, prims.mul(a, b), prims.cast(x, "int32"), prims.cast(x, "uint8"), prims.lt(a, b), prims.max(a, b)

    g = tracer.trace(f, ("int32", (64,)), ("int32", (64,)), ("float32", (64,)))
    rng = np.random.default_rng(2)
    a = rng.integers(-(2**31), 2**31 - 1, 64).astype(np.int32)
    b = rng.integers(-(2**31), 2**31 - 1, 64).astype(np.int32)
    b[:4] = 0
    a[4], b[4] = -(2**31), -1
    x = (rng.standard_normal(64) * 1e10).astype(np.float32)
    x[:3] = [np.nan, np.inf, -np.inf]
    got = device_run(g, (a, b, x), cuda)
    want = run_oracle(g, (a, b, x))
    for u, v in zip(got, want):
        np.testing.assert_array_equal(u, v)
    assert got[0][0] == -1


def test_unsigned_division_by_the_largest_value(cuda):
    """A divisor of all ones is -1 only for signed types (where the quotient is the wrapped negation and the remainder
    0); for unsigned types it is the largest value, an ordinary divisor."""
    for dtype in ("uint8", "uint32", "int32", "int8"):
        info = np.iinfo(dtype)
        rng = np.random.default_rng(4)
        a = rng.integers(info.min, info.max, 256, dtype=dtype, endpoint=True)
        b = rng.integers(info.min, info.max, 256, dtype=dtype, endpoint=True)
        b[::3] = np.array(-1).astype(dtype)  # all ones
        a[0], a[3] = info.min, info.max
        g = tracer.trace(lambda x, y: (prims.div(x, y), prims.rem(x, y)), (dtype, (256,)), (dtype, (256,)))
        got, want = device_run(g, (a, b), cuda), run_oracle(g, (a, b))
        for u, v in zip(got, want):
            np.testing.assert_array_equal(u, v, err_msg=dtype)


@pytest.mark.parametrize("dtype", ["int8", "int16", "int32", "int64"])
@pytest.mark.parametrize("shape", [(7, 5, 32), (300, 32), (40, 257)])
def test_integer_extrema_of_negations(cuda, dtype, shape):
    """Row minima and maxima of negated integers, however the negation is spelled (`neg`, `0 - x`, `x * -1`, `abs`), alone
    and beside a full-sized result of the same kernel. The toolchain turns a chain of signed 32-bit max over literal
    negations into the extremum over x and -x together; the generated kernels spell negations so that it cannot."""
    info = np.iinfo(dtype)
    rng = np.random.default_rng(6)
    x = rng.integers(info.min, info.max, shape, dtype=dtype, endpoint=True)
    y = rng.integers(info.min, info.max, shape, dtype=dtype, endpoint=True)

    def program(a, b):
        m = prims.max(a, b)
        return (F.amin(a, -1), F.amax(prims.neg(a), -1), F.amax(F.sub(0, a), -1), F.amax(F.mul(a, -1), -1), F.amax(F.abs(b), -1),
                m, F.amin(m, -1), F.amin(prims.neg(m), -1),
                prims.max(prims.max(prims.max(prims.neg(a), prims.neg(b)), prims.neg(m)), F.sub(0, prims.min(a, b))))  # fmt: skip

    g = tracer.trace(program, (dtype, shape), (dtype, shape))
    want = run_oracle(g, (x, y))
    import lumen_b200

    got = lumen_b200.compile(program)(to_torch(x, cuda), to_torch(y, cuda))
    torch.cuda.synchronize()
    for k, (u, v) in enumerate(zip(got, want)):
        np.testing.assert_array_equal(to_numpy(u), v, err_msg=f"output {k}")


def test_unsupported_primitive_is_named(cuda):
    from lumen_b200._lib import LumenError

    g = tracer.trace(lambda x: prims.reduce_sum(x, (1,), "float32"), ("float32", (4, 5, 6)))
    with pytest.raises(LumenError, match="reduce_sum"):
        Fusion(g)


def test_column_reductions(cuda):
    """Sums over the leading axis (weight gradients of a layer norm): partial sums per row slice, then a finalize
    pass, both in a fixed order; against the oracle's sequential sums."""
    rows, cols = 1000, 384

    def f(dy, x, mean, rstd):
        xhat = (x.float() - mean.reshape(rows, 1)) * rstd.reshape(rows, 1)
        g = dy.float()
        return prims.reduce_sum(g * xhat, (0,), "float32").bfloat16(), prims.reduce_sum(g, (0,), "float32")

    g = tracer.trace(f, ("bfloat16", (rows, cols)), ("bfloat16", (rows, cols)), ("float32", (rows,)), ("float32", (rows,)))
    rng = np.random.default_rng(7)
    inputs = (bf16(rng.standard_normal((rows, cols))), bf16(rng.standard_normal((rows, cols))),
              rng.standard_normal(rows).astype(np.float32), rng.uniform(0.5, 2, rows).astype(np.float32))
    got = device_run(g, inputs, cuda)
    want = run_oracle(g, inputs)
    np.testing.assert_allclose(got[0].astype(np.float32), want[0].astype(np.float32), rtol=2**-7, atol=2**-7 * np.abs(want[0].astype(np.float32)).max())
    np.testing.assert_allclose(got[1], want[1], rtol=1e-4, atol=1e-4 * np.abs(want[1]).max())
    again = device_run(g, inputs, cuda)
    np.testing.assert_array_equal(got[1], again[1])


def test_cross_entropy_rows(cuda):
    """Per-row logsumexp - x[target] with the target logit gathered by a data-dependent index, and its gradient."""
    rows, classes = 96, 1000
    rng = np.random.default_rng(8)
    x = (rng.standard_normal((rows, classes)) * 3).astype(np.float32)
    t = rng.integers(0, classes, rows)
    g = tracer.trace(lambda a, c: F.cross_entropy_forward_prims(a, c), ("float32", x.shape), ("int64", t.shape))
    loss, lse = device_run(g, (x, t), cuda)
    want_loss, want_lse = run_oracle(g, (x, t))
    np.testing.assert_allclose(lse, want_lse, rtol=1e-5)
    np.testing.assert_allclose(loss, want_loss, rtol=1e-5, atol=1e-5)
    gb = tracer.trace(lambda a, c, l, gg: F.cross_entropy_backward_prims(a, c, l, gg).bfloat16(),
                      ("float32", x.shape), ("int64", t.shape), ("float32", (rows,)), ("float32", (rows,)))
    gg = rng.standard_normal(rows).astype(np.float32)
    (dx,) = device_run(gb, (x, t, want_lse, gg), cuda)
    (want,) = run_oracle(gb, (x, t, want_lse, gg))
    np.testing.assert_allclose(dx.astype(np.float32), want.astype(np.float32), rtol=2**-7, atol=1e-6)


def test_inplace_update(cuda):
    """`p - lr * g` written over `p` (a donated output): the kernel is generated without read-only loads."""
    from lumen_b200 import nn
    from lumen_b200.compiler import compile_graph
    from lumen_b200.plan import Plan

    def step(p, gr):
        return nn.sgd_update(p, gr, 0.5)

    gph = tracer.trace(step, ("float32", (300, 70)), ("float32", (300, 70)))
    rng = np.random.default_rng(9)
    p0, gr = rng.standard_normal((300, 70)).astype(np.float32), rng.standard_normal((300, 70)).astype(np.float32)
    (want,) = run_oracle(gph, (p0, gr))
    plan = Plan(compile_graph(gph, {0: 0}), cuda)
    assert "option inplace" in plan.compiled.text
    p_t, g_t = to_torch(p0, cuda), to_torch(gr, cuda)
    plan.run([p_t, g_t], [p_t])
    torch.cuda.synchronize()
    np.testing.assert_array_equal(to_numpy(p_t), want)


_ = BF16


@pytest.mark.parametrize("shape", [(64, 64), (257, 40), (1000, 1000), (3, 4096), (5000, 33), (600, 8200), (2, 16384)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_row_and_column_reductions_in_one_kernel(cuda, shape, dtype):
    """Rows centred, and the column sums of the rows and of the centred rows, from one kernel: narrow rows (several to a
    block), rows of one and of several chunks per thread, fewer rows than blocks, widths without a vector's divisor.
    Sums within 1e-5 of the sums of magnitudes (float32 accumulation of at most 5000 terms in any order: 5000 * 2^-24
    = 3e-4 at the very worst, about its square root of terms in practice); a 16-bit result adds its own rounding."""
    rows, cols = shape
    x = np.random.default_rng(rows).standard_normal(shape).astype(np.float32)
    x = bf16(x) if dtype == "bfloat16" else x

    def program(a):
        w = a.to("float32")
        c = w - prims.reduce_sum(w, (1,), "float32").reshape(rows, 1) * (1.0 / cols)
        return c.to(dtype), prims.reduce_sum(w, (0,), "float32"), prims.reduce_sum(c * c, (0,), "float32").to(dtype)

    c, s, q = (to_numpy(t).astype(np.float64) for t in Fusion(tracer.trace(program, (dtype, shape)))(to_torch(x, cuda)))
    x64 = x.astype(np.float64)
    want = x64 - x64.mean(1, keepdims=True)
    half = 2.0**-8 if dtype == "bfloat16" else 0.0
    assert (np.abs(c - want) <= (half + 1e-6) * np.abs(want) + 1e-5).all()
    assert (np.abs(s - x64.sum(0)) <= 1e-5 * np.abs(x64).sum(0)).all()
    assert (np.abs(q - (want * want).sum(0)) <= (half + 2e-5) * (want * want).sum(0)).all()


# where the threads of a row and the blocks of an SM change (two vectors of eight bytes for 16 bits from 1024 columns on; one vector of 16 from
# 2^21 elements of float32 on), and more row blocks than slices
@pytest.mark.parametrize("dtype, shape", [("float32", s) for s in ((4100, 512), (2100, 1000), (1400, 1536), (700, 3072), (600, 4096), (420, 5000))]
                         + [("bfloat16", s) for s in ((2000, 1024), (1000, 2304), (900, 2600), (400, 5000), (300, 8192), (3000, 512))])
def test_threads_of_rows_with_column_sums(cuda, dtype, shape):
    """Row and column sums of one kernel against float64: `cols` terms of a row in any order, `rows` of a column, each within
    their number's root times 2^-24 of the sum of magnitudes in practice, four times that allowed."""
    rows, cols = shape
    x = torch.randn(shape, generator=torch.Generator(device=cuda).manual_seed(cols), device=cuda).to(getattr(torch, dtype))

    def program(a):
        w = a.to("float32")
        r = prims.reduce_sum(w, (1,), "float32")
        q = prims.reduce_sum(w * w, (1,), "float32")
        return r, q, prims.reduce_sum(w * r.reshape(rows, 1), (0,), "float32"), prims.reduce_sum(w, (0,), "float32")

    r, q, c, s = (to_numpy(t).astype(np.float64) for t in Fusion(tracer.trace(program, (dtype, shape)))(x))
    x64 = x.double().cpu().numpy()
    near = lambda got, terms, axis: (np.abs(got - terms.sum(axis)) <= 4 * terms.shape[axis] ** 0.5 * 2.0**-24 * np.abs(terms).sum(axis)).all()
    assert near(r, x64, 1) and near(q, x64 * x64, 1) and near(c, x64 * r[:, None], 0) and near(s, x64, 0)


# widths whose vectors are one or two elements: one thread per row up to a whole block, remainders of a thread's share
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("rows,cols", [(3, 1), (70, 15), (9, 17), (33, 257), (5, 511), (5, 514), (7, 3001), (4, 4097), (3, 8190), (2, 16383)])
def test_rows_of_odd_widths(cuda, rows, cols, dtype):
    """y is exact; a float32 sum of `cols` non-negative terms in any order is within cols * 2^-24 of the float64 one."""
    gen = torch.Generator(device=cuda).manual_seed(cols)
    t = getattr(torch, dtype)
    x, g, b = (torch.randn(s, generator=gen, device=cuda).to(t) for s in ((rows, cols), (cols,), (cols,)))

    def chain(x_, g_, b_):
        y_ = F.relu(x_ * g_ + b_)
        return y_, prims.reduce_sum(y_ * y_, (1,), "float32")

    y, s = lumen_b200.compile(chain)(x, g, b)
    y, s = torch.as_tensor(y, device=cuda), torch.as_tensor(s, device=cuda)
    want = torch.relu(x * g + b)
    assert torch.equal(y.view(t) if y.dtype != t else y, want)
    total = (want * want).double().sum(1)
    assert ((s.double() - total).abs() <= cols * 2.0**-24 * total + 1e-30).all()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("cols", [8, 96, 1024, 4100])
def test_rows_divided_by_one_value_each(cuda, cols, dtype):
    """Quotients by a row's own divisor - inside and outside the range in which they are taken by its reciprocal, at the ends of that
    range, with zeros, subnormals, infinities and NaN among the elements - are the correctly rounded ones, also where a later phase
    of the row divides the same again, and where few elements a thread keep them for it."""
    rng = np.random.default_rng(cols)
    edges = [1.0, 3.0, -3.0, 0.0, -0.0, np.inf, np.nan, 2.0**-40, 2.0**-41, 2.0**40, 2.0**41, 1e-45, 3e38, np.nextafter(np.float32(2), np.float32(1))]
    d = np.concatenate([np.array(edges, np.float32), np.exp2(rng.uniform(-39, 39, 50)).astype(np.float32)])
    rows = len(d)
    x = (rng.standard_normal((rows, cols)) * np.exp2(rng.uniform(-30, 30, (rows, cols)))).astype(np.float32)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, -1e-40, 3e38, 2.0**-61, 2.0**61, 2.0**-60, 2.0**60], np.float32)
    x[::3, : min(cols, 12)] = special[: min(cols, 12)]
    x[1] = 0.0
    if dtype == "bfloat16":
        x = bf16(x)

    def program(a, b):
        w = a.to("float32")
        q = w / b
        big = prims.reduce_max(q, (1,)).reshape(rows, 1)
        return q, w / b - big, prims.reduce_sum(q / b, (1,), "float32")

    g = tracer.trace(program, (dtype, (rows, cols)), ("float32", (rows, 1)))
    kernel = Fusion(g)
    assert "divide_chunk<" in kernel.source
    q, r, _ = (to_numpy(t) for t in kernel(to_torch(x, cuda), to_torch(d.reshape(rows, 1), cuda)))
    with np.errstate(all="ignore"):
        want = x.astype(np.float32) / d.reshape(rows, 1)
        big = np.maximum.reduce(want, axis=1, keepdims=True)  # (propagates NaN, as the kernel's maximum does)
        np.testing.assert_array_equal(q, want)
        np.testing.assert_array_equal(np.signbit(q[want == 0]), np.signbit(want[want == 0]))
        np.testing.assert_array_equal(r, want - big)


# odd rows of bfloat16 that start at every distance from an aligned address: several a block and one, one chunk a thread and four, fewer
# rows than eight a block's share, a last row whose last chunk ends with the tensor
@pytest.mark.parametrize("rows,cols", [(50001, 129), (25000, 257), (6300, 1001), (3100, 2047), (2500, 3001), (1601, 4095), (385, 16383), (97, 65533)])
def test_rows_at_any_address(cuda, rows, cols):
    """y is exact whether the tensors are aligned or not (then another kernel runs); float32 sums of `cols` non-negative terms are
    within cols * 2^-24 of the float64 ones; nothing beside the results is written."""
    gen = torch.Generator(device=cuda).manual_seed(cols)
    x, g, b = (torch.randn(s, generator=gen, device=cuda).bfloat16() for s in ((rows, cols), (cols,), (cols,)))
    r = torch.randn((rows, 1), generator=gen, device=cuda).bfloat16()

    def program(x_, g_, b_):
        y_ = F.relu(x_ * g_ + b_)
        return y_, prims.reduce_sum(y_ * y_, (1,), "float32")

    def largest(x_, r_):
        return prims.reduce_max(x_ * r_, (1,)), (x_ * r_).to("float32")

    def bare(x_, g_, b_):
        return x_ * g_ + b_, (x_ - b_).to("float32")

    def run(fn, *args):
        kernel = Fusion(tracer.trace(fn, *[("bfloat16", tuple(a.shape)) for a in args]))
        assert "PERIOD" in kernel.source or (fn is bare and cols < 1024)  # (shorter rows without a sum are put together)
        types = [kernel.body.types[v] for v in kernel.body.outputs]
        out = [torch.full((t.numel + 16,), 7.0, device=cuda, dtype=getattr(torch, t.dtype)) for t in types]
        views = [o[8 : 8 + t.numel].reshape(t.shape) for o, t in zip(out, types)]
        kernel(*args, out=views)
        for o, t in zip(out, types):
            assert (o[:8] == 7).all() and (o[8 + t.numel :] == 7).all()
        return views

    want = torch.relu(x * g + b)
    total = (want * want).double().sum(1)
    for shift in (0, 1):  # elements that the arguments start behind an aligned address
        xs, gs, bs = (torch.cat([a.new_zeros(shift), a.flatten()])[shift:].reshape(a.shape) for a in (x, g, b))
        y, s = run(program, xs, gs, bs)
        assert torch.equal(y, want)
        assert ((s.double() - total).abs() <= cols * 2.0**-24 * total + 1e-30).all()
    m, w = run(largest, x, r)
    assert torch.equal(m, (x * r).amax(1)) and torch.equal(w, (x * r).float())
    u, v = run(bare, x, g, b)
    assert torch.equal(u, x * g + b) and torch.equal(v, (x - b).float())


@pytest.mark.parametrize("rows,cols", [(50001, 129), (6300, 1001), (2503, 3001), (1601, 4095), (385, 16383), (97, 65533)])
def test_odd_rows_count_their_own_elements(cuda, rows, cols):
    """Sums of small whole numbers are exact in any order: every element of a row counts once and none of its neighbours' does, with
    float32 operands beside the 16-bit ones (vectors of 32 bytes, a column operand moved by its elements)."""
    gen = torch.Generator(device=cuda).manual_seed(cols)
    x = torch.randint(0, 4, (rows, cols), generator=gen, device=cuda).bfloat16()
    g, w = torch.randint(1, 5, (cols,), generator=gen, device=cuda).float(), torch.randint(0, 8, (rows, cols), generator=gen, device=cuda).float()

    def program(x_, g_, w_):
        z = (x_ * x_).to("float32") * g_ + w_
        return z, prims.reduce_sum(z, (1,), "float32")

    kernel = Fusion(tracer.trace(program, ("bfloat16", (rows, cols)), ("float32", (cols,)), ("float32", (rows, cols))))
    assert "PERIOD" in kernel.source and "ldv_shifted<float, VEC, idx_t>" in kernel.source
    z, total = kernel(x, g, w)
    want = (x * x).float() * g + w
    assert torch.equal(z, want) and torch.equal(total.double(), want.double().sum(1))


@pytest.mark.parametrize("rows,cols", [(50001, 129), (2503, 3001), (1601, 4095), (97, 65533)])
def test_odd_rows_in_place(cuda, rows, cols):
    """The result over its operand: neighbours that a vector brings along are never written back."""
    x = torch.randn((rows, cols), generator=torch.Generator(device=cuda).manual_seed(cols), device=cuda).bfloat16()
    g = torch.randn((cols,), generator=torch.Generator(device=cuda).manual_seed(1), device=cuda).bfloat16()
    kernel = Fusion("option inplace\n" + tracer.trace(lambda a, b: (a * b) * a, ("bfloat16", (rows, cols)), ("bfloat16", (cols,))).to_text())
    assert "ldv_within_plain<u16, VEC, idx_t>" in kernel.source or cols < 1024  # (shorter rows without a sum are put together)
    want = (x * g) * x
    kernel.launch_raw([desc(t) for t in (x, g, x)])
    assert torch.equal(x, want)


def test_rows_at_any_address_under_capture(cuda):
    """A program that has run on aligned tensors is captured on others, which take another kernel, and replays them."""
    rows, cols = 2503, 3001
    x = torch.randn((rows, cols), generator=torch.Generator(device=cuda).manual_seed(0), device=cuda).bfloat16()
    kernel = Fusion(tracer.trace(lambda a: F.relu(a * 0.375), ("bfloat16", (rows, cols))))
    assert "PERIOD" in kernel.source
    aligned, off = torch.empty_like(x), torch.cat([x.new_zeros(1), x.flatten()])[1:].reshape(rows, cols)
    out = torch.empty(rows * cols + 1, device=cuda, dtype=torch.bfloat16)[1:].reshape(rows, cols)
    kernel(x, out=[aligned])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        kernel(off, out=[out])
    out.zero_()
    graph.replay()
    assert torch.equal(out, torch.relu(x * 0.375)) and torch.equal(out, aligned)


def column_sums_in_slices(x):
    """float32 column sums in the order of the two-pass column reduction: slices of at least 64 rows, eight row lanes each that add every
    eighth row, eight slice lanes that add every eighth slice, lanes in order."""
    rows, cols = x.shape
    col_blocks = -(-cols // 128)
    slices = min(max(1, -(-592 // col_blocks)), max(rows // 64, 1))
    per = -(-rows // slices)

    def lanes(rows_, n=8):  # [.., k, cols] -> [.., cols]
        pad = -rows_.shape[-2] % n
        rows_ = torch.cat([rows_, rows_.new_zeros(*rows_.shape[:-2], pad, cols)], -2).unflatten(-2, (-1, n))
        total = rows_[..., 0, :, :]
        for k in range(1, rows_.shape[-3]):
            total = total + rows_[..., k, :, :]
        out = total[..., 0, :]
        for y in range(1, n):
            out = out + total[..., y, :]
        return out

    whole = torch.cat([x, x.new_zeros(-(-rows // per) * per - rows, cols)]).unflatten(0, (-1, per))
    return lanes(lanes(whole))


@pytest.mark.parametrize("rows,cols", [(4096, 64), (1020, 260), (512, 512), (8192, 1024), (20000, 1000), (2048, 4096)])
@pytest.mark.parametrize("beside", [False, True])
def test_column_sums_are_as_exact_as_in_slices(cuda, rows, cols, beside):
    """Alone and beside row outputs (one kernel for both), the root mean square of a column sum's error is no larger than in the
    order above, whose chains of adds are about as long; over the columns it varies by 1 / sqrt(2 * cols), of which three are allowed."""
    x = torch.randn((rows, cols), generator=torch.Generator(device=cuda).manual_seed(rows), device=cuda)

    def program(a):
        s = prims.reduce_sum(a, (0,), "float32")
        return (a - prims.reduce_sum(a, (1,), "float32").reshape(rows, 1), s) if beside else s

    s = lumen_b200.compile(program)(x)
    s = torch.as_tensor(s[1] if beside else s, device=cuda)
    want = x.double().sum(0)

    def rms(t):
        return float(((t.double() - want) ** 2).mean() ** 0.5)

    assert rms(s) <= (1 + 3 / (2 * cols) ** 0.5) * rms(column_sums_in_slices(x))


# rows that one block of 288 to 384 threads would take with eight elements a thread, and the widths beside them
@pytest.mark.parametrize("rows,cols", [(50, 2048), (50, 2052), (301, 2304), (40, 3001), (60, 3072), (33, 3076), (7, 2311)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_rows_between_one_and_two_blocks_an_sm(cuda, rows, cols, dtype):
    """As test_row_and_column_reductions_in_one_kernel, the column sums no worse than twice the error of a tree over the rows."""
    x = torch.randn((rows, cols), generator=torch.Generator(device=cuda).manual_seed(cols), device=cuda).to(getattr(torch, dtype))

    def program(a):
        w = a.to("float32")
        c = w - prims.reduce_sum(w, (1,), "float32").reshape(rows, 1) * (1.0 / cols)
        return c, prims.reduce_sum(w, (0,), "float32"), prims.reduce_sum(c * c, (0,), "float32")

    c, s, q = Fusion(tracer.trace(program, (dtype, (rows, cols))))(x)
    w = x.double()
    want = w - w.mean(1, keepdim=True)
    assert ((c.double() - want).abs() <= 1e-6 * want.abs() + 1e-5).all()
    assert ((s.double() - w.sum(0)).abs() <= rows * 2.0**-24 * w.abs().sum(0)).all()
    assert ((q.double() - (want * want).sum(0)).abs() <= (rows * 2.0**-24 + 1e-5) * (want * want).sum(0)).all()


@pytest.mark.parametrize("cols", [1024, 2048, 4096, 8192])
def test_a_rows_warps_are_added_as_a_tree(cuda, cols):
    """Row sums whose rows are taken by two to eight warps with four vectors of four a thread, bit for bit: a thread's elements in order,
    lanes by xor 16, 8, 4, 2, 1 (pairs differ in the lane's highest bit first), warps likewise."""
    x = torch.randn((70, cols), generator=torch.Generator(device=cuda).manual_seed(cols), device=cuda)
    threads = cols // 16
    v = x.reshape(70, 4, threads, 4)  # chunk, thread, element
    total = torch.zeros((70, threads), device=cuda)
    for chunk in range(4):
        for e in range(4):
            total = total + v[:, chunk, :, e]
    total = total.reshape(70, -1, 32)
    for half in (16, 8, 4, 2, 1):
        total = total[..., :half] + total[..., half:]
    total = total[..., 0]
    while total.shape[1] > 1:
        total = total[:, : total.shape[1] // 2] + total[:, total.shape[1] // 2 :]
    s = Fusion(tracer.trace(lambda a: prims.reduce_sum(a, (1,), "float32"), ("float32", (70, cols))))(x)[0]
    assert torch.equal(s, total[:, 0])


@pytest.mark.parametrize("cols", [1001, 2047, 3001, 3002, 4095, 8190])
def test_row_sums_of_odd_widths_are_as_exact_as_of_1024_threads(cuda, cols):
    """Narrow vectors of a row are many to a thread; the root mean square of a sum's error is no larger than with four of them to a
    thread, added one by one, and trees over a warp's lanes and over the warps. 4000 rows: it varies by 1 / sqrt(8000), of which
    three are allowed."""
    rows, vec = 4000, 2 if cols % 2 == 0 else 1
    x = torch.randn((rows, cols), generator=torch.Generator(device=cuda).manual_seed(cols), device=cuda)
    threads = 32
    while threads < min(1024, -(-cols // (4 * vec))):
        threads *= 2
    chunks = -(-cols // (threads * vec))
    v = torch.cat([x, x.new_zeros(rows, chunks * threads * vec - cols)], 1).reshape(rows, chunks, threads, vec)
    total = torch.zeros((rows, threads), device=cuda)
    for chunk in range(chunks):
        for e in range(vec):
            total = total + v[:, chunk, :, e]
    while total.shape[1] > 1:
        total = total[:, : total.shape[1] // 2] + total[:, total.shape[1] // 2 :]
    s = Fusion(tracer.trace(lambda a: prims.reduce_sum(a, (1,), "float32"), ("float32", (rows, cols))))(x)[0]
    want = x.double().sum(1)

    def rms(t):
        return float(((t.double() - want) ** 2).mean() ** 0.5)

    assert rms(s) <= (1 + 3 / 8000**0.5) * rms(total[:, 0])


# totals of 257 slices and more over few columns take 128 slice lanes (on eight column lanes): beside a row sum and alone, two columns a
# thread and one, columns that are no multiple of a block's, one column, the widest of them and one past; 256 slices do not
@pytest.mark.parametrize("rows,cols,beside,many", [
    (5000, 1024, True, True), (5000, 64, True, True), (5000, 1022, True, True), (600, 3072, True, True), (257, 500, True, True),
    (5000, 1023, True, True), (20000, 17, True, True), (700, 2047, True, True),
    (256, 500, True, False), (700, 2049, True, False), (300, 4096, True, False),
    (20000, 64, False, True), (40000, 20, False, True), (65536, 256, False, True), (65536, 1, False, True), (16448, 64, False, True),
    (16384, 64, False, False), (40000, 300, False, False),
])  # fmt: skip
@pytest.mark.parametrize("sums", [1, 6])  # six: more than shared memory holds at once
def test_totals_of_many_slices(cuda, rows, cols, beside, many, sums):
    """Small integers: every order of the additions gives the same sum."""
    x = torch.randint(-8, 9, (rows, cols), generator=torch.Generator(device=cuda).manual_seed(cols), device=cuda).float()

    def program(a):
        totals = [prims.reduce_sum(a * float(k + 1), (0,), "float32") for k in range(sums - 1)] + [prims.reduce_max(a, (0,)) if sums > 1 else
                                                                                                   prims.reduce_sum(a, (0,), "float32")]
        return tuple(totals + ([a + prims.reduce_sum(a, (1,), "float32").reshape(rows, 1)] if beside else []))

    fusion = Fusion(tracer.trace(program, ("float32", (rows, cols))))
    assert ("row_lane = tid / 8;" in fusion.source) == many
    out = fusion(x)
    for k in range(max(sums - 1, 1)):
        assert torch.equal(out[k], x.sum(0) * (k + 1))
    if sums > 1:
        assert torch.equal(out[sums - 1], x.amax(0))
    if beside:
        assert torch.equal(out[sums], x + x.sum(1, keepdim=True))


@pytest.mark.parametrize("own", [False, True])  # torch's memory, the backend's own
def test_one_fusion_on_several_streams_and_threads(cuda, own):
    """Column totals of different inputs at once: small integers, so every order of the additions gives the same sum."""
    import threading

    from lumen_b200 import device as D

    rows, cols = 20000, 512
    fusion = Fusion(tracer.trace(lambda a: prims.reduce_sum(a, (0,), "float32"), ("float32", (rows, cols))))
    gen = torch.Generator(device=cuda).manual_seed(5)
    xs = [torch.randint(-8, 9, (rows, cols), generator=gen, device=cuda).float() for _ in range(4)]
    wants = [x.sum(0) for x in xs]
    streams = [D.Stream() for _ in range(2)]
    region = D.Region(256 << 20)
    outs = [[region.empty((cols,), "float32") if own else torch.empty(cols, device=cuda) for _ in range(20)] for _ in xs]
    if own:
        inputs = [region.empty((rows, cols), "float32") for _ in xs]
        for a, x in zip(inputs, xs):
            a.copy_from_host(x.cpu().numpy())
    else:
        inputs = xs
    torch.cuda.synchronize()
    errors = []

    def work(i):  # two threads to a stream
        try:
            torch.cuda.set_device(cuda)
            for out in outs[i]:
                fusion(inputs[i], out=[out], stream=streams[i % 2].handle)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(xs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    for got, want in zip(outs, wants):
        for out in got:
            assert torch.equal(torch.as_tensor(out, device=cuda), want)
