"""How many elements of a row each of a thread's sums takes: no more than with the threads that a row would have by its vectors alone, four to
a thread (eight elements in kernels that sum columns too, twelve of packed pairs), so that float32 sums are no less exact for the fewer threads that walk it. Pairs that
are added packed (bfloat16) keep two sums."""

import re

import numpy as np
import pytest

from lumen_b200 import functional as F
from lumen_b200 import nn, prims, tracer
from lumen_b200.runtime import Fusion


def rms_norm(x, w):
    return F.rms_norm(x.float(), w.float()).to(x.dtype)


def layer_norm(x, w):
    return nn._ln_forward(x, w, w, 1e-5)[0]


def log_sum_exp(x, w):
    y = x.float()
    top = prims.reduce_max(y, (1,))
    return F.log(prims.reduce_sum(F.exp(y - top.reshape(y.shape[0], 1)), (1,), "float32"))


def gradients(x, w, g):
    y = x.float() * F.rsqrt(F.mean(x.float() * x.float(), -1, keepdim=True) + 1e-5)
    t = g.float() * w.float()
    return (t - y * F.mean(t * y, -1, keepdim=True)).to(x.dtype), prims.reduce_sum(g.float() * y, (0,), "float32")


def row_sums(program, rows, cols, dtype):
    """Threads of a row, elements of a vector, vectors of a thread, and the sums that each row total keeps a thread."""
    types = [(dtype, (rows, cols)), (dtype, (cols,))] + [(dtype, (rows, cols))] * (program is gradients)
    source = Fusion(tracer.trace(program, *types)).source
    threads, vector, vectors = (int(re.search(rf"#define {name} (\d+)", source)[1]) for name in ("TPR", "VEC", "NCH"))
    totals = re.findall(r"float (acc\d+)(?:\[(\d+)\])? = \{?0\.0f", source)
    assert totals
    return threads, vector, vectors, [int(n or 1) for _, n in totals]


def former_threads(cols, vector):
    threads = 1
    while threads < (cols // vector + 3) // 4 and threads < 1024:
        threads *= 2
    return threads


@pytest.mark.parametrize("dtype", ["float16", "float32"])
@pytest.mark.parametrize("program", [rms_norm, layer_norm, log_sum_exp])
@pytest.mark.parametrize("cols", [256, 1536, 2040, 8200, 9872, 16384, 32768, 43704, 50304, 87376])
def test_no_longer_than_with_a_thread_to_four_vectors(cols, program, dtype):
    threads, vector, vectors, totals = row_sums(program, 700, cols, dtype)
    former = former_threads(cols, vector)
    for n in totals:
        assert threads >= former or vectors * vector <= n * max(vector, cols // former), (threads, vector, vectors, n)


@pytest.mark.parametrize("program", [rms_norm, layer_norm, log_sum_exp])
@pytest.mark.parametrize("cols", [8200, 9872, 32768])
def test_packed_pairs_keep_two_sums(cols, program):
    threads, _, _, totals = row_sums(program, 700, cols, "bfloat16")
    assert set(totals) == {2} and cols / threads <= 88


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("cols", [264, 384, 392, 512, 640, 760, 768, 776, 1016])
@pytest.mark.parametrize("elements", [1 << 20, 3 << 20, 1 << 24])
def test_kernels_that_sum_columns_keep_short_chains(cols, elements, dtype):
    threads, _, _, totals = row_sums(gradients, elements // cols, cols, dtype)
    for n in totals:
        assert -(-cols // threads) <= (12 if dtype == "bfloat16" else 8) * n, (threads, n)


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("program", [rms_norm, layer_norm, log_sum_exp])
def test_narrow_vectors_keep_four_sums(program, dtype):
    _, vector, vectors, totals = row_sums(program, 5000, 3002, dtype)
    assert vector == 2 and vectors > 4 and set(totals) == {4}


def enacted(terms, threads, vector, vectors, n):
    """The float32 total of each row: a thread's vectors lie `threads` vectors apart, element e goes to sum e % n; sums, then threads, as trees."""
    rows, cols = terms.shape
    dealt = np.zeros((rows, vectors * threads * vector), np.float32)
    dealt[:, :cols] = terms
    dealt = dealt.reshape(rows, vectors, threads, vector)
    sums = np.zeros((rows, threads, n), np.float32)
    for ch in range(vectors):
        for e in range(vector):
            sums[:, :, e % n] += dealt[:, ch, :, e]
    width = 1 << (threads - 1).bit_length()
    tree = np.zeros((rows, width), np.float32)
    while n > 1:
        sums, n = sums[:, :, 0::2] + sums[:, :, 1::2], n // 2
    tree[:, :threads] = sums[:, :, 0]
    while tree.shape[1] > 1:
        tree = tree[:, 0::2] + tree[:, 1::2]
    return tree[:, 0]


@pytest.mark.parametrize("cols", [8200, 9872, 32768])
def test_sums_are_no_less_exact(cols):
    """The emitted kernel's order of a sum of squares, re-enacted, against a thread to four vectors with one sum each."""
    threads, vector, vectors, (n,) = row_sums(rms_norm, 700, cols, "float16")
    former = former_threads(cols, vector)
    rng = np.random.default_rng(cols)
    terms = rng.standard_normal((400, cols)).astype(np.float16).astype(np.float32) ** 2
    exact = terms.astype(np.float64).sum(1)

    def error(*order):
        return np.sqrt(np.mean((enacted(terms, *order) / exact - 1) ** 2))

    # (two estimates from 400 rows each, whose quotient is known to a twentieth)
    assert error(threads, vector, vectors, n) <= 1.05 * error(former, vector, -(-cols // vector // former), 1)
