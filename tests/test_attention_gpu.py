"""Parity of the tcgen05 flash-attention kernels with the traced program evaluated by the oracle, and with a
float64 NumPy attention at sizes the oracle is too slow for."""

import numpy as np
import pytest
import torch

from lumen_b200 import functional as F
from lumen_b200 import tracer
from lumen_b200._lib import LumenError
from lumen_b200.runtime import attention_backward, attention_forward, device_status
from tests.helpers import attention_kernel, attention_f64, bf16, run_oracle, to_numpy, to_torch

pytestmark = pytest.mark.gpu

TOL = 2e-2  # bfloat16, rtol = atol (tests/functional/test_attention.py:54)


def qkv(b, sq, sk, n, nkv, h, seed=3):
    rng = np.random.default_rng(seed)
    return tuple(bf16(rng.standard_normal(s)) for s in ((b, sq, n, h), (b, sk, nkv, h), (b, sk, nkv, h)))


# (B, Sq, Sk, N, Nkv, H), causal: ragged lengths, GQA, a KV cache shape, both head dims
CASES = [
    ((2, 128, 128, 2, 2, 128), False),
    ((1, 256, 256, 2, 2, 128), True),
    ((2, 100, 100, 4, 2, 64), True),
    ((1, 130, 77, 2, 2, 64), False),
    ((1, 70, 200, 2, 1, 128), True),
    ((1, 300, 300, 3, 3, 128), True),
    ((1, 1, 300, 8, 2, 128), True),
]


@pytest.mark.parametrize("case", CASES)
def test_forward_matches_the_traced_program(cuda, case):
    (b, sq, sk, n, nkv, h), causal = case
    q, k, v = qkv(b, sq, sk, n, nkv, h)
    g = tracer.trace(lambda a, c, d: F.attention_forward_prims(a, c, d, h**-0.5, causal),
                     ("bfloat16", q.shape), ("bfloat16", k.shape), ("bfloat16", v.shape))
    want_o, want_lse = run_oracle(g, [q, k, v])
    o, lse = attention_forward(to_torch(q, cuda), to_torch(k, cuda), to_torch(v, cuda), causal=causal)
    device_status()
    np.testing.assert_allclose(to_numpy(o).astype(np.float32), want_o.astype(np.float32), rtol=TOL, atol=TOL)
    np.testing.assert_allclose(to_numpy(lse), want_lse[..., 0], rtol=1e-3, atol=1e-3)


def test_forward_reads_strided_views_in_place(cuda):
    """q, k, v as slices of one packed [B, S, 3, N, H] projection: no copies (strided accesses,
    lumen/graph_compiler/passes/attention/forward.rs:598-772)."""
    rng = np.random.default_rng(5)
    packed = to_torch(bf16(rng.standard_normal((2, 192, 3, 2, 64))), cuda)
    q, k, v = packed[:, :, 0], packed[:, :, 1], packed[:, :, 2]
    o, _ = attention_forward(q, k, v, causal=True)
    device_status()
    want, _ = attention_f64(to_numpy(q.contiguous()), to_numpy(k.contiguous()), to_numpy(v.contiguous()), True)
    np.testing.assert_allclose(to_numpy(o).astype(np.float64), want, rtol=TOL, atol=TOL)


def test_forward_at_benchmark_length(cuda):
    """Sequence 4096, head dim 128, causal (the benchmark shape at batch 1, 2 heads): against float64."""
    q, k, v = qkv(1, 4096, 4096, 2, 2, 128)
    o, lse = attention_forward(to_torch(q, cuda), to_torch(k, cuda), to_torch(v, cuda), causal=True)
    device_status()
    want, want_lse = attention_f64(q, k, v, True)
    np.testing.assert_allclose(to_numpy(o).astype(np.float64), want, rtol=TOL, atol=TOL)
    np.testing.assert_allclose(to_numpy(lse), want_lse, rtol=1e-3, atol=1e-3)
    # size-independent property: a row's output is a convex combination of value rows
    assert np.isfinite(to_numpy(o).astype(np.float32)).all()
    assert float(np.abs(to_numpy(o).astype(np.float32)).max()) <= float(np.abs(v.astype(np.float32)).max()) + 1e-2


def close(got, want, tol=TOL):
    """rtol = atol = tol with atol scaled by max|want| (tests/functional/test_attention.py:409-413)."""
    want = want.astype(np.float64)
    np.testing.assert_allclose(got.astype(np.float64), want, rtol=tol, atol=tol * max(np.abs(want).max(), 1e-6))


BWD_CASES = [
    ((1, 128, 128, 1, 1, 128), False),
    ((2, 128, 128, 2, 2, 128), True),
    ((1, 256, 256, 2, 2, 64), True),
    ((2, 100, 100, 4, 2, 64), True),
    ((1, 130, 77, 2, 2, 64), False),
    ((1, 70, 200, 2, 1, 128), True),
    ((1, 300, 300, 3, 3, 128), True),
]


@pytest.mark.parametrize("case", BWD_CASES)
def test_backward_matches_the_traced_program(cuda, case):
    """dq, dk, dv against the CPU running the same traced forward+backward program
    (tests/functional/test_attention.py:382-413), including grouped-query heads and ragged lengths."""
    (b, sq, sk, n, nkv, h), causal = case
    q, k, v = qkv(b, sq, sk, n, nkv, h)
    do = bf16(np.random.default_rng(9).standard_normal(q.shape))
    scale = h**-0.5

    def program(q_, k_, v_, do_):
        o, lse = F.attention_forward_prims(q_, k_, v_, scale, causal)
        return F.attention_backward_prims(q_, k_, v_, o, lse, do_, scale, causal)

    g = tracer.trace(program, *[("bfloat16", a.shape) for a in (q, k, v, do)])
    want = run_oracle(g, [q, k, v, do])
    tq, tk, tv, tdo = (to_torch(a, cuda) for a in (q, k, v, do))
    o, lse = attention_forward(tq, tk, tv, causal=causal)
    got = attention_backward(tq, tk, tv, o, tdo, lse, causal=causal)
    device_status()
    for name, a, w in zip(("dq", "dk", "dv"), got, want):
        close(to_numpy(a).astype(np.float32), w.astype(np.float32))


def test_backward_is_deterministic_and_finite_at_benchmark_length(cuda):
    """Sequence 4096, head dim 128, causal: two runs are bit-identical (no atomics;
    tests/functional/test_attention.py:403-407), and dV matches P^T dO recomputed in float64 for one head."""
    q, k, v = qkv(1, 4096, 4096, 2, 2, 128)
    do = bf16(np.random.default_rng(9).standard_normal(q.shape))
    tq, tk, tv, tdo = (to_torch(a, cuda) for a in (q, k, v, do))
    o, lse = attention_forward(tq, tk, tv, causal=True)
    first = attention_backward(tq, tk, tv, o, tdo, lse, causal=True)
    second = attention_backward(tq, tk, tv, o, tdo, lse, causal=True)
    device_status()
    for a, b in zip(first, second):
        assert torch.equal(a, b)
        assert torch.isfinite(a.float()).all()
    qh, kh, vh, doh = (a[0, :, 0].astype(np.float64) for a in (q, k, v, do))
    s = qh @ kh.T / np.sqrt(128)
    s = np.where(np.tril(np.ones((4096, 4096), bool)), s, -np.inf)
    p = np.exp(s - s.max(-1, keepdims=True))
    p /= p.sum(-1, keepdims=True)
    close(to_numpy(first[2])[0, :, 0].astype(np.float32), p.T @ doh)
    dp = doh @ vh.T
    delta = (doh * (p @ vh)).sum(-1, keepdims=True)
    ds = p * (dp - delta) / np.sqrt(128)
    close(to_numpy(first[0])[0, :, 0].astype(np.float32), ds @ kh)
    close(to_numpy(first[1])[0, :, 0].astype(np.float32), ds.T @ qh)


# The shapes the 12-layer training step runs (head dim 64, sequence 2048) and the next length up: 16 to 64 key tiles per
# query tile, so the K/V ring, the barrier parities and the lazy rescaling all wrap many times.
LONG_D64 = [
    ((2, 2048, 2048, 2, 2, 64), True),
    ((1, 2048, 2048, 4, 2, 64), True),   # grouped-query heads 4:2
    ((1, 4096, 4096, 2, 2, 64), True),
    ((1, 2048, 2048, 2, 2, 64), False),
]


@pytest.mark.parametrize("case", LONG_D64)
def test_head_dim_64_at_training_lengths(cuda, case):
    """Forward and backward of the head-dim-64 kernels at the training step's sequence length against float64:
    o, dq, dk, dv within 2e-2 (of the largest value), the log-sum-exp within 1e-3; two backward runs bit-identical."""
    (b, sq, sk, n, nkv, h), causal = case
    q, k, v = qkv(b, sq, sk, n, nkv, h, seed=11)
    do = bf16(np.random.default_rng(12).standard_normal(q.shape))
    tq, tk, tv, tdo = (to_torch(a, cuda) for a in (q, k, v, do))
    o, lse = attention_forward(tq, tk, tv, causal=causal)
    got = attention_backward(tq, tk, tv, o, tdo, lse, causal=causal)
    again = attention_backward(tq, tk, tv, o, tdo, lse, causal=causal)
    device_status()
    want_o, want_lse, want = attention_f64(q, k, v, causal, do)
    close(to_numpy(o).astype(np.float32), want_o)
    np.testing.assert_allclose(to_numpy(lse), want_lse, rtol=1e-3, atol=1e-3)
    for name, a, a2, w in zip(("dq", "dk", "dv"), got, again, want):
        assert torch.equal(a, a2), name
        close(to_numpy(a).astype(np.float32), w)


# The single-kernel backward (head dim 64): ragged lengths, grouped-query heads, Sq != Sk, several query tiles per key
# tile, and the training step's length.
ATOMIC_CASES = [
    ((1, 128, 128, 1, 1, 64), False),
    ((1, 256, 256, 2, 2, 64), True),
    ((2, 100, 100, 4, 2, 64), True),
    ((1, 130, 77, 2, 2, 64), False),
    ((1, 70, 200, 2, 1, 64), True),
    ((1, 300, 300, 3, 3, 64), True),
    ((1, 640, 640, 4, 1, 64), True),   # four query heads accumulate into one kv head over five query tiles
]


@pytest.mark.parametrize("case", ATOMIC_CASES)
def test_single_kernel_backward_matches_the_traced_program(cuda, case):
    """`lb_attention_bwd_atomic` (dQ added atomically into a float32 accumulator, the reference backend's default mode)
    against the CPU running the traced forward+backward program, at the tolerance of the deterministic pair; dK and dV
    are bit-identical between two runs, dQ agrees to the last bfloat16 bits."""
    (b, sq, sk, n, nkv, h), causal = case
    q, k, v = qkv(b, sq, sk, n, nkv, h)
    do = bf16(np.random.default_rng(9).standard_normal(q.shape))
    scale = h**-0.5

    def program(q_, k_, v_, do_):
        o, lse = F.attention_forward_prims(q_, k_, v_, scale, causal)
        return F.attention_backward_prims(q_, k_, v_, o, lse, do_, scale, causal)

    g = tracer.trace(program, *[("bfloat16", a.shape) for a in (q, k, v, do)])
    want = run_oracle(g, [q, k, v, do])
    tq, tk, tv, tdo = (to_torch(a, cuda) for a in (q, k, v, do))
    o, lse = attention_forward(tq, tk, tv, causal=causal)
    got = attention_backward(tq, tk, tv, o, tdo, lse, causal=causal, deterministic=False)
    again = attention_backward(tq, tk, tv, o, tdo, lse, causal=causal, deterministic=False)
    device_status()
    for name, a, a2, w in zip(("dq", "dk", "dv"), got, again, want):
        close(to_numpy(a).astype(np.float32), w.astype(np.float32))
        if name == "dq":
            close(to_numpy(a2).astype(np.float32), to_numpy(a).astype(np.float32), tol=1e-2)
        else:
            assert torch.equal(a, a2), name


@pytest.mark.parametrize("case", LONG_D64)
def test_single_kernel_backward_at_training_lengths(cuda, case):
    """The single-kernel backward at sequence 2048 / 4096 against float64 and against the deterministic pair."""
    (b, sq, sk, n, nkv, h), causal = case
    q, k, v = qkv(b, sq, sk, n, nkv, h, seed=11)
    do = bf16(np.random.default_rng(12).standard_normal(q.shape))
    tq, tk, tv, tdo = (to_torch(a, cuda) for a in (q, k, v, do))
    o, lse = attention_forward(tq, tk, tv, causal=causal)
    got = attention_backward(tq, tk, tv, o, tdo, lse, causal=causal, deterministic=False)
    pair = attention_backward(tq, tk, tv, o, tdo, lse, causal=causal)
    device_status()
    _, _, want = attention_f64(q, k, v, causal, do)
    for name, a, a2, w in zip(("dq", "dk", "dv"), got, pair, want):
        close(to_numpy(a).astype(np.float32), w)
        close(to_numpy(a).astype(np.float32), to_numpy(a2).astype(np.float32), tol=1e-2)


def test_single_kernel_entry_runs_other_head_dims_as_the_pair(cuda):
    """`lb_attention_bwd_atomic` covers head dim 64; at head dim 128 it runs exactly what `lb_attention_bwd` runs
    (the accumulator is left unused), so the results are bit-identical to the deterministic entry's."""
    q, k, v = qkv(1, 256, 256, 2, 2, 128)
    do = bf16(np.random.default_rng(9).standard_normal(q.shape))
    tq, tk, tv, tdo = (to_torch(a, cuda) for a in (q, k, v, do))
    o, lse = attention_forward(tq, tk, tv, causal=True)
    pair = attention_backward(tq, tk, tv, o, tdo, lse, causal=True)
    other = attention_backward(tq, tk, tv, o, tdo, lse, causal=True, deterministic=False)
    device_status()
    for a, b in zip(pair, other):
        assert torch.equal(a, b)


def random_attention_case(seed):
    """Batch 1-3, query and key lengths 1-700 (equal, or ragged either way), 1-6 query heads over a divisor of key/value
    heads, head dim 64 or 128 (the tensor-core kernels) or 32 / 80 (the SIMT kernels), causal or not."""
    rng = np.random.default_rng(seed + 400)
    h = int(rng.choice([64, 64, 128, 128, 32, 80]))
    n = int(rng.choice([1, 2, 3, 4, 6]))
    nkv = int(rng.choice([d for d in (1, 2, 3, 4, 6) if n % d == 0]))
    sq = int(rng.choice([1, 17, 64, 127, 128, 129, 255, 256, 300, 513, 700]))
    sk = sq if rng.random() < 0.5 else int(rng.choice([1, 17, 64, 127, 128, 129, 255, 256, 300, 513, 700]))
    causal = bool(rng.random() < 0.6)
    if causal and sk < sq:
        sk = sq  # a causal mask aligned to the last key needs at least as many keys as queries
    return (int(rng.integers(1, 4)), sq, sk, n, nkv, h), causal


@pytest.mark.parametrize("seed", range(32))
def test_random_attention_shapes_against_float64(cuda, seed):
    """Forward and both backward forms (the deterministic pair; the single kernel with atomic dQ, which head dim 64
    takes) on random shapes against float64: o, dq, dk, dv within 2e-2 (of the value and of the largest value), the
    log-sum-exp within 1e-3; the deterministic backward repeats bit for bit."""
    (b, sq, sk, n, nkv, h), causal = random_attention_case(seed)
    q, k, v = qkv(b, sq, sk, n, nkv, h, seed=seed + 50)
    do = bf16(np.random.default_rng(seed + 60).standard_normal(q.shape))
    tq, tk, tv, tdo = (to_torch(a, cuda) for a in (q, k, v, do))
    o, lse = attention_forward(tq, tk, tv, causal=causal)
    pair = attention_backward(tq, tk, tv, o, tdo, lse, causal=causal)
    again = attention_backward(tq, tk, tv, o, tdo, lse, causal=causal)
    single = attention_backward(tq, tk, tv, o, tdo, lse, causal=causal, deterministic=False)
    device_status()
    want_o, want_lse, grads = attention_f64(q, k, v, causal, do)
    close(to_numpy(o).astype(np.float32), want_o)
    np.testing.assert_allclose(to_numpy(lse), want_lse, rtol=1e-3, atol=1e-3)
    for name, a, a2, s, w in zip(("dq", "dk", "dv"), pair, again, single, grads):
        # with a single key the probabilities are 1 and dq, dk are exactly zero: the tolerance is then 2e-2 of the
        # operands' unit scale times bfloat16's epsilon rather than of a zero maximum
        for result in (a, s):
            np.testing.assert_allclose(to_numpy(result).astype(np.float64), w, rtol=TOL, atol=TOL * max(np.abs(w).max(), 2.0**-8), err_msg=name)
        assert torch.equal(a, a2), name


# (B, Sq, Sk, N, Nkv, H): the CUDA-core kernels' edges - rows per CTA (8), streamed chunks (32), head-dim elements per lane
SIMT_CASES = [((1, 8, 32, 1, 1, 32), True), ((2, 9, 33, 2, 1, 33), True), ((1, 7, 31, 3, 3, 1), False), ((1, 65, 64, 2, 2, 65), False),
              ((1, 40, 40, 4, 2, 129), True), ((1, 33, 70, 1, 1, 256), True)]


# ... and of few rows with few to stream: tiles of as many rows as are streamed
SIMT_SHORT_CASES = [((40, 1, 1, 8, 8, 256), True), ((3, 2, 5, 4, 2, 128), False), ((2, 3, 16, 2, 1, 64), True), ((2, 5, 17, 2, 1, 64), True),
                    ((2, 16, 3, 2, 2, 200), False), ((1, 31, 31, 2, 1, 256), True)]


@pytest.mark.parametrize("case", SIMT_CASES + SIMT_SHORT_CASES)
def test_cuda_core_attention_against_float64(cuda, case):
    """float32 operands: every result within 2e-5 of its largest value. A score is a float32 sum of H <= 256 products of
    size about 1 / sqrt(H) each (error under 256 * 2^-24 = 1.5e-5 of a score, typically its square root), and __expf is
    accurate to 2 ulp + 2^-21 |x|."""
    (b, sq, sk, n, nkv, h), causal = case
    rng = np.random.default_rng(h)
    q, k, v, do = (rng.standard_normal(s).astype(np.float32) for s in ((b, sq, n, h), (b, sk, nkv, h), (b, sk, nkv, h), (b, sq, n, h)))
    tq, tk, tv, tdo = (to_torch(x, cuda) for x in (q, k, v, do))
    o, lse = attention_forward(tq, tk, tv, causal=causal)
    grads = attention_backward(tq, tk, tv, o, tdo, lse, causal=causal)
    device_status()
    x = [torch.from_numpy(a.astype(np.float64)).requires_grad_(True) for a in (q, k, v)]
    qq, kk, vv = x[0].transpose(1, 2), x[1].repeat_interleave(n // nkv, 2).transpose(1, 2), x[2].repeat_interleave(n // nkv, 2).transpose(1, 2)
    s = qq @ kk.transpose(-1, -2) * h**-0.5
    if causal:
        s = s.masked_fill(torch.arange(sk)[None, :] > torch.arange(sq)[:, None] + sk - sq, float("-inf"))
    out = (torch.softmax(s, -1) @ vv).transpose(1, 2)
    out.backward(torch.from_numpy(do.astype(np.float64)))
    for name, got, want in zip(("o", "lse", "dq", "dk", "dv"), (o, lse, *grads), (out, torch.logsumexp(s, -1), *(t.grad for t in x))):
        want = want.detach().numpy()
        assert np.abs(to_numpy(got) - want).max() <= 2e-5 * max(np.abs(want).max(), 1.0), name


# (B, Sq, Sk, N, Nkv, H): few query rows per key head - one and two 16-row tiles, one key, ragged slices of 16 keys, fewer
# slices than warps, one and many CTAs per key head, positions that see different numbers of keys
DECODE_CASES = [((1, 1, 1, 1, 1, 64), False), ((2, 1, 17, 4, 4, 128), True), ((1, 1, 4097, 8, 1, 128), True), ((3, 4, 1000, 8, 2, 64), True),
                ((1, 4, 333, 16, 4, 128), True), ((2, 2, 2050, 32, 2, 128), True), ((1, 16, 40, 2, 1, 64), False), ((1, 5, 3, 2, 2, 64), False),
                ((40, 1, 129, 16, 16, 64), True), ((1, 1, 16384, 2, 2, 128), True), ((1, 32, 32, 1, 1, 64), True)]


# ... that the choice of kernel sends to the one for few rows, with two 16-row tiles (17 to 32 rows per key head)
TWO_ROW_TILES = [((1, 17, 4000, 2, 2, 64), True), ((1, 32, 16384, 4, 4, 128), True), ((2, 3, 2070, 32, 4, 64), True), ((1, 5, 3001, 5, 1, 128), False),
                 ((1, 1, 3000, 32, 1, 128), True)]


@pytest.mark.parametrize("case", DECODE_CASES + TWO_ROW_TILES)
def test_few_query_rows_against_float64(cuda, case):
    """The reference's 16-bit tolerance (2e-2), log-sum-exp to 1e-3, on strided views."""
    (b, sq, sk, n, nkv, h), causal = case
    if case in TWO_ROW_TILES:
        assert attention_kernel(*case[0], causal) == "few rows"
    q, k, v = qkv(b, sq, sk, n, nkv, h)
    cache = torch.empty((b, sk, 2, nkv, h), dtype=torch.bfloat16, device=cuda)
    cache[:, :, 0], cache[:, :, 1] = to_torch(k, cuda), to_torch(v, cuda)
    o, lse = attention_forward(to_torch(q, cuda), cache[:, :, 0], cache[:, :, 1], causal=causal)
    device_status()
    want, want_lse = attention_f64(q, k, v, causal)
    np.testing.assert_allclose(to_numpy(o).astype(np.float64), want, rtol=TOL, atol=TOL)
    np.testing.assert_allclose(to_numpy(lse), want_lse, rtol=1e-3, atol=1e-3)


# (B, Sq, Sk, N, Nkv, H): the backward's 128-row streamed tiles at head dim 128 - one row of a second tile on either side, rings
# that wrap (more tiles than stages), a group of heads walked by one CTA, more keys than queries, keys no query sees
TILE_EDGE_CASES = [((1, 129, 129, 1, 1, 128), True), ((1, 1, 129, 2, 1, 128), False), ((1, 128, 257, 2, 2, 128), True), ((1, 641, 640, 4, 1, 128), False),
                   ((2, 900, 1030, 4, 2, 128), True), ((1, 40, 400, 1, 1, 128), True)]


# ... and those of its 64-row tiles, which one, three and five blocks of 64 streamed rows take on either side
SHORT_CASES = [((1, 1, 1, 1, 1, 128), False), ((2, 64, 64, 4, 1, 128), True), ((1, 65, 64, 2, 2, 128), False), ((2, 129, 130, 4, 2, 128), True), ((1, 192, 320, 2, 1, 128), True),
               ((1, 320, 300, 4, 4, 128), False), ((1, 321, 384, 1, 1, 128), True), ((3, 20, 500, 8, 2, 128), True)]


@pytest.mark.parametrize("case", TILE_EDGE_CASES + SHORT_CASES)
def test_backward_tile_edges_against_float64(cuda, case):
    """The reference's 16-bit tolerance (2e-2 of the value and of the largest), bit-identical from run to run."""
    (b, sq, sk, n, nkv, h), causal = case
    q, k, v = qkv(b, sq, sk, n, nkv, h)
    do = bf16(np.random.default_rng(4).standard_normal(q.shape))
    tq, tk, tv, tdo = (to_torch(a, cuda) for a in (q, k, v, do))
    o, lse = attention_forward(tq, tk, tv, causal=causal)
    got = attention_backward(tq, tk, tv, o, tdo, lse, causal=causal)
    again = attention_backward(tq, tk, tv, o, tdo, lse, causal=causal)
    device_status()
    for a, a2, w in zip(got, again, attention_f64(q, k, v, causal, do)[2]):
        close(to_numpy(a).astype(np.float32), w)
        assert torch.equal(a, a2)


# (B, Sq, Sk, N, Nkv, H): enough query tiles for the two-tile forward kernel (more than two per SM at head dim 128, four at
# 64) - a second tile of one row, a last CTA with one tile, a key tail, more keys than queries, CTAs that go on to further
# work with more and with fewer key tiles
PAIR_CASES = [((20, 129, 129, 16, 4, 128), True), ((10, 257, 257, 16, 16, 128), False), ((2, 300, 777, 64, 8, 128), True), ((1, 1024, 1024, 40, 8, 128), True),
              ((20, 129, 129, 32, 4, 64), True), ((10, 257, 257, 32, 16, 64), False), ((4, 300, 500, 64, 8, 64), True), ((2, 1100, 1100, 40, 8, 64), True)]


# ... that the choice of kernel sends to the two-tile kernel
TWO_TILE_CASES = [((20, 129, 129, 32, 4, 64), True), ((4, 385, 500, 40, 8, 64), True), ((1, 1200, 1337, 40, 8, 64), True), ((20, 255, 255, 16, 4, 128), False),
                  ((2, 639, 777, 64, 8, 128), False), ((1, 1024, 1024, 40, 8, 128), True), ((40, 129, 513, 16, 4, 128), True)]


@pytest.mark.parametrize("case", PAIR_CASES + TWO_TILE_CASES)
def test_two_tile_forward_against_float64(cuda, case):
    """The reference's 16-bit tolerance (2e-2), log-sum-exp to 1e-3. Later keys have larger scores, so that the reference
    maximum is raised on the way (a factor of 2^8 between raises), and the result repeats bit for bit."""
    (b, sq, sk, n, nkv, h), causal = case
    if case in TWO_TILE_CASES:
        assert attention_kernel(*case[0], causal) == "two tiles"
    q, k, v = qkv(b, sq, sk, n, nkv, h)
    k = bf16(k.astype(np.float32) * np.linspace(0.1, 6.0, sk, dtype=np.float32)[None, :, None, None])
    tq, tk, tv = (to_torch(a, cuda) for a in (q, k, v))
    o, lse = attention_forward(tq, tk, tv, causal=causal)
    again, _ = attention_forward(tq, tk, tv, causal=causal)
    device_status()
    want, want_lse = attention_f64(q, k, v, causal)
    close(to_numpy(o).astype(np.float32), want)
    np.testing.assert_allclose(to_numpy(lse), want_lse, rtol=1e-3, atol=1e-3)
    assert torch.equal(o, again)


@pytest.mark.parametrize("n", [2, 40])
def test_forward_rows_that_see_no_key_and_rows_of_nan(cuda, n):
    """One and two query tiles per CTA: a causal mask aligned to the last of fewer keys leaves the first rows none (0 / 0 in
    the traced program); a NaN key makes the rows that see it NaN and no other."""
    q, k, v = (to_torch(a, cuda) for a in qkv(4, 300, 200, n, n, 128))
    o, lse = attention_forward(q, k, v, causal=True)
    device_status()
    assert torch.isnan(o[:, :100]).all() and not torch.isnan(o[:, 100:]).any() and not torch.isnan(lse[..., 100:]).any()
    k[:, 150] = float("nan")
    o, _ = attention_forward(q, k, v, causal=True)
    device_status()
    assert torch.isnan(o[:, 250:]).all() and not torch.isnan(o[:, 100:250]).any()


@pytest.mark.parametrize("h", [64, 128])
def test_log_sum_exp_of_few_rows_is_as_exact_as_of_many(cuda, h):
    """The same query rows through the kernel for few rows and, repeated over 64 positions, through the tile kernel: the
    former cuts the keys into ranges and may not pay for it with a larger error of the (float32) log-sum-exp. 512 rows:
    the root mean square of an error varies by 1 / sqrt(2 * 512) = 3 % from sample to sample; three of these are allowed."""
    b, sk, n, nkv = 16, 1394, 32, 4
    q, k, v = qkv(b, 1, sk, n, nkv, h)
    want = attention_f64(q, k, v, False)[1]
    tq, tk, tv = (to_torch(a, cuda) for a in (q, k, v))
    _, few = attention_forward(tq, tk, tv)
    _, many = attention_forward(tq.expand(b, 64, n, h).contiguous(), tk, tv)
    device_status()

    def rms(lse):
        return float(np.sqrt(np.mean((to_numpy(lse)[:, :, :1].astype(np.float64) - want) ** 2)))

    assert rms(few) <= 1.09 * rms(many)


@pytest.mark.parametrize("h", [32, 64, 128, 256])
def test_cuda_core_scores_are_as_exact_as_a_warp_wide_sum(cuda, h):
    """The error of a score, seen in the log-sum-exp of a peaked softmax, against that of scores summed by a warp: lane l adds the
    products of elements l, l + 32, ... one by one, then the lanes are added as a tree of five (emulated here, a float64
    multiply-add rounded to float32 being a fused one). 1600 rows: a root mean square varies by 1 / sqrt(3200) = 1.8 %; a tenth
    is allowed. Two running sums a score, as the kernel once had, are 1.3 to 2.3 times that at 64 to 256 elements."""
    b, s, n = 2, 200, 4
    rng = np.random.default_rng(h)
    q, k, v = (rng.standard_normal((b, s, n, h)).astype(np.float32) for _ in range(3))
    q *= 6.0
    _, lse = attention_forward(*(to_torch(x, cuda) for x in (q, k, v)), causal=True)
    device_status()
    lanes = torch.zeros((b, n, s, s, 32), dtype=torch.float32, device=cuda)
    for u in range(0, h, 32):
        x, y = (to_torch(a[..., u : u + 32], cuda).double().transpose(1, 2) for a in (q, k))
        lanes = (x[:, :, :, None] * y[:, :, None] + lanes.double()).float()
    for m in (16, 8, 4, 2, 1):
        lanes = lanes[..., :m] + lanes[..., m:]
    scores = (lanes[..., 0] * np.float32(h**-0.5)).double().masked_fill(torch.ones((s, s), dtype=torch.bool, device=cuda).triu(1), float("-inf"))
    want = attention_f64(q, k, v, True)[1]

    def rms(x):
        return float(np.sqrt(np.mean((to_numpy(x).astype(np.float64) - want) ** 2)))

    assert rms(lse) <= 1.1 * rms(torch.logsumexp(scores, -1).float())


@pytest.mark.parametrize("h,dtype", [(32, "float32"), (128, "float32"), (200, "float32"), (80, "bfloat16")])
def test_cuda_core_attention_keeps_masked_rows_of_nan_out(cuda, h, dtype):
    """A causal mask: a NaN in a value, key, query or gradient row reaches the rows that see it (or that it sees) and no other,
    wherever the rows lie in their blocks of eight and chunks of 32."""
    s = 70
    rng = np.random.default_rng(h)
    q, k, v, do = (to_torch(rng.standard_normal((1, s, 2, h)).astype(np.float32), cuda).to(getattr(torch, dtype)) for _ in range(4))
    o, lse = attention_forward(q, k, v, causal=True)
    nan = float("nan")

    def with_nan(x, row):
        x = x.clone()
        x[:, row] = nan
        return x

    def rows_of_nan(x):
        return torch.isnan(x).flatten(2).any(2)[0].nonzero().flatten().tolist()

    for at in (0, 5, 31, 37, 64):
        assert rows_of_nan(attention_forward(q, k, with_nan(v, at), causal=True)[0]) == list(range(at, s))
        dq, _, _ = attention_backward(q, with_nan(k, at), v, o, do, lse, causal=True)
        assert rows_of_nan(dq) == list(range(at, s))
        _, dk, dv = attention_backward(with_nan(q, at), k, v, o, do, lse, causal=True)
        assert rows_of_nan(dk) == list(range(at + 1)) and rows_of_nan(dv) == list(range(at + 1))
        _, dk, dv = attention_backward(q, k, v, o, with_nan(do, at), lse, causal=True)
        assert rows_of_nan(dk) == list(range(at + 1)) and rows_of_nan(dv) == list(range(at + 1))
    device_status()


@pytest.mark.parametrize("sq", [1, 32, 64])
def test_attention_without_keys_is_refused(cuda, sq):
    q, k = (torch.zeros((1, s, 2, 64), dtype=torch.bfloat16, device=cuda) for s in (sq, 0))
    with pytest.raises(LumenError):
        attention_forward(q, k, k)


def test_two_tiles_rows_that_see_no_key_and_rows_of_nan(cuda):
    """As the test above, on a problem that the two-tile kernel takes."""
    assert attention_kernel(12, 400, 300, 32, 32, 128) == "two tiles"
    q, k, v = (to_torch(a, cuda) for a in qkv(12, 400, 300, 32, 32, 128))
    o, lse = attention_forward(q, k, v, causal=True)
    device_status()
    assert torch.isnan(o[:, :100]).all() and not torch.isnan(o[:, 100:]).any() and not torch.isnan(lse[..., 100:]).any()
    k[:, 150] = float("nan")
    o, _ = attention_forward(q, k, v, causal=True)
    device_status()
    assert torch.isnan(o[:, 250:]).all() and not torch.isnan(o[:, 100:250]).any()


@pytest.mark.parametrize("h", [64, 128])
def test_backward_leaves_blocks_behind_the_mask_out(cuda, h):
    """Blocks of 64 rows that a tile of 128 does not see at all (more keys than queries, so that the mask's edge lies 64 off the
    tiles) do not enter it: a NaN there changes no bit of its gradients."""
    q, k, v, do = (to_torch(bf16(np.random.default_rng(i).standard_normal((1, s, 2, h))), cuda) for i, s in enumerate((200, 264, 264, 200)))
    o, lse = attention_forward(q, k, v, causal=True)
    dq, dk, dv = attention_backward(q, k, v, o, do, lse, causal=True)
    for name in ("q", "do"):
        t = {"q": q.clone(), "do": do.clone()}
        t[name][:, 10] = float("nan")  # sees keys up to 74: the second tile of keys starts at 128
        _, dk2, dv2 = attention_backward(t["q"], k, v, o, t["do"], lse, causal=True)
        assert torch.equal(dk2[:, 128:], dk[:, 128:]) and torch.equal(dv2[:, 128:], dv[:, 128:])
    k2 = k.clone()
    k2[:, 200] = float("nan")  # seen from query 136 on: the first tile of queries ends at 127
    dq2, _, _ = attention_backward(q, k2, v, o, do, lse, causal=True)
    device_status()
    assert torch.equal(dq2[:, :128], dq[:, :128]) and torch.isnan(dq2[:, 136:]).all()
