"""Parity of lb_gemm with the oracle's dot_general, small shapes and large: the CUDA-core kernel accumulates in the interpreter's order and
is bit-exact; the tcgen05 kernel sums in tensor-core order and is held to the reference's bf16 tolerance."""

import numpy as np
import pytest
import torch

from lumen_b200 import functional as F
from lumen_b200 import tracer
from lumen_b200.runtime import device_status, gemm, gemm_scratch_bytes
from tests.helpers import bf16, run_oracle, to_numpy, to_torch

pytestmark = pytest.mark.gpu


def operands(m, n, k, seed, batch=None):
    rng = np.random.default_rng(seed)
    lead = () if batch is None else (batch,)
    a = (rng.standard_normal(lead + (m, k)) / np.sqrt(k)).astype(np.float32)
    b = (rng.standard_normal(lead + (k, n)) / np.sqrt(k)).astype(np.float32)
    return a, b


def oracle_matmul(a, b, dtype, out_dtype):
    g = tracer.trace(lambda x, y: F.matmul(x, y, "float32", out_dtype), (dtype, a.shape), (dtype, b.shape))
    return run_oracle(g, [a, b])[0]


@pytest.mark.parametrize("shape", [(64, 48, 40), (130, 70, 33), (1, 5, 7)])
def test_float32_gemm_is_bit_exact(cuda, shape):
    """float32 operands: products and sums rounded one by one in contracting order (lumen/reference/mod.rs:958-970)."""
    m, n, k = shape
    a, b = operands(m, n, k, 0)
    out = torch.empty((m, n), dtype=torch.float32, device=cuda)
    gemm(to_torch(a, cuda), to_torch(b, cuda), out)
    np.testing.assert_array_equal(to_numpy(out), oracle_matmul(a, b, "float32", "float32"))


@pytest.mark.parametrize("shape", [(300, 320, 1), (1100, 1121, 3), (400, 410, 15), (40, 70, 63), (16, 32, 64), (17, 33, 65), (400, 410, 70), (416, 384, 128), (1100, 1121, 33), (1152, 1152, 64)])
@pytest.mark.parametrize("majors", ["nn", "nt", "tn", "tt"])
def test_float32_gemm_tiles_and_majors_are_bit_exact(cuda, shape, majors):
    """Each tile size the CUDA-core kernel picks (few, some, many output tiles), whole and ragged, with either operand
    contiguous along either axis (aligned groups of four and element by element)."""
    m, n, k = shape
    a, b = operands(m, n, k, 5)
    ta, tb = (to_torch(x if major == "n" else np.ascontiguousarray(x.T), cuda) for x, major in zip((a, b), majors))
    out = torch.full((m, n), float("nan"), dtype=torch.float32, device=cuda)
    gemm(ta if majors[0] == "n" else ta.t(), tb if majors[1] == "n" else tb.t(), out)
    np.testing.assert_array_equal(to_numpy(out), oracle_matmul(a, b, "float32", "float32"))


def test_simt_bf16_gemm_is_bit_exact(cuda):
    a, b = operands(96, 80, 72, 1)
    a, b = bf16(a), bf16(b)
    for out_dtype, td in (("float32", torch.float32), ("bfloat16", torch.bfloat16)):
        out = torch.empty((96, 80), dtype=td, device=cuda)
        gemm(to_torch(a, cuda), to_torch(b, cuda), out, kernel="simt")
        want = oracle_matmul(a, b, "bfloat16", out_dtype)
        np.testing.assert_array_equal(to_numpy(out).astype(np.float32), want.astype(np.float32))


MAJORS = [("row", "row"), ("row", "col"), ("col", "row"), ("col", "col")]


def with_major(x, major, cuda):
    """A [.., R, C] device tensor whose memory is row-major ("row") or column-major ("col")."""
    t = to_torch(x, cuda)
    if major == "col":
        t = t.transpose(-1, -2).contiguous().transpose(-1, -2)
    return t


@pytest.mark.parametrize("kernel", ["tcgen05", "tcgen05_1cta"])
@pytest.mark.parametrize("majors", MAJORS)
@pytest.mark.parametrize("shape", [(128, 256, 64), (256, 512, 320), (200, 264, 136), (384, 1000, 72), (8, 8, 8), (1152, 520, 448)])
def test_tcgen05_gemm_all_majors(cuda, shape, majors, kernel):
    """Both tensor-core kernels (CTA pairs for M > 128 under "tcgen05", one CTA per tile under "tcgen05_1cta"),
    every operand major (the transposed views of the backward GEMMs), ragged edges in M, N and K: float32
    outputs differ from the oracle only by the order of the float32 sums, so they are held to 1e-4 (far inside the
    reference's 1e-2 * max|want| for bf16 operands, tests/codegen/test_dot_general.py:41-42,168-169)."""
    m, n, k = shape
    a, b = operands(m, n, k, 2)
    a, b = bf16(a), bf16(b)
    want = oracle_matmul(a, b, "bfloat16", "float32")
    out = torch.full((m, n), float("nan"), dtype=torch.float32, device=cuda)
    gemm(with_major(a, majors[0], cuda), with_major(b, majors[1], cuda), out, kernel=kernel)
    device_status()
    got = to_numpy(out)
    np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-4 * np.abs(want).max())
    assert np.abs(got - want).max() <= 1e-2 * np.abs(want).max()


def test_tcgen05_gemm_bf16_output_batched_relu(cuda):
    a, b = operands(192, 320, 128, 3, batch=3)
    a, b = bf16(a), bf16(b)
    want = oracle_matmul(a, b, "bfloat16", "float32")
    out = torch.empty((3, 192, 320), dtype=torch.bfloat16, device=cuda)
    gemm(to_torch(a, cuda), to_torch(b, cuda), out, epilogue="relu", kernel="tcgen05")
    device_status()
    want = np.maximum(want, 0)
    np.testing.assert_allclose(to_numpy(out).astype(np.float32), want, rtol=2**-6, atol=2**-6 * np.abs(want).max())


def test_tcgen05_matches_exact_accumulation_at_large_k(cuda):
    """K = 4096 over several waves of tiles, against the ORACLE's dot_general on the same operands: the CUDA-core
    kernel (the interpreter's order) bit for bit, the tensor-core result within 1e-3 of the largest value; and linearity
    in A as a size-independent property."""
    m, n, k = 1024, 2048, 4096
    a, b = operands(m, n, k, 4)
    want = oracle_matmul(bf16(a), bf16(b), "bfloat16", "float32")
    a_t, b_t = to_torch(bf16(a), cuda), to_torch(bf16(b), cuda)
    fast = torch.empty((m, n), dtype=torch.float32, device=cuda)
    exact = torch.empty((m, n), dtype=torch.float32, device=cuda)
    gemm(a_t, b_t, fast, kernel="tcgen05")
    gemm(a_t, b_t, exact, kernel="simt")
    device_status()
    np.testing.assert_array_equal(to_numpy(exact), want)
    scale = float(np.abs(want).max())
    assert float(np.abs(to_numpy(fast) - want).max()) <= 1e-3 * scale
    doubled = torch.empty_like(fast)
    gemm(a_t * 2, b_t, doubled, kernel="tcgen05")
    torch.testing.assert_close(doubled, fast * 2, rtol=0, atol=0)


@pytest.mark.parametrize("shape", [(256, 512, 8192), (1024, 1024, 16384), (200, 264, 4104)])
def test_split_k_weight_gradient_shapes(cuda, shape):
    """Few output tiles and a long K (dW = dY^T X with both operands transposed views): K is cut into ranges,
    partial tiles are added in a fixed order. Same tolerance as the unsplit kernel, bf16 output, reproducible."""
    m, n, k = shape
    rng = np.random.default_rng(5)
    a = bf16(rng.standard_normal((k, m)) / np.sqrt(k))  # stored [K, M]: A = a.T is a transposed view
    b = bf16(rng.standard_normal((k, n)))
    nbytes = gemm_scratch_bytes(m, n, k)
    assert nbytes > 0
    scratch = torch.empty(nbytes, dtype=torch.uint8, device=cuda)
    a_t, b_t = to_torch(a, cuda), to_torch(b, cuda)
    split = torch.empty((m, n), dtype=torch.bfloat16, device=cuda)
    whole = torch.empty((m, n), dtype=torch.float32, device=cuda)
    gemm(a_t.t(), b_t, split, kernel="tcgen05", scratch=scratch)
    gemm(a_t.t(), b_t, whole, kernel="simt")
    device_status()
    want = oracle_matmul(np.ascontiguousarray(a.T), b, "bfloat16", "float32")  # the oracle's dot_general on the same operands
    np.testing.assert_array_equal(to_numpy(whole), want)
    np.testing.assert_allclose(to_numpy(split).astype(np.float32), want, rtol=2**-7, atol=2**-7 * np.abs(want).max())
    again = torch.empty_like(split)
    gemm(a_t.t(), b_t, again, kernel="tcgen05", scratch=scratch)
    assert torch.equal(split, again)


@pytest.mark.parametrize("kernel", ["tcgen05", "tcgen05_1cta"])
@pytest.mark.parametrize("shape", [(384, 512, 256), (200, 264, 136), (256, 512, 8192)])
@pytest.mark.parametrize("epilogue", ["add", "mask_positive"])
def test_tcgen05_gemm_add_and_mask_epilogues(cuda, shape, epilogue, kernel):
    """The elementwise tails a `dot_general` fusion carries into the GEMM: `other + product` (a residual add) and
    `other > 0 ? product : 0` (a relu's backward), on aligned, ragged and split-K shapes. The product is rounded to
    bfloat16 first, as its own primitive; the reference value applies the tail to the CUDA-core kernel's exactly
    accumulated, rounded product, so the two differ only where tensor-core summation order moved a rounding."""
    m, n, k = shape
    rng = np.random.default_rng(11)
    a, b = bf16(rng.standard_normal((m, k)) / np.sqrt(k)), bf16(rng.standard_normal((k, n)))
    other = bf16(rng.standard_normal((m, n)))
    a_t, b_t, o_t = to_torch(a, cuda), to_torch(b, cuda), to_torch(other, cuda)
    nbytes = gemm_scratch_bytes(m, n, k)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device=cuda) if nbytes else None
    got = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device=cuda)
    gemm(a_t, b_t, got, epilogue=epilogue, aux=o_t, kernel=kernel, scratch=scratch)
    exact = torch.empty((m, n), dtype=torch.bfloat16, device=cuda)
    gemm(a_t, b_t, exact, kernel="simt")
    device_status()
    np.testing.assert_array_equal(to_numpy(exact), oracle_matmul(a, b, "bfloat16", "bfloat16"))  # the oracle's rounded product
    product, oth = exact.float(), o_t.float()
    want = (oth + product).bfloat16().float() if epilogue == "add" else torch.where(oth > 0, product, torch.zeros_like(product))
    scale = float(want.abs().max())
    torch.testing.assert_close(got.float(), want, rtol=2**-6, atol=2**-6 * scale)
    if epilogue == "mask_positive":
        assert torch.equal(got.float() == 0, (oth <= 0) | (got.float() == 0)) and bool(((got.float() == 0) | (oth > 0)).all())


def test_gemm_epilogue_operand_is_checked(cuda):
    a = torch.zeros((256, 64), dtype=torch.bfloat16, device=cuda)
    b = torch.zeros((64, 256), dtype=torch.bfloat16, device=cuda)
    out = torch.zeros((256, 256), dtype=torch.bfloat16, device=cuda)
    with pytest.raises(Exception, match="epilogue"):
        gemm(a, b, out, epilogue="add")
    with pytest.raises(Exception, match="shape"):
        gemm(a, b, out, epilogue="add", aux=torch.zeros((256, 128), dtype=torch.bfloat16, device=cuda))


def test_benchmark_size_checksums(cuda):
    """8192 x 8192 x 8192 (the matmul benchmark's forward and both backward products), checked through properties
    that need no full-size reference: the column sums of A B equal (column sums of A) B and the row sums equal
    A (row sums of B), both evaluated in float64 from the same bfloat16 operands; a sampled block of the output
    equals the oracle's product of the matching operand slices."""
    n = 8192
    gen = torch.Generator(device=cuda).manual_seed(2)
    a = (torch.randn((n, n), generator=gen, device=cuda) / n**0.5).bfloat16()
    b = (torch.randn((n, n), generator=gen, device=cuda) / n**0.5).bfloat16()
    dy = torch.randn((n, n), generator=gen, device=cuda).bfloat16()
    y = torch.empty((n, n), dtype=torch.float32, device=cuda)
    da = torch.empty((n, n), dtype=torch.bfloat16, device=cuda)
    db = torch.empty((n, n), dtype=torch.bfloat16, device=cuda)
    gemm(a, b, y)
    gemm(dy, b.t(), da)  # dA = dY B^T
    gemm(a.t(), dy, db)  # dB = A^T dY
    device_status()
    for left, right, out, tol in ((a, b, y, 1e-4), (dy, b.t(), da, 2**-7), (a.t(), dy, db, 2**-7)):
        l64, r64, o64 = left.double(), right.double(), out.double()
        cols = l64.sum(0) @ r64
        rows = l64 @ r64.sum(1)
        scale = float(o64.abs().max()) * n**0.5  # a sum of n outputs, each off by at most tol * max|out|
        assert float((o64.sum(0) - cols).abs().max()) <= tol * scale
        assert float((o64.sum(1) - rows).abs().max()) <= tol * scale
        # a [128, 256] block of the output against the oracle's dot_general of the matching operand slices
        want = oracle_matmul(to_numpy(left[4096:4224].contiguous()), to_numpy(right[:, 7936:8192].contiguous()), "bfloat16", "float32")
        block = to_numpy(out[4096:4224, 7936:8192].float())
        assert float(np.abs(block - want).max()) <= tol * float(np.abs(want).max())


@pytest.mark.parametrize("kernel", ["tcgen05", "tcgen05_1cta"])
def test_tcgen05_gemm_takes_float16_operands(cuda, kernel):
    """float16 operands on the tensor-core kernels (the MMA's operand-format bit): float32 and float16 outputs, a
    transposed operand and a ragged shape, against the oracle's float16 dot_general
    (tests/codegen/test_dot_general.py:128-169 runs the same dtypes)."""
    m, n, k = 264, 328, 200
    a, b = operands(m, n, k, 7)
    a, b = a.astype(np.float16), b.astype(np.float16)
    want = oracle_matmul(a, b, "float16", "float32")
    out = torch.full((m, n), float("nan"), dtype=torch.float32, device=cuda)
    gemm(to_torch(a, cuda), to_torch(np.ascontiguousarray(b.T), cuda).t(), out, kernel=kernel)
    device_status()
    np.testing.assert_allclose(to_numpy(out), want, rtol=1e-4, atol=1e-4 * np.abs(want).max())
    narrow = torch.full((m, n), float("nan"), dtype=torch.float16, device=cuda)
    gemm(to_torch(a, cuda), to_torch(b, cuda), narrow, epilogue="relu", kernel=kernel)
    device_status()
    want16 = np.maximum(want, 0).astype(np.float16).astype(np.float32)
    np.testing.assert_allclose(to_numpy(narrow).astype(np.float32), want16, rtol=2**-9, atol=2**-9 * np.abs(want16).max())


# (batch, M, N, K): the narrow tiles' edges - one element, one row past a tile, N that is no multiple of 8, a K tail, 1 to 8 K
# ranges in a cluster, two CTAs per SM, batches
NARROW_CASES = [(1, 1, 8, 8), (1, 129, 72, 200), (1, 128, 64, 64), (1, 200, 136, 1096), (1, 300, 1000, 512), (1, 64, 64, 2056), (1, 1100, 1024, 4608),
                (3, 130, 200, 264)]


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("majors", ["kn", "kk", "mn", "mk"])
@pytest.mark.parametrize("case", NARROW_CASES)
def test_narrow_tiles_against_float64(cuda, case, majors, dtype):
    """Products of the automatically chosen kernel in every operand order, float32 and rounded outputs and epilogues: a
    float32 sum of K terms of size 1/sqrt(K) is off by less than sqrt(K) * 2^-24 * 4 of the largest result, a rounded one by a
    unit in the last place more; bit-identical from run to run."""
    b, m, n, k = case
    if (majors[0] == "m" and m % 8) or (majors[1] == "n" and n % 8):
        m, n = (m + 7) // 8 * 8, (n + 7) // 8 * 8  # a contiguous axis has to be a multiple of 16 bytes
    if majors in ("kk", "kn", "mk") and k % 8:
        k = (k + 7) // 8 * 8
    gen = torch.Generator(device=cuda).manual_seed(7)
    t = getattr(torch, dtype)
    a = (torch.randn((b, m, k) if majors[0] == "k" else (b, k, m), generator=gen, device=cuda) / k**0.5).to(t)
    w = torch.randn((b, k, n) if majors[1] == "n" else (b, n, k), generator=gen, device=cuda).to(t)
    a, w = a if majors[0] == "k" else a.transpose(1, 2), w if majors[1] == "n" else w.transpose(1, 2)
    aux = torch.randn((b, m, n), generator=gen, device=cuda).to(t)
    if b == 1:
        a, w, aux = a[0], w[0], aux[0]
    want = a.double() @ w.double()
    top = want.abs().max()
    out32 = torch.full(want.shape, float("nan"), device=cuda)
    gemm(a, w, out32)
    assert (out32.double() - want).abs().max() <= 4 * k**0.5 * 2.0**-24 * top
    ulp = 2.0**-8 if dtype == "bfloat16" else 2.0**-11
    for epilogue in (None, "relu", "add", "mask_positive"):
        out, again = (torch.full(want.shape, float("nan"), dtype=t, device=cuda) for _ in range(2))
        for o in (out, again):
            gemm(a, w, o, epilogue=epilogue, aux=aux if epilogue in ("add", "mask_positive") else None)
        ref = {None: want, "relu": want.clamp(min=0), "add": want + aux.double(), "mask_positive": torch.where(aux > 0, want, torch.zeros_like(want))}[epilogue]
        # one rounding of the product and, for "add", one of the sum
        assert ((out.double() - ref).abs() <= 2 * ulp * torch.maximum(ref.abs(), want.abs()) + 4 * k**0.5 * 2.0**-24 * top).all(), epilogue
        assert torch.equal(out, again)
    device_status()


# (batch, M, N, K) whose K is cut: whole and ragged columns of a partial tile's 32, N that no group of four divides, rows past a tile, one
# row tile of the one-CTA kernel, several problems; `pad`: rows of the result further apart than N, where its groups of four are not
# aligned; `gap`: elements between the results of a batch, which no group of four divides
@pytest.mark.parametrize("shape, kernel", [
    ((1, 300, 520, 8192), "tcgen05"), ((1, 257, 40, 16384), "tcgen05"), ((1, 130, 33, 8192), "tcgen05"), ((1, 300, 264, 8200), "tcgen05"),
    ((2, 300, 264, 8192), "tcgen05"), ((3, 130, 33, 8192), "tcgen05"),
    ((1, 100, 520, 8192), "tcgen05"), ((1, 128, 33, 16384), "tcgen05"), ((2, 70, 296, 8192), "tcgen05"), ((1, 300, 520, 8192), "tcgen05_1cta"), ((2, 257, 33, 8192), "tcgen05_1cta"),
])  # fmt: skip
@pytest.mark.parametrize("operands, dtype, epilogue", [
    ("bfloat16", "float32", None), ("bfloat16", "bfloat16", None), ("bfloat16", "bfloat16", "add"), ("bfloat16", "bfloat16", "mask_positive"),
    ("float16", "float32", "relu"), ("float16", "float16", None), ("float16", "float16", "add"),
])  # fmt: skip
@pytest.mark.parametrize("pad, gap", [(0, 0), (2, 0), (0, 6)])
def test_split_products_at_edges(cuda, shape, kernel, operands, dtype, epilogue, pad, gap):
    """Against float64: 16-bit products are exact in float32, so only the order of K additions differs (K * 2^-24 of the sum of magnitudes
    at the very worst, its root in practice: 64 * 2^-24 allowed), and the result's own rounding, twice with an epilogue."""
    batch, m, n, k = shape
    gen = torch.Generator(device=cuda).manual_seed(n)
    od, td = getattr(torch, operands), getattr(torch, dtype)

    def rows_apart(fill):  # [batch, m, n] in rows of n + pad, problems m * (n + pad) + gap apart
        memory = torch.full((batch, m * (n + pad) + gap), 7.0, dtype=td, device=cuda)
        view = memory[:, : m * (n + pad)].view(batch, m, n + pad)[:, :, :n]
        if fill is not None:
            view.copy_(fill)
        return memory, view

    a = torch.randn(batch, m, k, generator=gen, device=cuda).to(od)
    b = torch.randn(batch, n, k, generator=gen, device=cuda).to(od).transpose(1, 2)
    aux = rows_apart(torch.randn(batch, m, n, generator=gen, device=cuda))[1] if epilogue in ("add", "mask_positive") else None
    memory, out = rows_apart(None)
    nbytes = gemm_scratch_bytes(m, n, k, batch)
    assert nbytes > 0
    scratch = torch.full((nbytes,), 255, dtype=torch.uint8, device=cuda)  # NaN: every partial sum that is read has been written
    one = (lambda t: t) if batch > 1 else (lambda t: None if t is None else t[0])
    gemm(one(a), one(b), one(out), epilogue=epilogue, aux=one(aux), scratch=scratch, kernel=kernel)
    want, size = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    tol, half = 64 * 2.0**-24 * size, {"float32": 0.0, "bfloat16": 2.0**-8, "float16": 2.0**-11}[dtype]
    tol = tol + half * want.abs()
    if epilogue == "relu":
        want = want.clamp(min=0)
    elif epilogue == "add":
        want = want + aux.double()
        tol = tol + half * want.abs() + half * half * size
    elif epilogue == "mask_positive":
        want = torch.where(aux > 0, want, 0.0)
    assert ((out.double() - want).abs() <= tol).all()
    out.fill_(7.0)
    assert (memory == 7.0).all()  # nothing was written beside the result
    device_status()


@pytest.mark.parametrize("shape, large", [((768, 768, 8192), True), ((300, 1000, 8200), True), ((816, 512, 17376), True), ((70, 9216, 12288), True),
                                          ((768, 768, 8128), False), ((384, 1536, 8192), False), ((128, 8192, 4096), False)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_scratch_decides_between_narrow_and_cut_large_tiles(cuda, shape, large, dtype):
    """Both sides of the line, by the bits of the kernel that is named: with enough scratch large tiles where the rule says so, with
    too little or none (or where it does not) the narrow ones. All within the K-order bound of float64."""
    m, n, k = shape
    gen = torch.Generator(device=cuda).manual_seed(k)
    a = torch.randn(m, k, generator=gen, device=cuda).bfloat16()
    b = torch.randn(n, k, generator=gen, device=cuda).bfloat16().t()
    nbytes = gemm_scratch_bytes(m, n, k)
    assert nbytes > 0

    def product(kernel, scratch_bytes):
        out = torch.empty(m, n, dtype=getattr(torch, dtype), device=cuda)
        return gemm(a, b, out, kernel=kernel, scratch=torch.empty(scratch_bytes, dtype=torch.uint8, device=cuda) if scratch_bytes else None)

    narrow, cut = product("auto", 0), product("tcgen05", nbytes)
    assert not torch.equal(narrow, cut)  # else the test could not tell them apart
    assert torch.equal(product("auto", nbytes), cut if large else narrow)
    assert torch.equal(product("auto", nbytes - 16), narrow)
    want, size = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    for out in (narrow, cut):  # 64 * 2^-24 of the sum of magnitudes for the order of K additions, the result's rounding
        assert ((out.double() - want).abs() <= 64 * 2.0**-24 * size + (2.0**-8 * want.abs() if dtype == "bfloat16" else 0)).all()
    device_status()


def products_plan(shapes):
    from lumen_b200.compiler import compile_graph
    from lumen_b200.plan import Plan

    def program(*x):
        return tuple(F.matmul(x[2 * i], x[2 * i + 1], "float32", "float32") for i in range(len(shapes)))

    specs = [("float32", s) for m, n, k in shapes for s in ((m, k), (k, n))]
    return Plan(compile_graph(tracer.trace(program, *specs)))


@pytest.mark.parametrize("shapes", [
    [(64, 48, 40), (33, 65, 70)], [(16, 32, 0), (1, 5, 7), (16, 33, 64)],  # tiles of 16 rows, one product without a sum
    [(400, 410, 15), (17, 33, 65), (416, 384, 128), (40, 70, 63), (130, 70, 33), (64, 64, 64)],  # two sizes of tile, more than a launch takes
    [(1100, 1121, 33), (256, 128, 512), (128, 512, 64)]])  # one that fills the GPU beside two that do not
def test_float32_products_of_one_launch_are_those_of_several(cuda, shapes):
    """Products of a plan that do not depend on one another share launches; every sum keeps its order."""
    x = [to_torch(t, cuda) for i, (m, n, k) in enumerate(shapes) for t in (operands(m, n, k, i) if k else (np.zeros((m, 0), "f"), np.zeros((0, n), "f")))]
    outs = [torch.full((m, n), float("nan"), device=cuda) for m, n, k in shapes]
    products_plan(shapes).run(x, outs)
    for i, out in enumerate(outs):
        assert torch.equal(out, gemm(x[2 * i], x[2 * i + 1], torch.empty_like(out)))


def test_batches_and_epilogues_of_one_launch(cuda):
    """Batched products (one with a transposed operand) and a relu beside a plain product: each as it is alone."""
    from lumen_b200.compiler import CompiledPlan, dense_strides
    from lumen_b200.plan import Plan

    products = [((3, 33, 65, 40), 1, False), ((1, 64, 64, 64), 0, False), ((2, 128, 17, 70), 0, True), ((5, 16, 32, 64), 1, True)]  # (batch, M, N, K), epilogue, B as [N, K]
    lines, steps, x, outs = [], [], [], []
    for i, ((batch, m, n, k), epilogue, across) in enumerate(products):
        a, b = (to_torch(t, cuda) for t in operands(m, n, k, i, batch))
        b = b.mT.contiguous().mT if across else b
        x += [a, b]
        outs.append(torch.full((batch, m, n), float("nan"), device=cuda))
        for at, (t, base) in enumerate([(a, f"i{2 * i}"), (b, f"i{2 * i + 1}"), (outs[-1], f"o{i}")]):
            lines.append(" ".join(map(str, ("t", 3 * i + at, "float32", base, 0, 3, *t.shape, *t.stride()))))
        steps.append(f"s gemm dot_general {3 * i} {3 * i + 1} {3 * i + 2} {epilogue} -1 -1")
    plan = Plan(CompiledPlan("\n".join([f"plan {len(x)} {len(outs)} 0", *lines, *steps, "end"]) + "\n", 0, len(x), len(outs)))
    assert plan.lib.lb_plan_kernel_launches(plan.handle) == 1
    plan.run(x, outs)
    for i, (_, epilogue, _) in enumerate(products):
        assert torch.equal(outs[i], gemm(x[2 * i], x[2 * i + 1], torch.empty_like(outs[i]), epilogue="relu" if epilogue else None))


def test_a_float32_product_that_reads_anothers_result_comes_after_it(cuda):
    """The memory given to a run decides: here the first result lies where the second product's operand does, the third's result where
    the second reads."""
    x = [to_torch(t, cuda) for i in range(3) for t in operands(64, 64, 64, i)]
    first, second = torch.empty(64, 64, device=cuda), torch.empty(64, 64, device=cuda)
    gemm(x[0], x[1], first)
    gemm(first, x[3], second)
    third = gemm(x[4], x[5], torch.empty_like(first))
    got = torch.empty_like(second)
    products_plan([(64, 64, 64)] * 3).run(x, [x[2], got, x[3]])
    assert torch.equal(x[2], first) and torch.equal(got, second) and torch.equal(x[3], third)
