"""Division of a chunk's elements by their row's value in generated kernels: which programs take it, and its arithmetic, compiled for
the host (fused multiply-adds and reciprocals are correctly rounded there too)."""

import ctypes
import re
import subprocess

import numpy as np
import pytest

from lumen_b200 import functional as F
from lumen_b200 import prims, tracer
from lumen_b200.runtime import Fusion

SHAPE = (64, 1024)


def source_of(program, dtype="float32"):
    return Fusion(tracer.trace(program, (dtype, SHAPE), ("float32", (SHAPE[0], 1)))).source


def by_row_sum(x):
    return x / prims.reduce_sum(x, (1,), "float32").reshape(SHAPE[0], 1)


PROGRAMS = [
    (lambda x, b: x / b, True),
    (lambda x, b: by_row_sum(F.relu(x)), True),
    (lambda x, b: by_row_sum(F.exp(x)), False),
    (lambda x, b: F.softmax(x, 1) + b, False),
    (lambda x, b: F.exp(x) * x / b, False),
    (lambda x, b: (F.exp(x) + 1.0) / b, True),
]


@pytest.mark.parametrize("program, chunks", PROGRAMS)
def test_what_is_divided_in_chunks(program, chunks):
    """Elements by one value a row, but not exponentials: some of them are too small for the reciprocal, and then their chunk is slower."""
    assert bool(re.search(r"divide_chunk<[^>]*>\(num", source_of(program))) == chunks


HOST = r"""
#include <cmath>
#define __device__
#define __forceinline__ inline
#define __noinline__
struct float4 { float x, y, z, w; };
static float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
template <class T> struct p2 { T x, y; };
static float __fmul_rn(float a, float b) { return a * b; }
static float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static float __frcp_rn(float a) { return 1.0f / a; }
static int divisions;
static float __fdiv_rn(float a, float b) { divisions++; return a / b; }
using std::fabs;
static p2<float> f32x2_mul(p2<float> a, p2<float> b) { return {a.x * b.x, a.y * b.y}; }
static p2<float> f32x2_fma(p2<float> a, p2<float> b, p2<float> c) { return {std::fma(a.x, b.x, c.x), std::fma(a.y, b.y, c.y)}; }
%s
template <class T> static int run(const float* a, const float* b, float* q, int rows) {
    divisions = 0;
    for (int r = 0; r < rows; r++) divide_chunk<8 * (int)sizeof(float) / (int)sizeof(T), T>((const T*)(a + 8 * r), (T*)(q + 8 * r), b[r], row_reciprocal(b[r]));
    return divisions;
}
extern "C" int single(const float* a, const float* b, float* q, int rows) { return run<float>(a, b, q, rows); }
extern "C" int pairs(const float* a, const float* b, float* q, int rows) { return run<p2<float>>(a, b, q, rows); }
"""


@pytest.fixture(scope="module")
def divide(tmp_path_factory):
    source = source_of(PROGRAMS[0][0])
    code = source[source.index("#define LEAST_DIVIDEND") :]
    end = code.index("divide_chunk(")
    end = code.index("\n}\n", end) + 3
    path = tmp_path_factory.mktemp("quotients")
    (path / "q.cpp").write_text(HOST % code[:end])
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-march=native", "-fPIC", "-shared", "-w", "-o", str(path / "q.so"), str(path / "q.cpp")], check=True)
    lib = ctypes.CDLL(str(path / "q.so"))

    def call(form, a, b):
        q = np.empty_like(a)
        pointers = [t.ctypes.data_as(ctypes.c_void_p) for t in (a, b, q)]
        return getattr(lib, form)(*pointers, len(b)), q

    return call


def same_bits(got, a, b):
    with np.errstate(all="ignore"):
        want = a / b[:, None]
    same = (got.view(np.uint32) == want.view(np.uint32)) | (np.isnan(got) & np.isnan(want))
    assert same.all()


def floats(rng, shape, low, high):
    return (rng.choice([-1.0, 1.0], shape) * np.ldexp(1.0 + rng.integers(0, 1 << 23, shape) / (1 << 23), rng.integers(low, high, shape))).astype(np.float32)


@pytest.mark.parametrize("form", ["single", "pairs"])
def test_zeros_are_divided_like_their_neighbours(divide, form):
    """Chunks with zeros of both signs, up to nothing else: no division, every bit that of one."""
    rng = np.random.default_rng(0)
    a, b = floats(rng, (200000, 8), -60, 60), np.abs(floats(rng, 200000, -40, 40))
    a[rng.random(a.shape) < rng.random((len(a), 1))] = 0.0
    a[rng.random(a.shape) < 0.1] *= -0.0
    a[:3] = 0.0
    divisions, q = divide(form, a, b)
    assert divisions == 0
    same_bits(q, a, b)


@pytest.mark.parametrize("form", ["single", "pairs"])
def test_what_has_no_exact_residual_is_divided(divide, form):
    """One element outside the range sends its four to divisions, whatever zeros lie beside it, and a divisor outside the whole chunk."""
    rng = np.random.default_rng(1)
    a, b = floats(rng, (4096, 8), -60, 60), np.abs(floats(rng, 4096, -40, 40))
    a[:, 3] = 0.0
    edges = np.array([2.0**-61, 1e-45, -1e-40, 2.0**61, np.inf, -np.inf, 3e38], np.float32)
    a[np.arange(2048), rng.integers(4, 8, 2048)] = rng.choice(edges, 2048)
    b[2048:] = rng.choice(np.array([0.0, -1.0, 2.0**-41, 2.0**41, np.inf, np.nan], np.float32), 2048)
    divisions, q = divide(form, a, b)
    assert divisions == 4 * 2048 + 8 * 2048
    same_bits(q, a, b)
