"""A chunk divided twice by the same value of its row (a normalisation's gradient): the second division takes the elements' range from the
first. And the packed sums of pairs."""

import ctypes
import subprocess

import numpy as np
import pytest

from lumen_b200 import prims, tracer
from lumen_b200.runtime import Fusion
from tests.test_quotients import HOST, PROGRAMS, SHAPE, floats, same_bits, source_of

TWICE = r"""
template <class T> static int twice(const float* a, const float* b, float* q, int rows) {
    divisions = 0;
    constexpr int n = 8 * (int)sizeof(float) / (int)sizeof(T);
    for (int r = 0; r < rows; r++) {
        const float y = row_reciprocal(b[r]);
        T once[n];
        const auto range = divide_chunk<n, T>((const T*)(a + 8 * r), once, b[r], y);
        divide_again<n, T>(once, (T*)(q + 8 * r), b[r], y, range);
    }
    return divisions;
}
extern "C" int single_again(const float* a, const float* b, float* q, int rows) { return twice<float>(a, b, q, rows); }
extern "C" int pairs_again(const float* a, const float* b, float* q, int rows) { return twice<p2<float>>(a, b, q, rows); }
"""


@pytest.fixture(scope="module")
def divide_twice(tmp_path_factory):
    source = source_of(PROGRAMS[0][0])
    code = source[source.index("#define LEAST_DIVIDEND") :]
    end = code.index("\n}\n", code.index("divide_again(")) + 3
    path = tmp_path_factory.mktemp("quotients")
    (path / "q.cpp").write_text(HOST % code[:end] + TWICE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-march=native", "-fPIC", "-shared", "-w", "-o", str(path / "q.so"), str(path / "q.cpp")], check=True)
    lib = ctypes.CDLL(str(path / "q.so"))

    def call(form, a, b):
        q = np.empty_like(a)
        return getattr(lib, form)(*[t.ctypes.data_as(ctypes.c_void_p) for t in (a, b, q)], len(b)), q

    return call


@pytest.mark.parametrize("form", ["single_again", "pairs_again"])
@pytest.mark.parametrize("low, high", [(-2, 2), (-20, 20), (-60, 60), (-127, 127)])
def test_a_quotient_divided_again_is_that_quotient(divide_twice, form, low, high):
    """Every bit of (a / b) / b, where the quotients leave the range, and with zeros, infinities and divisors that have no reciprocal."""
    rng = np.random.default_rng(low & 0xFF)
    a, b = floats(rng, (60000, 8), low, high), np.abs(floats(rng, 60000, max(low, -42), min(high, 42)))
    plain = a.copy()
    a[rng.random(a.shape) < 0.02] = 0.0
    a[rng.random(a.shape) < 0.001] = -np.inf
    a[::2] = plain[::2]
    divisions, q = divide_twice(form, a, b)
    with np.errstate(all="ignore"):
        same_bits(q, a / b[:, None], b)
    if low == -2:  # (nothing near the ends of the range: only the infinities' chunks are divided)
        assert divisions <= 2 * 4 * np.isinf(a).sum()


def test_which_programs_divide_again():
    """The same divisor twice, and no other."""
    twice = source_of(lambda x, b: x / b / b)
    assert "= divide_again<" in twice and "= divide_chunk<" in twice
    other = source_of(lambda x, b: x / b / (b + 1.0))
    assert "= divide_again<" not in other and other.count("= divide_chunk<") == 2


def test_pairs_are_added_as_pairs():
    def program(x):
        return prims.reduce_sum(x.to("float32"), (1,), "float32"), prims.reduce_max(x.to("float32"), (1,))

    source = Fusion(tracer.trace(program, ("bfloat16", SHAPE))).source
    assert source.count("const p2<float> sum = f32x2_add(") == 1 and "fmax_nan(acc" in source
