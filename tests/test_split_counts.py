"""How many ranges K of a product of CTA pairs is cut into. And plans that were saved with scratch for a former number run as they did."""

import ctypes

import pytest

from lumen_b200 import _lib, prims, tracer
from lumen_b200.compiler import compile_graph
from lumen_b200.plan import _bind


def ranges(m, n, k):
    return max(1, _lib.lib().lb_gemm_scratch_bytes(m, n, k, 1) // (4 * m * n))


@pytest.mark.parametrize("m, n, k, count", [(1500, 1024, 4096, 3), (304, 920, 20424, 9), (1086, 608, 14504, 4), (1024, 3072, 16384, 3), (128, 2048, 8192, 8)])
def test_counts(m, n, k, count):
    assert ranges(m, n, k) == count


@pytest.mark.parametrize("m, n, k, former", [(176, 1616, 10248, 9), (1000, 480, 10096, 8), (224, 1392, 14744, 11)])
def test_saved_scratch_keeps_large_tiles(m, n, k, former):
    """Narrow tiles would take these without scratch for K ranges."""
    dims = (((1,), (0,)), ((), ()))
    graph = tracer.trace(lambda a, b: prims.dot_general(a, b, dims, "float32", "bfloat16"), ("bfloat16", (m, k)), ("bfloat16", (k, n)))
    lines = compile_graph(graph).text.splitlines(keepends=True)
    (at,) = [i for i, line in enumerate(lines) if line.startswith("t ") and " uint8 " in line]
    words = lines[at].split()
    words[6] = str(former * m * n * 4)
    lines[at] = " ".join(words) + "\n"
    lib, plan = _bind(), ctypes.c_void_p()
    _lib.check(lib.lb_plan_create("".join(lines).encode(), ctypes.byref(plan)))
    try:
        assert lib.lb_plan_kernel_launches(plan) == 2  # partial sums and their reduction
    finally:
        lib.lb_plan_destroy(plan)
