"""A warp to a row in kernels that sum rows of 520 to 768 columns and columns: where no lane lacks its last vector with few row sums, elsewhere up to
five million elements (csrc/fused_codegen.cpp)."""

import re

import pytest

from lumen_b200 import functional as F
from lumen_b200 import prims, tracer
from lumen_b200.runtime import Fusion


def rms_gradients(g, a, w):
    x = a.float() * F.rsqrt(F.mean(a.float() * a.float(), -1, keepdim=True) + 1e-5)
    t = g.float() * w.float()
    return (t - x * F.mean(t * x, -1, keepdim=True)).to(a.dtype), prims.reduce_sum(g.float() * x, (0,), "float32")


def layer_norm_gradients(g, a, w):
    mean = F.mean(a.float(), -1, keepdim=True)
    d = a.float() - mean
    x = d * F.rsqrt(F.mean(d * d, -1, keepdim=True) + 1e-5)
    t = g.float() * w.float()
    return (t - F.mean(t, -1, keepdim=True) - x * F.mean(t * x, -1, keepdim=True)).to(a.dtype), prims.reduce_sum(g.float() * x, (0,), "float32")


def threads(program, rows, cols, dtype):
    types = [(dtype, (rows, cols)), (dtype, (rows, cols)), (dtype, (cols,))]
    return int(re.search(r"#define TPR (\d+)", Fusion(tracer.trace(program, *types)).source)[1])


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("program, cols, elements, warp", [
    (rms_gradients, 760, 4 << 20, True), (rms_gradients, 760, 6 << 20, False), (rms_gradients, 760, 9 << 20, False), (rms_gradients, 768, 4 << 20, True),
    (rms_gradients, 768, 6 << 20, True), (rms_gradients, 768, 9 << 20, True), (layer_norm_gradients, 640, 4 << 20, True), (layer_norm_gradients, 640, 9 << 20, False),
    (layer_norm_gradients, 768, 4 << 20, False), (layer_norm_gradients, 768, 9 << 20, False), (layer_norm_gradients, 512, 9 << 20, True), (rms_gradients, 776, 4 << 20, False),
])
def test_a_warp_to_a_row(program, cols, elements, warp, dtype):
    assert (threads(program, elements // cols, cols, dtype) == 32) == warp


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("rows, cols", [(5500, 760), (7200, 760), (12500, 760), (7200, 768), (12500, 768), (7001, 752)])
def test_gradients(rows, cols, dtype):
    from tests import test_narrow_gradients_gpu as others

    for with_sum in (False, True):
        others.test_gradients(rows, cols, with_sum, dtype)
