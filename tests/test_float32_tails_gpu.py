"""Products of float32 operands with a residual or a relu's backward behind them in plans: every bit of the primitives one by one, also where
products that share a launch read or write what the tail reads."""

import numpy as np
import pytest
import torch

from lumen_b200 import functional as F
from lumen_b200 import nn, prims, tracer
from lumen_b200.compiler import compile_graph
from lumen_b200.plan import Plan
from lumen_b200._lib import LumenError
from lumen_b200.runtime import TORCH_DTYPES, device_status, gemm
from tests.helpers import run_oracle, to_numpy, to_torch

pytestmark = pytest.mark.gpu

DIMS = (((1,), (1,)), ((), ()))


def plus(x, w, r):
    return nn.fused(lambda a, b, c: c + prims.dot_general(a, b, DIMS, "float32"), x, w, r, name="dot_general", label="linear_add")


def masked(x, w, u):
    return nn.fused(lambda a, b, c: F.where(F.gt(c, 0), prims.dot_general(a, b, DIMS, "float32"), 0), x, w, u, name="dot_general", label="linear_backward_relu")


def program(x, w1, w2, r, u):
    y = plus(x, w1, r)
    z = plus(x, w2, y)  # behind the product whose result it adds
    m = masked(x, w1, u)  # beside it
    return y, z, m, masked(x, w2, z)


@pytest.mark.parametrize("rows, width, k", [(64, 64, 32), (33, 31, 7), (1, 96, 100), (257, 130, 64), (16, 32, 1), (512, 384, 65), (2000, 640, 48)])
def test_tails_of_float32_products(rows, width, k, cuda):
    rng = np.random.default_rng(rows)
    arrays = [rng.standard_normal(s).astype(np.float32) for s in ((rows, k), (width, k), (width, k), (rows, width), (rows, width))]
    arrays[4][rng.random((rows, width)) < 0.2] = 0.0
    g = tracer.trace(program, *[("float32", a.shape) for a in arrays])
    want = run_oracle(g, arrays)
    for plan in (Plan.native(g), Plan(compile_graph(g), cuda)):
        outs = [torch.full(g.types[v].shape, float("nan"), dtype=TORCH_DTYPES[g.types[v].dtype], device=cuda) for v in g.outputs]
        plan.run([to_torch(a, cuda) for a in arrays], outs)
        device_status()
        for got, exact in zip(outs, want):
            assert to_numpy(got).tobytes() == np.ascontiguousarray(exact).tobytes()


def test_the_entry_refuses_them_as_before(cuda):
    a, b, c, d = (torch.ones(32, 32, device=cuda) for _ in range(4))
    with pytest.raises(LumenError, match="16-bit outputs"):
        gemm(a, b, c, epilogue="add", aux=d)
