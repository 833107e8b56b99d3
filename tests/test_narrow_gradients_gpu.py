"""Kernels that sum rows and columns, at the widths and sizes where a row's threads and an SM's warps change, against float64."""

import pytest
import torch

import lumen_b200
from lumen_b200 import functional as F
from lumen_b200 import prims

pytestmark = pytest.mark.gpu

SHAPES = [(8192, 256), (7944, 264), (7945, 264), (5001, 504), (4096, 512), (4097, 512), (8200, 512), (4035, 520), (3001, 760), (2732, 768),
          (3971, 264), (3972, 264), (63550, 264), (5462, 384), (5400, 392), (2048, 512), (1638, 640), (16200, 640), (11000, 768), (1352, 776), (4200, 1000), (1033, 1016),
          (8191, 1024), (8192, 1024), (9001, 1024), (5462, 1536), (4096, 2048), (4097, 2048), (8193, 1028)]


def backward(rows, with_sum):
    def body(g, a, w, mu, rs, acc):
        g32 = g.float()
        xhat = (a.float() - mu.reshape(rows, 1)) * rs.reshape(rows, 1)
        gf = g32 * w.float()
        c1, c2 = F.mean(gf, -1, keepdim=True), F.mean(gf * xhat, -1, keepdim=True)
        dx = (gf - c1 - xhat * c2) * rs.reshape(rows, 1)
        if with_sum:
            dx = dx + acc.float()
        return dx.to(a.dtype), prims.reduce_sum(g32 * xhat, (0,), "float32"), prims.reduce_sum(g32, (0,), "float32")

    return body


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("with_sum", [False, True])
@pytest.mark.parametrize("rows,cols", SHAPES)
def test_gradients(rows, cols, with_sum, dtype):
    t = getattr(torch, dtype)
    gen = torch.Generator(device="cuda").manual_seed(rows + cols)
    g, a, acc = (torch.randn(rows, cols, generator=gen, device="cuda").to(t) for _ in range(3))
    w = torch.randn(cols, generator=gen, device="cuda").to(t)
    mu = torch.randn(rows, generator=gen, device="cuda")
    rs = torch.rand(rows, generator=gen, device="cuda") + 0.5
    dx, dw, db = lumen_b200.compile(backward(rows, with_sum))(g, a, w, mu, rs, acc)
    G, A, W, MU, RS = g.double(), a.double(), w.double(), mu.double()[:, None], rs.double()[:, None]
    X = (A - MU) * RS
    terms = G * W
    want = (terms - terms.mean(1, keepdim=True) - X * (terms * X).mean(1, keepdim=True)) * RS + (acc.double() if with_sum else 0)
    # a rounding of the result, and float32 means of `cols` terms (24 a thread and a tree) times what they are multiplied with
    ulp = {"bfloat16": 2.0**-8, "float16": 2.0**-11}[dtype]
    scale = (terms.abs() + terms.abs().mean(1, keepdim=True) + X.abs() * (terms * X).abs().mean(1, keepdim=True)) * RS + 5
    assert ((dx.double() - want).abs() <= ulp * want.abs() + 40 * 2.0**-24 * scale).all()
    # column sums: a block's rows one after another in float32, the blocks' totals after that
    depth = rows / 148 + 148 * 24
    for got, term in ((dw, G * X), (db, G)):
        assert ((got.double() - term.sum(0)).abs() <= depth * 2.0**-24 * term.abs().sum(0)).all()
