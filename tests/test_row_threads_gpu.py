"""Norms, cross entropy and softmax on rows at the edges of what decides the threads of a row and the blocks of an SM, against float64."""

import pytest
import torch

import lumen_b200
from lumen_b200 import functional as F
from lumen_b200 import nn

pytestmark = pytest.mark.gpu

WIDTHS = [256, 1536, 2040, 8200, 9872, 32768, 43704, 50304]


@pytest.mark.parametrize("dtype", ["bfloat16", "float16", "float32"])
@pytest.mark.parametrize("rows", [1, 700])
@pytest.mark.parametrize("cols", WIDTHS)
def test_rows(cols, rows, dtype):
    if rows * cols > 1 << 23:
        rows = (1 << 23) // cols
    t = getattr(torch, dtype)
    gen = torch.Generator(device="cuda").manual_seed(cols + rows)
    x = torch.randn(rows, cols, generator=gen, device="cuda").to(t)
    w, b = (torch.randn(cols, generator=gen, device="cuda").to(t) for _ in range(2))
    at = torch.randint(0, cols, (rows,), generator=gen, device="cuda")
    y, mean, rstd = lumen_b200.compile(lambda a, w, b: nn._ln_forward(a, w, b, 1e-5))(x, w, b)
    rms = lumen_b200.compile(lambda a, w: F.rms_norm(a.float(), w.float()).to(a.dtype))(x, w)
    loss, lse = lumen_b200.compile(lambda a, at: F.cross_entropy_forward_prims(a.float(), at))(x, at)
    soft = lumen_b200.compile(lambda a: F.softmax(a, 1))(x)
    d, dw, db = x.double(), w.double(), b.double()
    spread = (d - d.mean(1, keepdim=True)).pow(2).mean(1) + 1e-5
    # a rounding of each result, and float32 sums of `cols` terms in trees of at most 2^6 a thread
    ulp = {"bfloat16": 2.0**-8, "float16": 2.0**-11, "float32": 0.0}[dtype]

    def close(got, want, scale, rounding):
        assert ((got.double() - want).abs() <= 2e-5 * scale + 2 * rounding * want.abs()).all()

    close(mean.flatten(), d.mean(1), d.abs().mean(1), 0.0)
    close(rstd.flatten(), spread.rsqrt(), spread.rsqrt(), 0.0)
    xhat = (d - d.mean(1, keepdim=True)) * spread.rsqrt()[:, None]
    close(y, xhat * dw + db, xhat.abs() * dw.abs() + db.abs() + 1, ulp)
    norm = d * (d.pow(2).mean(1, keepdim=True) + torch.finfo(torch.float32).eps).rsqrt() * dw
    close(rms, norm, norm.abs() + 1, max(ulp, 1e-4))  # (the epsilon is the function's)
    close(lse.flatten(), torch.logsumexp(d, 1), 1 + torch.logsumexp(d, 1).abs(), 0.0)
    close(loss.flatten(), torch.logsumexp(d, 1) - d.gather(1, at[:, None])[:, 0], 10.0, 0.0)
    if dtype == "float32":
        close(soft, torch.softmax(d, 1), torch.softmax(d, 1), 1e-6)
    else:  # rounded to 16 bits after every primitive: exponentials, their sum and the quotient
        assert ((soft.double() - torch.softmax(d, 1)).norm() / torch.softmax(d, 1).norm()) < 16 * ulp
