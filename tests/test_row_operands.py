"""Threads of a row and blocks of an SM by what a thread holds of the row: operands that do not fit eleven vectors a thread keep the threads that
their vectors ask for (csrc/fused_codegen.cpp, row_residency)."""

import re

import pytest

from lumen_b200 import functional as F
from lumen_b200 import prims, tracer
from lumen_b200.runtime import Fusion


def cross_entropy(x, t):
    return F.cross_entropy_forward_prims(x.float(), t)


def cross_entropy_of_two(x, y, t):
    return F.cross_entropy_forward_prims(x.float() + y.float(), t)


def layer_norm(x, w, y=None):
    s = x.float() if y is None else x.float() + y.float()
    d = s - F.mean(s, -1, keepdim=True)
    return (d * F.rsqrt(F.mean(d * d, -1, keepdim=True) + 1e-5) * w.float() + w.float()).to(w.dtype)


def rms_norm(x, w, y=None):
    s = x.float() if y is None else x.float() + y.float()
    return (s * F.rsqrt(F.mean(s * s, -1, keepdim=True) + 1e-5) * w.float()).to(w.dtype)


def kernel(program, cols, *dtypes, rows=700):
    """Threads of a row and the least blocks an SM (0: the compiler's choice)."""
    shapes = {"cross_entropy": "xt", "cross_entropy_of_two": "xxt"}.get(program.__name__, "xw" + "x" * (len(dtypes) - 2))
    types = [(d, {"x": (rows, cols), "w": (cols,), "t": (rows,)}[s]) for s, d in zip(shapes, dtypes)]
    source = Fusion(tracer.trace(program, *types)).source
    bounds = re.search(r"__launch_bounds__\((\d+)(?:, (\d+))?\) fused_kernel", source)
    return int(re.search(r"#define TPR (\d+)", source)[1]), int(bounds[2] or 0)


B, H, W, IDS = "bfloat16", "float16", "float32", "int64"


@pytest.mark.parametrize("program, cols, dtypes, threads, blocks", [
    # one operand of 16 bits: eleven vectors a thread
    (cross_entropy, 32768, (B, IDS), 384, 4), (layer_norm, 32768, (H, H), 384, 2), (rms_norm, 9872, (B, W), 128, 8),
    # two, or float32 rows beside 16 bits: a thread to four vectors
    (cross_entropy_of_two, 32768, (B, B, IDS), 1024, 0), (cross_entropy_of_two, 9872, (H, H, IDS), 512, 0), (layer_norm, 16384, (W, B), 512, 0),
    (rms_norm, 9872, (W, B), 512, 0), (layer_norm, 9872, (B, B, B), 512, 0), (layer_norm, 32768, (W, B, B), 1024, 0), (cross_entropy_of_two, 9872, (W, W, IDS), 1024, 0),
    # ... from where they have more than four, two operands of 16 bits fit
    (layer_norm, 50304, (B, B, B), 608, 1), (rms_norm, 33000, (H, H, H), 416, 2), (layer_norm, 33000, (H, H, H), 1024, 0), (layer_norm, 50304, (W, B, B), 1024, 0),
    # float32 cross entropy reads its logits twice, the second time by a gather
    (cross_entropy, 8200, (W, IDS), 544, 2), (cross_entropy, 12000, (W, IDS), 768, 0),
    # warps of an SM
    (layer_norm, 1024, (B, B), 32, 2), (layer_norm, 1024, (B, W), 32, 0), (layer_norm, 2048, (B, B, B), 64, 0), (layer_norm, 4096, (B, B, B), 128, 4),
    (rms_norm, 1024, (W, B), 32, 0), (rms_norm, 1536, (B, B), 64, 0), (rms_norm, 1024, (B, B), 32, 2),
])
def test_what_fits(program, cols, dtypes, threads, blocks):
    assert kernel(program, cols, *dtypes) == (threads, blocks)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("cols", [33000, 40968, 50304])
@pytest.mark.parametrize("program", [layer_norm, rms_norm])
def test_norms_of_two_wide_operands(program, cols, dtype):
    import torch

    import lumen_b200

    gen = torch.Generator(device="cuda").manual_seed(cols)
    x, y = (torch.randn(31, cols, generator=gen, device="cuda").to(getattr(torch, dtype)) for _ in range(2))
    w = torch.randn(cols, generator=gen, device="cuda").to(x.dtype)
    s, d = x.double() + y.double(), w.double()
    if program is layer_norm:
        s = s - s.mean(1, keepdim=True)
    want = s * (s.pow(2).mean(1, keepdim=True) + 1e-5).rsqrt() * d + (d if program is layer_norm else 0)
    got = lumen_b200.compile(program)(x, w, y).double()
    # a rounding of the result, and float32 sums of chains of 2^6 and trees of 2^10
    bound = {"bfloat16": 2.0**-8, "float16": 2.0**-11}[dtype] * want.abs() + 2.0**-18 * (s.abs() + 1) * (d.abs() + 1)
    assert ((got - want).abs() <= bound).all()


def gradients(g, a, w):
    x = a.float() * F.rsqrt(F.mean(a.float() * a.float(), -1, keepdim=True) + 1e-5)
    t = g.float() * w.float()
    return (t - x * F.mean(t * x, -1, keepdim=True)).to(a.dtype), prims.reduce_sum(g.float() * x, (0,), "float32"), prims.reduce_sum(g.float(), (0,), "float32")


@pytest.mark.parametrize("cols, dtypes, blocks", [(1024, (B, B, B), 6), (1536, (B, B, B), 4), (2048, (H, H, W), 3), (1024, (W, B, B), 6), (1536, (W, B, B), 3), (1536, (B, W, B), 3),
                                                  (2048, (B, W, W), 2), (1024, (W, W, B), 4)])
def test_warps_of_kernels_that_sum_columns(cols, dtypes, blocks):
    """24 warps an SM for operands of 16 bits, one of float32 at 128 threads a row; sixteen for others."""
    rows = (1 << 24) // cols
    types = [(d, shape) for d, shape in zip(dtypes, ((rows, cols), (rows, cols), (cols,)))]
    source = Fusion(tracer.trace(gradients, *types)).source
    assert int(re.search(r"__launch_bounds__\(\d+, (\d+)\) fused_kernel", source)[1]) == blocks
