"""Kernels that become resident before the one before them has completed read nothing early: dependent kernels of every family, queued
without a wait between them, on inputs that change from pass to pass, give the bits that they give one at a time."""

import pytest
import torch

import lumen_b200
from lumen_b200 import functional as F
from lumen_b200 import prims
from lumen_b200.runtime import attention_backward, attention_forward, gemm, scatter_add_rows

pytestmark = pytest.mark.gpu


def norm(x, w, b):
    return F.layer_norm(x.to("float32"), w.to("float32"), b.to("float32")).to(x.dtype)


def column_sums(x):
    return prims.reduce_sum(x.to("float32"), (0,), "float32")


COMPILED = {"norm": lumen_b200.compile(norm), "columns": lumen_b200.compile(column_sums)}


def chain(s, after):
    """One pass: every call reads what the one before it wrote; `after` runs between them. Rows 512 and 2048 wide: narrow and wide
    products, one and several blocks of a row."""
    out = []

    def step(t):
        after()
        out.append(t)
        return t

    h = step(COMPILED["norm"](s["x"], s["w"], s["b"]))
    y = step(gemm(h, s["u"], torch.empty(s["x"].shape[0], s["u"].shape[1], dtype=h.dtype, device=h.device)))
    g = step(gemm(h.t(), y, torch.empty(h.shape[1], y.shape[1], dtype=torch.float32, device=h.device)))  # float32: K cut or not
    q = y.view(2, -1, y.shape[1] // 64, 64)
    o, lse = attention_forward(q, q, q, causal=True)
    step(o), step(lse)
    for det in (True, False):
        dq, dk, dv = attention_backward(q, q, q, o, o, lse, causal=True, deterministic=det)
        after()
        out += [dk, dv] + ([dq] if det else [])
    wide = torch.empty(g.shape[0], g.shape[0], dtype=torch.float32, device=h.device)
    step(gemm(g, g.t(), wide))  # CUDA cores
    step(scatter_add_rows(h, s["ids"], y[:, : h.shape[1]].contiguous()))
    step(COMPILED["columns"](h))
    return out


@pytest.mark.parametrize("rows, width", [(256, 512), (1024, 2048)])
def test_queued_passes_equal_passes_one_at_a_time(cuda, rows, width):
    gen = torch.Generator(device=cuda).manual_seed(rows)

    def normal(*shape, std=1.0):
        return (torch.randn(shape, generator=gen, device=cuda) * std).to(torch.bfloat16)

    s = {"w": normal(width), "b": normal(width), "u": normal(width, 2 * width, std=width**-0.5), "x": normal(rows, width),
         "ids": torch.randint(0, rows, (rows,), generator=gen, device=cuda)}
    inputs = [normal(rows, width) for _ in range(6)]

    def run(after):
        got = []
        for x in inputs:
            s["x"].copy_(x)
            after()
            got.append(chain(s, after))
        torch.cuda.synchronize()
        return got

    want = run(torch.cuda.synchronize)
    for _ in range(5):
        for g, w in zip(run(lambda: None), want):
            assert all(torch.equal(a, b) for a, b in zip(g, w))


def test_captured_beside_another_stream(cuda):
    """Captured by the caller, the first kernel behind the join of a second stream, whose work it reads."""
    gen = torch.Generator(device=cuda).manual_seed(1)
    a, b = (torch.randn(512, 512, generator=gen, device=cuda).to(torch.bfloat16) for _ in range(2))
    left, right, out = (torch.empty(512, 512, dtype=torch.bfloat16, device=cuda) for _ in range(3))
    other = torch.cuda.Stream()

    def work():
        main = torch.cuda.current_stream()
        other.wait_stream(main)
        gemm(a, b, left)
        with torch.cuda.stream(other):
            for _ in range(8):
                gemm(b, a, right)
        main.wait_stream(other)
        gemm(left, right, out)

    work()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        work()
    for seed in range(4):
        a.copy_(torch.randn(512, 512, generator=gen, device=cuda))
        graph.replay()
        torch.cuda.synchronize()
        got = out.clone()
        work()
        torch.cuda.synchronize()
        assert torch.equal(got, out)
