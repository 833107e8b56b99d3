"""Kernels that become resident before the one before them has completed read nothing early: dependent kernels of every family, queued
without a wait between them, on inputs that change from pass to pass, give the bits that they give one at a time."""

import ctypes

import pytest
import torch

import lumen_b200
from lumen_b200 import _lib, prims, tracer
from lumen_b200 import functional as F
from lumen_b200.runtime import Fusion, attention_backward, attention_forward, current_stream, desc, gemm, scatter_add_rows

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


@pytest.fixture(scope="module")
def fusions():
    """Kernels of a block a row whose operands are a scalar and a value of each row (their addresses depend on the block at most),
    row and column totals in one, and the horizontal form."""
    rows, cols = 600, 4096
    shape = ("float32", (rows, cols))
    body = tracer.trace(lambda p, g: p - g * 0.5, ("float32", (2, 64)), ("float32", (2, 64)))
    return {
        "totals": Fusion(tracer.trace(lambda x: (prims.reduce_sum(x, (1,), "float32").reshape(rows, 1), prims.reduce_sum(x, (0,), "float32")), shape)),
        "one": Fusion(tracer.trace(lambda c: prims.reduce_sum(c, (0,), "float32").reshape(1, 1), ("float32", (cols,)))),
        "scale": Fusion(tracer.trace(lambda x, r, o: x * r + o, shape, ("float32", (rows, 1)), ("float32", (1, 1)))),
        "multi": Fusion("option multi\n" + body.to_text()),
        # through transpose_kernel, tiled_copy_kernel and strided_copy_kernel
        "turned": lumen_b200.compile(lambda x: prims.transpose(x, (1, 0))),
        "swapped": lumen_b200.compile(lambda x: prims.transpose(x, (2, 1, 0))),
        "cut": lumen_b200.compile(lambda x: prims.slice(x, (1, 1, 1), x.shape)),
    }


def horizontal(fusion, groups):
    lib = _lib.lib()
    lib.lb_fusion_launch_groups.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    tensors = [desc(t) for g in groups for t in g]
    _lib.check(lib.lb_fusion_launch_groups(fusion.handle, (_lib.LbTensor * len(tensors))(*tensors), len(groups), current_stream()))
    return [g[-1] for g in groups]


def others(s, f, after):
    """One pass over the families that `chain` leaves out; every call reads what the one before it wrote."""
    out = []

    def step(t):
        after()
        out.append(t)
        return t

    x = s["x"]
    r, c = f["totals"](x)
    after()
    y = step(f["scale"](x, r, f["one"](c)[0])[0])
    t = step(f["turned"](y).clone())
    u = step(f["swapped"](t.view(64, 64, 600)).clone())
    w = step(f["cut"](u).clone())  # [599, 63, 63]
    q = (w.reshape(-1)[: 8 * 128 * 2 * 64].view(8, 128, 2, 64) * 1e-3).contiguous()
    o, lse = attention_forward(q, q, q, causal=True)  # CUDA cores
    step(o), step(lse)
    for g in attention_backward(q, q, q, o, o, lse, causal=True):
        step(g)
    kv = o.to(torch.bfloat16)
    d, lse = attention_forward(kv[:, :1].repeat(1, 1, 4, 1), kv, kv)  # decode
    step(d), step(lse)
    table = o.reshape(-1, 64)  # 2048 rows
    for g in horizontal(f["multi"], [[table[:n], table[n : 2 * n], torch.empty(n, 64, device=x.device)] for n in (1, 7, 300, 1024)]):
        step(g)
    step(scatter_add_rows(table, s["ids"], table.flip(0).contiguous(), deterministic=False))  # every row once: one order of additions
    step(scatter_add_rows(table, s["many"], table.repeat(3, 1)))  # more updates than one kernel takes
    return out


def test_queued_passes_of_the_other_families(cuda, fusions):
    gen = torch.Generator(device=cuda).manual_seed(3)
    s = {"x": torch.empty(600, 4096, device=cuda), "ids": torch.randperm(2048, generator=gen, device=cuda),
         "many": torch.randint(0, 2048, (3 * 2048,), generator=gen, device=cuda)}
    inputs = [torch.randn(600, 4096, generator=gen, device=cuda) for _ in range(6)]

    def run(after):
        got = []
        for x in inputs:
            s["x"].copy_(x)
            after()
            got.append(others(s, fusions, after))
        torch.cuda.synchronize()
        return got

    want = run(torch.cuda.synchronize)
    x, y = inputs[0], want[0][0]
    assert torch.allclose(y.double(), x.double() * x.double().sum(1, keepdim=True) + x.double().sum(), rtol=1e-4, atol=1e-1)
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
