"""Plan texts whose scratch holds the slices of sixteen warps an SM, where the library's kernels have more by now."""

import ctypes

import pytest

from lumen_b200 import _lib, prims, tracer
from lumen_b200 import functional as F
from lumen_b200.fusion_pass import fuse
from lumen_b200.plan import _bind
from lumen_b200.simplify import clean


@pytest.mark.parametrize("rows, cols, slices, former", [(16384, 1024, 888, 592), (5462, 1536, 592, 444), (8192, 2048, 444, 296)])
def test_fewer_slices_are_taken(rows, cols, slices, former):
    from lumen_b200.compiler import compile_graph

    def body(g, a, w):
        x = a.float() * F.rsqrt(F.mean(a.float() * a.float(), -1, keepdim=True) + 1e-5)
        t = g.float() * w.float()
        return (t - x * F.mean(t * x, -1, keepdim=True)).to(a.dtype), prims.reduce_sum(g.float() * x, (0,), "float32")

    graph = tracer.trace(body, ("bfloat16", (rows, cols)), ("bfloat16", (rows, cols)), ("bfloat16", (cols,)))
    lines = compile_graph(fuse(clean(graph))).text.splitlines(keepends=True)
    (at,) = [i for i, line in enumerate(lines) if line.startswith("t ") and " uint8 " in line]
    lib = _bind()
    for bytes_, taken in ((slices * cols * 4, True), (former * cols * 4, True), (former * cols * 4 - 4, False)):
        words = lines[at].split()
        if bytes_ == slices * cols * 4:
            assert int(words[6]) == bytes_
        words[6] = str(bytes_)
        text, plan = "".join(lines[:at] + [" ".join(words) + "\n"] + lines[at + 1 :]), ctypes.c_void_p()
        if taken:
            _lib.check(lib.lb_plan_create(text.encode(), ctypes.byref(plan)))
            lib.lb_plan_destroy(plan)
        else:
            with pytest.raises(_lib.LumenError, match="scratch"):
                _lib.check(lib.lb_plan_create(text.encode(), ctypes.byref(plan)))
