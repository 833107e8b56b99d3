"""Every kernel that is launched so that it may become resident before the one before it has completed waits for that one first
(launch.cuh): the hand-written kernels by their source, the generated ones by what the generator writes."""

import pathlib
import re

import pytest

from lumen_b200 import functional as F
from lumen_b200 import prims, tracer
from lumen_b200.runtime import Fusion

CSRC = pathlib.Path(__file__).parent.parent / "lumen_b200" / "csrc"


def bodies(source):
    """`(name, body)` of the kernels in a CUDA source."""
    for m in re.finditer(r"__global__[^;{]*?(\w+)\((?:[^(){}]|\([^()]*\))*\)\s*\{", source):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(source[at], 0)
            at += 1
        yield m.group(1), source[m.end() : at]


def test_every_overlapped_kernel_waits():
    launched, waits = set(), {}
    for path in CSRC.glob("*.cu"):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        launched |= set(re.findall(r"launch_overlapped\(\s*(\w+)", text)) - {"kernel"}
        waits.update({name: "grid_wait()" in body for name, body in bodies(text)})
    assert len(launched) >= 15 and launched <= set(waits)
    assert [name for name, ok in waits.items() if not ok] == ["wait_timeout_kernel"]  # launched in the ordinary way


@pytest.mark.parametrize("program, shapes", [
    (lambda x, g: F.relu(x * g), [(64, 256), (256,)]),
    (lambda x, g: prims.reduce_sum(x * g, (1,), "float32"), [(3, 4001), (4001,)]),
    (lambda x, g: prims.reduce_sum(x * g, (0,), "float32"), [(512, 100), (100,)]),
])
def test_generated_kernels_wait_before_their_first_access(program, shapes):
    source = Fusion(tracer.trace(program, *[("float32", s) for s in shapes])).source
    kernels = [body for name, body in bodies(source) if name.startswith("fused_")]
    assert kernels
    for body in kernels:
        before = body.split("grid_wait()")[0]
        assert len(before) < len(body) and not re.search(r"\b(in|out)\d|scratch", before)
