"""Every kernel that is launched so that it may become resident before the one before it has completed waits for that one first
(launch.cuh): the hand-written kernels by their source, the generated ones by what the generator writes."""

import pathlib
import re

import pytest

from lumen_b200 import functional as F
from lumen_b200 import prims, tracer
from lumen_b200._lib import LumenError
from lumen_b200.runtime import Fusion

CSRC = pathlib.Path(__file__).parent.parent / "lumen_b200" / "csrc"


def kernels(source):
    """`(name, parameters, body)` of the kernels in a CUDA source."""
    for m in re.finditer(r"__global__[^;{]*?(\w+)\(((?:[^(){}]|\([^()]*\))*)\)\s*\{", source):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(source[at], 0)
            at += 1
        yield m.group(1), m.group(2), source[m.end() : at]


def faults(name, params, body):
    """What is wrong with a kernel's wait: none, one that some threads or paths do not reach, pointers used in front of it,
    read-only parameters (whose loads a compiler may move across a barrier) that do not come out of it."""
    wait = re.search(r"\bgrid_wait\(([^)]*)\);", body)
    if not wait:
        return [f"{name}: no wait"]
    before, found = re.sub(r"\[[^\]]*\]\s*\([^()]*\)\s*\{[^{}]*\}", "", body[: wait.start()]), []  # without one-line lambdas
    if before.count("{") != before.count("}") or re.search(r"\breturn\b", before) or re.search(r"\b(if|for|while)\b[^;{}]*$", before):
        found.append(f"{name}: the wait is not reached by every thread")
    given = [x.strip() for x in wait.group(1).split(",")]
    for stands_for, pointer in re.findall(r"const \w+\* (\w+) = (\w+) \+ [^;]*;", before):  # an address, and not a load through it
        if stands_for in given and not re.search(rf"\b{pointer}\b", body[wait.end() :]):
            before = re.sub(rf"const \w+\* {stands_for} = [^;]*;", "", before)
            given.append(pointer)
    pointers = re.findall(r"\*\s*(?:__restrict__\s*)?(\w+)\s*(?:,|$)", params)
    found += [f"{name}: {p} is used in front of the wait" for p in pointers if re.search(rf"\b{p}\b", before)]
    if re.search(r"\b__ldg\(|\bp\.\w+\[|ld\.global", before):
        found.append(f"{name}: a load in front of the wait")
    constant = re.findall(r"const \w+\s*\* __restrict__ (\w+)", params)
    found += [f"{name}: {p} does not come out of the wait" for p in constant if p not in given]
    found += [f"{name}: __ldg of {p}" for p in re.findall(r"__ldg\((?:\([^()]*\)\(?)?(\w+)", body) if p not in given]
    return found


def test_every_overlapped_kernel_waits():
    launched, waits = set(), {}
    for path in CSRC.glob("*.cu"):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        launched |= set(re.findall(r"launch_overlapped\(\s*(\w+)", text)) - {"kernel"}
        waits.update({name: faults(name, params, body) for name, params, body in kernels(text)})
    assert len(launched) >= 15 and launched <= set(waits)
    assert waits.pop("wait_timeout_kernel") == ["wait_timeout_kernel: no wait"]  # launched in the ordinary way
    assert not sum(waits.values(), [])


PROGRAMS = [
    (lambda x, g: F.relu(x * g), [(64, 256), (256,)]),
    (lambda x, r, s: x * r + s, [(64, 4096), (64, 1), (1, 1)]),  # one row a block: neither r's nor s's address depends on the thread
    (lambda x, g: prims.reduce_sum(x * g, (1,), "float32"), [(3, 4001), (4001,)]),
    (lambda x, g: prims.reduce_sum(x * g, (0,), "float32"), [(512, 100), (100,)]),
    (lambda x, s: prims.reduce_sum(x, (0,), "float32") * s, [(512, 100), (1,)]),
    (lambda x, r: (x + prims.reduce_sum(x * r, (1,), "float32").reshape(512, 1), prims.reduce_sum(x, (0,), "float32")), [(512, 1000), (512, 1)]),
]


@pytest.mark.parametrize("option", ["", "option multi\n", "option inplace\n"])
@pytest.mark.parametrize("program, shapes", PROGRAMS)
def test_generated_kernels_wait_before_their_first_access(program, shapes, option):
    try:
        source = Fusion(option + tracer.trace(program, *[("float32", s) for s in shapes]).to_text()).source
    except LumenError:
        assert option  # reductions and row operands have no horizontal form, column totals none in place
        return
    found = [k for k in kernels(source) if k[0].startswith("fused_")]
    assert found
    for name, params, body in found:
        before = body.split("const u32 tid = grid_wait();")[0]
        assert len(before) < len(body) and not re.search(r"\b(in|out)\d|scratch|table|[{}]", before)
        uses = re.findall(r"\b(?:in\d+|scratch)\b[^;]*;", body)
        reads = set(re.findall(r"\bin\d+\b", body)) | ({"scratch"} if name == "fused_finalize" else set())
        for pointer in reads:
            first = next(u for u in uses if re.match(rf"{pointer}\b", u))
            assert re.fullmatch(rf"{pointer} = behind_wait\((?:{pointer}|table\.ptr\[group\]\[\d+\]), tid\);", first), first


def test_every_commit_is_waited_for():
    """A block leaves once the last commit aimed at each of its barriers has arrived: those that say that something is there (`_full`)
    are waited for by what reads it, the others, which hand a buffer back, by the producer behind its last tile's load."""
    waits = {}
    for path in CSRC.glob("*.cu"):
        for name, _, body in kernels(re.sub(r"//[^\n]*", "", path.read_text())):
            committed = set(re.findall(r"mma_commit(?:_pair)?\(&?(\w+)", body))
            if committed:
                after = body[body.rindex("tma_load") :]
                waits[name] = {c for c in committed if not c.endswith("_full") and not re.search(rf"mbar_wait(?:_ring<\w+>\({c},|\({c}, [^;]* - 1\))", after)}
    assert len(waits) >= 7 and not any(waits.values()), waits
