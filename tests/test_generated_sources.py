"""Properties of the generated sources that no result shows."""

import re

import pytest

from lumen_b200 import functional as F
from lumen_b200 import prims, tracer
from lumen_b200.runtime import Fusion

ROWS_AND_COLUMNS = (lambda x, g: (x * g, prims.reduce_sum(x.float(), (1,), "float32"), prims.reduce_sum(x.float(), (0,), "float32")))
ODD_ROWS = (lambda x, g: F.relu(x * g))


@pytest.mark.parametrize("program, shape, dtype", [(ODD_ROWS, (5000, 3001), "bfloat16"), (ODD_ROWS, (64, 256), "float32"),
                                                   (ROWS_AND_COLUMNS, (512, 1024), "bfloat16"), (ROWS_AND_COLUMNS, (512, 1000), "float32")])
def test_arrays_that_vectors_are_written_to_are_aligned(program, shape, dtype):
    """Whole vectors are loaded into local arrays and stored from them: the array has a vector's alignment, not its elements'."""
    source = Fusion(tracer.trace(program, (dtype, shape), (dtype, shape[1:]))).source
    aligned = {}
    for line in source.splitlines():
        for name, size in re.findall(r"\b(?:u16|u32|u64|float|__nv_bfloat16|__half) (\w+)\[(\w+)\](?:\[\w+\])?;", line):
            aligned[name] = "__align__(16)" in line and aligned.get(name, True)
    vectors = set(re.findall(r"\bldv\w*<[^;]*?, (?:\(T\*\))?\(?(\w+)(?: \+ \d+)?\)?(?:\[ch\])?\);", source)) | set(re.findall(r"\bstv\w*<[^;]*, (\w+)\);", source))
    vectors &= set(aligned)
    assert len(vectors) >= 2 and all(aligned[v] for v in vectors), {v: aligned[v] for v in vectors}


def threads_and_blocks(shape, operands, sums):
    def program(*x):
        r = prims.reduce_sum(x[0], (1,), "float32").reshape(shape[0], 1)
        return tuple(prims.reduce_sum(x[k % operands] * (r + float(k)), (0,), "float32") for k in range(sums))

    source = Fusion(tracer.trace(program, *[("float32", shape)] * operands)).source
    return tuple(map(int, re.search(r"__launch_bounds__\((\d+), (\d+)\)", source).groups()))


# threads a block and blocks an SM: 32 warps (64 registers a thread) where what a thread holds fits them, otherwise 16 and those of smaller operands
@pytest.mark.parametrize("cols, operands, sums, launch", [
    (4096, 1, 2, (1024, 1)), (4096, 4, 8, (1024, 1)), (4096, 4, 9, (512, 1)), (4096, 3, 11, (512, 1)), (1024, 4, 8, (256, 4)), (1024, 4, 9, (128, 4)),
    (1536, 4, 4, (192, 5)), (1536, 1, 5, (192, 2)), (2304, 2, 4, (288, 3)), (2304, 2, 5, (192, 2)), (512, 4, 9, (64, 8)), (512, 4, 8, (128, 8))])
def test_rows_with_column_sums_have_the_registers_for_them(cols, operands, sums, launch):
    rows = -(-(1 << 21) // cols)
    assert threads_and_blocks((rows, cols), operands, sums) == launch
    if launch[0] * launch[1] <= 512:
        assert threads_and_blocks((rows // 4, cols), operands, sums) == launch
