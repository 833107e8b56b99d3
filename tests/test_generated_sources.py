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
