"""Row ends (test_gemm_row_ends_gpu.py) of narrow products whose K two CTAs of a cluster share: four 64-wide blocks of K, few tiles."""

import pytest
from tests.test_gemm_row_ends_gpu import test_row_ends as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("epilogue", ["none", "relu", "add", "mask_positive", "float32"])
def test_two_ranges(epilogue, dtype):
    check("auto", 60, 248, False, epilogue, dtype)
