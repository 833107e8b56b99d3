"""What `lb_gemm` says about an epilogue's operand, in the order in which it looks: that there is one, its shape and dtype, and whether the kernels
take such results."""

import pytest

from lumen_b200 import _lib
from tests.test_host_path import Array


def status(dtype, aux, result=None):
    a, b = Array((4, 8), dtype), Array((8, 6), dtype)
    with pytest.raises(_lib.LumenError) as error:
        _lib.host().gemm(a, b, Array((4, 6), result or dtype), aux, 2, 0, 0, 0, 0)
    return error.value.status


def test_an_operand_that_is_missing_or_another_shape_is_invalid():
    for dtype in ("float32", "bfloat16"):
        assert status(dtype, None) == 1
        assert status(dtype, Array((4, 5), dtype)) == 1
        assert status(dtype, Array((4, 6), "float16")) == 1


def test_float32_results_are_not_supported():
    assert status("float32", Array((4, 6))) == 2
    assert status("bfloat16", Array((4, 6)), "float32") == 2
