"""The native call path (lumen_b200._host) on stand-ins for tensors: what it reads, what it refuses and which calls it leaves to the
general path. No GPU: entries that get as far as the library raise its error."""

import pytest
import torch

from lumen_b200 import _lib
from lumen_b200.runtime import desc


class Array:
    """An array of another framework: the attributes the package reads, `shape` and `stride()` as any sequence."""

    def __init__(self, shape, dtype="float32", strides=None, sequence=tuple, cuda=True):
        self.shape, self.dtype, self.is_cuda, self._sequence = sequence(shape), dtype, cuda, sequence
        dense = [1] * len(shape)
        for d in range(len(shape) - 2, -1, -1):
            dense[d] = dense[d + 1] * shape[d + 1]
        self._strides = dense if strides is None else strides

    def data_ptr(self):
        return 1 << 20

    def stride(self):
        return self._sequence(self._strides)


def gemm(a, b, out):
    _lib.host().gemm(a, b, out, None, 0, 0, 0, 0, 0)


@pytest.mark.parametrize("sequence", [tuple, list, torch.Size])
def test_shapes_and_strides_are_any_sequence(sequence):
    a, b, out = Array((4, 8), sequence=sequence), Array((8, 6), sequence=sequence), Array((4, 5), sequence=sequence)
    with pytest.raises(_lib.LumenError, match=r"\[1,4,8\] x \[1,8,6\] -> \[1,4,5\]"):  # read right: the shapes do not match
        gemm(a, b, out)
    d = desc(a)
    assert (d.rank, list(d.shape[:2]), list(d.stride[:2])) == (2, [4, 8], [8, 1])


def test_what_is_not_a_tensor_on_the_gpu_is_refused():
    a, b, out = Array((4, 8)), Array((8, 6)), Array((4, 6))
    with pytest.raises(ValueError, match="expected a CUDA tensor"):
        gemm(Array((4, 8), cuda=False), b, out)
    with pytest.raises(TypeError, match="at most 8 integers"):
        gemm(Array((1,) * 9), b, out)
    with pytest.raises(TypeError, match="as many strides as dimensions"):
        gemm(Array((4, 8), strides=[1]), b, out)
    with pytest.raises(TypeError, match="no lumen dtype"):
        gemm(Array((4, 8), dtype=complex), b, out)
    with pytest.raises(AttributeError):
        gemm(3.0, b, out)
    with pytest.raises(TypeError, match="expected 9 arguments"):
        _lib.host().gemm(a, b)
