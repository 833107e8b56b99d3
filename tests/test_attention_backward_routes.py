"""What the attention backward takes where one batch entry, head or token has a stride that no tensor map takes: the tensor cores what they
accept, the CUDA cores the rest."""

import pytest
import torch

from lumen_b200 import _lib


def odd_strides(shape, strides):
    return [1 if size == 1 and dim < 3 else step for dim, (size, step) in enumerate(zip(shape, strides))]


class Operand:
    """A [B, S, N, H] tensor that the host path reads and nothing touches."""

    is_cuda = True

    def __init__(self, shape, dtype="bfloat16", strides=None, address=1 << 20):
        self.shape, self.dtype, self.address = shape, dtype, address
        dense = [1] * len(shape)
        for d in range(len(shape) - 2, -1, -1):
            dense[d] = dense[d + 1] * shape[d + 1]
        self.strides = dense if strides is None else strides(shape, dense)

    def data_ptr(self):
        return self.address

    def stride(self):
        return self.strides


def backward(scale, strides, shape=(1, 64, 4, 64), accumulator=None):
    b, s, n, _ = shape
    q = Operand(shape, strides=strides)
    stats = Operand((b, n, s), "float32")
    _lib.host().attention_bwd(scale, True, 0, q, q, q, q, q, stats, stats, accumulator, q, q, q, 0, 0, 0)


@pytest.mark.skipif(torch.cuda.is_available(), reason="calls that are not refused run")
def test_what_is_refused():
    for scale in (-0.5, 0.0, float("nan")):
        with pytest.raises(_lib.LumenError, match="must be positive"):
            backward(scale, None)
    # whatever gets as far as the driver is taken
    taken = [dict(scale=scale, strides=odd_strides) for scale in (0.5, -0.5, 0.0, float("nan"))]
    taken += [dict(scale=0.5, strides=odd_strides, accumulator=Operand((1, 64, 4, 64), "float32", address=(1 << 20) + 4)),
              dict(scale=0.5, strides=odd_strides, shape=(70000, 64, 1, 64)), dict(scale=0.5, strides=odd_strides, shape=(1, 16, 70000, 64))]
    for call in taken:
        with pytest.raises(_lib.LumenError) as error:
            backward(**call)
        assert error.value.status == 3, error.value  # no CUDA device


@pytest.mark.gpu
@pytest.mark.parametrize("h", [64, 128])
def test_a_negative_scale_with_such_strides(h):
    from lumen_b200 import runtime

    s, n, scale = 96, 3, -0.1
    gen = torch.Generator(device="cuda").manual_seed(h)
    q, k, v, g = (torch.randn(1, s, n, h, generator=gen, device="cuda").bfloat16() for _ in range(4))
    odd = [t.as_strided(t.shape, odd_strides(t.shape, t.stride())) for t in (q, k, v, g)]
    o, lse = runtime.attention_forward(*odd[:3], scale=scale)
    grads = runtime.attention_backward(*odd[:3], o.as_strided(o.shape, odd_strides(o.shape, o.stride())), odd[3], lse, scale=scale)
    wide = [t.double().requires_grad_() for t in (q, k, v)]
    scores = torch.einsum("bqnh,bknh->bnqk", wide[0], wide[1]) * scale
    out = torch.einsum("bnqk,bknh->bqnh", scores.softmax(-1), wide[2])
    for got, want in zip(grads, torch.autograd.grad(out, wide, g.double())):
        # P and dS are rounded to bfloat16 (2^-9 of each), and the result once more
        assert (got.double() - want).norm() <= 4 * 2.0**-9 * want.norm()
    runtime.device_status()
