"""The attention backward of one batch entry, one head or one token whose stride is none that a tensor map takes: what it is with any other."""

import pytest
import torch

from lumen_b200 import runtime

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s, n, nkv, d, causal", [(64, 4, 4, 64, True), (257, 8, 2, 64, True), (200, 4, 4, 128, False), (96, 1, 1, 64, True), (1, 4, 4, 64, False)])
def test_strides_of_single_elements_do_not_matter(s, n, nkv, d, causal):
    gen = torch.Generator(device="cuda").manual_seed(s)
    q, g = (torch.randn(1, s, n, d, generator=gen, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(1, s, nkv, d, generator=gen, device="cuda").bfloat16() for _ in range(2))
    o, lse = runtime.attention_forward(q, k, v, causal=causal)

    def odd(t):
        return t.as_strided(t.shape, [1 if size == 1 and dim < 3 else step for dim, (size, step) in enumerate(zip(t.shape, t.stride()))])

    want = runtime.attention_backward(q, k, v, o, g, lse, causal=causal)
    got = runtime.attention_backward(*(odd(t) for t in (q, k, v, o, g)), lse, causal=causal)
    for x, y in zip(got, want):
        assert torch.equal(x, y)
    runtime.device_status()
