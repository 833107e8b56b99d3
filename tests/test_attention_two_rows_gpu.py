"""CUDA-core attention with two rows a warp (many blocks) gives the bits of one row a warp (few): the same heads in a small and a large batch."""

import pytest
import torch

from lumen_b200 import runtime

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("sq, sk, n, nkv, d", [(1, 1, 2, 1, 32), (7, 40, 4, 2, 32), (33, 33, 2, 2, 64), (64, 31, 2, 1, 96), (65, 97, 2, 1, 128), (31, 64, 1, 1, 256)])
def test_every_bit_is_that_of_one_row(sq, sk, n, nkv, d, causal):
    few, many = 2, 2 + 512 // max(1, nkv * min((sq + 7) // 8, (sk + 7) // 8))
    gen = torch.Generator(device="cuda").manual_seed(sq + sk)
    q, g = (torch.randn(many, sq, n, d, generator=gen, device="cuda") for _ in range(2))
    k, v = (torch.randn(many, sk, nkv, d, generator=gen, device="cuda") for _ in range(2))
    o, lse = runtime.attention_forward(q, k, v, causal=causal)
    grads = runtime.attention_backward(q, k, v, o, g, lse, causal=causal)
    for b in (0, many - few):
        part = slice(b, b + few)
        o1, lse1 = runtime.attention_forward(q[part], k[part], v[part], causal=causal)
        assert torch.equal(o1, o[part]) or (o1.isnan() == o[part].isnan()).all() and torch.equal(o1.nan_to_num(), o[part].nan_to_num())
        assert torch.equal(lse1.nan_to_num(), lse[part].nan_to_num())
        if causal and sk < sq:  # queries that see no key have no finite log-sum-exp
            continue
        for x, y in zip(runtime.attention_backward(q[part], k[part], v[part], o1, g[part], lse1, causal=causal), grads):
            assert torch.equal(x, y[part])
    runtime.device_status()
