"""Products of CTA pairs whose K is cut, with all the scratch they ask for, with what fewer ranges take and with none, against float64."""

import pytest
import torch

from lumen_b200.runtime import device_status, gemm, gemm_scratch_bytes

pytestmark = pytest.mark.gpu

# (M, N, K, ranges): one wave of pairs' tiles, two, ragged on each side, a last range that is shorter, ranges of 16 blocks
SHAPES = [(1500, 1024, 4096, 3), (1530, 1536, 6144, 2), (1024, 3072, 16384, 3), (129, 1000, 20000, 18), (2048, 1024, 4104, 2), (411, 3072, 3080, 3)]


@pytest.mark.parametrize("out", ["bfloat16", "float32"])
@pytest.mark.parametrize("m, n, k, ranges", SHAPES)
def test_ranges(m, n, k, ranges, out):
    assert gemm_scratch_bytes(m, n, k) == ranges * m * n * 4
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    a, b = (torch.randn(s, generator=gen, device="cuda").bfloat16() for s in ((m, k), (k, n)))
    want = a.double() @ b.double()
    bound = a.double().abs() @ b.double().abs()
    for held in (ranges, ranges - 1, 1, 0):
        room = torch.full((held * m * n + 64,), 7.0, device="cuda")
        y = torch.empty(m, n, device="cuda", dtype=getattr(torch, out))
        gemm(a, b, y, scratch=room[: held * m * n] if held else None)
        device_status()
        # float32 sums of K terms in blocks of 16 on the tensor cores, then the ranges; one rounding of the result
        limit = (k / 16 + ranges) * 2.0**-24 * bound + (2.0**-8 * want.abs() if out == "bfloat16" else 0)
        assert ((y.double() - want).abs() <= limit).all(), held
        assert (room[held * m * n:] == 7.0).all()
