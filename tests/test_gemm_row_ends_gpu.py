"""The ends of rows in the tensor-core products' epilogues: lengths of a multiple of eight (which leave in 16-byte pieces), others, and
operands that are not aligned, against float64; nothing beside the result is written."""

import pytest

pytestmark = pytest.mark.gpu

KERNELS = [
    # kernel, m, k, scratch: CTA pairs, one CTA, pairs with K cut, and narrow tiles of one, two, four and eight ranges
    ("tcgen05", 300, 72, False), ("tcgen05_1cta", 300, 72, False), ("tcgen05", 130, 4096, True), ("auto", 60, 64, False), ("auto", 60, 136, False),
    ("auto", 130, 520, False), ("auto", 60, 2048, False),
]
WIDTHS = [8, 24, 64, 72, 120, 128, 136, 184, 256, 264, 312, 320, 376, 500, 37]


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("epilogue", ["none", "relu", "add", "mask_positive", "float32"])
@pytest.mark.parametrize("kernel, m, k, scratch", KERNELS)
def test_row_ends(kernel, m, k, scratch, epilogue, dtype):
    import torch

    from lumen_b200 import runtime

    t = getattr(torch, dtype)
    gen = torch.Generator(device="cuda").manual_seed(m + k)
    for n in WIDTHS:
        pad_n = (n + 7) // 8 * 8  # operands in whole 16-byte rows
        a = torch.randn(m, k, generator=gen, device="cuda").to(t)
        b = torch.randn(k, pad_n, generator=gen, device="cuda").to(t)[:, :n]
        want = a.double() @ b.double()
        size = want.abs().max().item()
        for shift in (0, 1):  # the result's and the operand's rows: aligned, and one element off
            wide = pad_n + 8
            out_t = torch.float32 if epilogue == "float32" else t
            whole = torch.full((m * wide + 8,), 7.0, device="cuda", dtype=out_t)
            out = whole[shift : shift + m * wide].view(m, wide)[:, :n]
            aux_whole = torch.randn(m * wide + 8, generator=gen, device="cuda").to(t)
            aux = aux_whole[shift : shift + m * wide].view(m, wide)[:, :n]
            kind = "none" if epilogue == "float32" else epilogue
            space = torch.empty(1 << 22, dtype=torch.uint8, device="cuda") if scratch else None
            runtime.gemm(a, b, out, epilogue=kind, kernel=kernel, scratch=space, aux=aux if kind in ("add", "mask_positive") else None)
            rounded = want.float().to(t).double()
            expect = {"none": want, "relu": want.clamp(min=0), "add": aux.double() + rounded,
                      "mask_positive": torch.where(aux > 0, rounded, torch.zeros_like(rounded))}[kind]
            # float32 sums of k products, and for 16 bits a rounding of the product and one of the sum, 2^-8 or 2^-11 of the value each
            ulp = 0.0 if epilogue == "float32" else 2.0**-7 if dtype == "bfloat16" else 2.0**-10
            bound = k * 2.0**-24 * size * 4 + ulp * (expect.abs() + want.abs())
            assert ((out.double() - expect).abs() <= bound).all(), (n, shift)
            rest = torch.ones_like(whole, dtype=torch.bool)
            rest[shift : shift + m * wide].view(m, wide)[:, :n] = False
            assert (whole[rest] == 7.0).all(), (n, shift)
    runtime.device_status()
