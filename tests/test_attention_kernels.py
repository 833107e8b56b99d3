"""Which forward kernel a problem takes (no GPU: the choice is arithmetic on sizes)."""

import pytest

from tests.helpers import attention_kernel

# (B, Sq, Sk, N, Nkv, H) and the faster kernel, with the times (us on a B200) of the tile kernel and of the one for few rows
FEW_ROWS_OR_A_TILE = [
    ((16, 1, 4097, 32, 8, 128), "few rows"),   # 156 / 43: decoding
    ((1, 32, 16384, 4, 4, 128), "few rows"),   # 242 / 29: few heads, keys cut into ranges
    ((32, 4, 4096, 32, 4, 128), "few rows"),   # 296 / 86: a tile per query head reads the keys eight times
    ((512, 4, 64, 16, 16, 64), "few rows"),    # 143 / 80
    ((16, 16, 4096, 32, 32, 64), "few rows"),  # 118 / 88
    ((64, 32, 32, 16, 16, 64), "one tile"),    # 20 / 38: short sequences
    ((64, 32, 32, 16, 16, 128), "one tile"),   # 23 / 98
    ((32, 16, 512, 32, 32, 128), "one tile"),  # 55 / 77
    ((32, 32, 128, 32, 32, 128), "one tile"),  # 23 / 110
    ((16, 32, 4096, 32, 32, 128), "one tile"),  # 169 / 347
    ((8, 17, 512, 32, 32, 128), "one tile"),   # 15 / 36
    ((1, 33, 4096, 1, 1, 64), "one tile"),     # more rows than the kernel has
]


@pytest.mark.parametrize("case,kernel", FEW_ROWS_OR_A_TILE)
def test_few_rows_take_the_faster_kernel(case, kernel):
    assert attention_kernel(*case) == kernel


# (B, Sq, Sk, N, Nkv, H), causal, the faster kernel, and the times with one and with two tiles per CTA
ONE_OR_TWO_TILES = [
    ((16, 4096, 4096, 16, 16, 128), True, "two tiles"),   # 1438 / 1050
    ((8, 4096, 4096, 16, 16, 64), True, "two tiles"),     # 469 / 423
    ((2, 1531, 1531, 32, 8, 128), True, "two tiles"),     # 77 / 59
    ((4, 2048, 2048, 16, 16, 128), False, "two tiles"),
    ((16, 257, 257, 16, 16, 128), True, "one tile"),      # 30 / 41: the second tile of every other CTA has one row
    ((16, 300, 500, 16, 16, 64), False, "one tile"),      # 34 / 43
    ((2, 4096, 4096, 16, 16, 64), False, "one tile"),     # 206 / 224
    ((2, 1100, 1100, 16, 16, 128), True, "one tile"),     # 25 / 31: fewer tiles than the first kernel takes at once
    ((64, 128, 4096, 32, 32, 128), False, "one tile"),    # no second tile
    ((1, 1 << 20, 1 << 20, 1, 1, 128), True, "two tiles"),
]


@pytest.mark.parametrize("case,causal,kernel", ONE_OR_TWO_TILES)
def test_one_or_two_tiles_by_the_faster(case, causal, kernel):
    assert attention_kernel(*case, causal) == kernel


def test_what_the_tensor_core_kernels_do_not_take():
    assert attention_kernel(16, 1, 100, 8, 8, 64, dtype="float32") == "cuda cores"
    assert attention_kernel(16, 1, 100, 8, 8, 96) == "cuda cores"


@pytest.mark.parametrize("source,kernel,registers,count", [("attention_fwd", "attention_fwd_pair_kernel", 168, 2), ("attention_bwd", "attention_bwd_kernelILi128ELb[01]ELi128E", 168, 2),
                                                           ("attention_bwd_atomic", "attention_bwd_atomic_kernel", 128, 1)])
def test_kernels_with_register_budgets_have_the_registers_they_divide(source, kernel, registers, count):
    """Budgets (setmaxnreg) add up to what a block is launched with. Another compiler may assign another number: the library then
    takes its other kernels (or refuses, for the single-kernel backward), which is slower; this is where that shows."""
    import os
    import re

    log = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lumen_b200", "csrc", "build", source + ".ptxas.log")
    if not os.path.exists(log):
        pytest.skip("the library was not built here")
    entries = re.findall(r"Compiling entry function '(\S+)'.*?Used (\d+) registers", open(log).read(), flags=re.S)
    used = [int(n) for name, n in entries if re.search(kernel, name)]
    assert used == [registers] * count
