"""The dK/dV kernel that leaves dS in memory divides the registers of its block like the one that does not (csrc/attention_bwd.cu)."""

import os
import re

import pytest

LOG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lumen_b200", "csrc", "build", "attention_bwd.ptxas.log")


def test_a_kernel_of_its_own_with_the_registers_it_divides():
    if not os.path.exists(LOG):
        pytest.skip("the library was not built here")
    entries = re.findall(r"Compiling entry function '(\S+)'.*?Used (\d+) registers", open(LOG).read(), flags=re.S)
    assert [int(n) for name, n in entries if "attention_bwd_kernelILi128ELb1ELi129E" in name] == [168]
