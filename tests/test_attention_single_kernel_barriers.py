"""The warps of the single-kernel backward that move dQ' out meet at barriers of their own, which have no limit: no warp may leave in front of one
while another goes there, as when a wait of one has run out (csrc/attention_bwd_atomic.cu)."""

import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lumen_b200", "csrc", "attention_bwd_atomic.cu")


def test_the_warps_stay_together():
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    body = text[text.index("regs_dec<kRegsDrain>") : text.index("bulk_wait_all();\n    } else {")]
    assert re.findall(r"\bfor \(int j = 0;[^)]*\)", body) == ["for (int j = 0; j < n_iter; j++)"]
    assert not re.search(r"\b(break|return|continue)\b", body)
    for barrier in re.finditer(r"\n( *)named_barrier\(1, 128\);", body):
        assert barrier[1] == " " * 12  # in the loop, under no condition
    assert body.count("named_barrier(1, 128)") == 2
