"""The warps of the single-kernel backward that move dQ' out meet at barriers of their own, which have no limit: no warp may leave in front of one
while another goes there, as when a wait of one has run out (csrc/attention_bwd_atomic.cu)."""

import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lumen_b200", "csrc", "attention_bwd_atomic.cu")


def test_the_warps_leave_together():
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    loop = text[text.index("regs_dec<kRegsDrain>") : text.index("bulk_wait_all();")]
    body = loop[loop.index("for (int j = 0; j < n_iter && ok; j++)") :]
    vote = re.search(r"if \(!\(ok = named_barrier_all\(1, 128, ok\)\)\) break;", body)
    assert vote and not re.search(r"\b(break|return|continue)\b", body[: vote.start()])
    assert len(re.findall(r"\b(break|return|continue)\b", body)) == 1 and body.count("named_barrier(1, 128)") == 1
