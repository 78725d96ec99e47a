"""Length-2 candidates at the edges of the pair index: targets of 3, 4 and
more bytes (size classes of the pairs), no, one and all registers dead (no
bucket sharing up to buckets of millions of pairs) and no, some and all flags
dead, against the CPU oracle."""
import pytest

import z80b
from test_c3_gpu import dev_keys

pytestmark = pytest.mark.gpu

TARGETS = ["LD B, 12h : INC C", "SLA B : INC C", "LD B, 12h : LD C, 34h", "LD A, 12h : INC A : INC A",
           "SLA B : SLA B : RES 0, B", "INC B : INC B : INC B"]


@pytest.mark.parametrize("dregs", [0x00, 0x01, 0x3F])
@pytest.mark.parametrize("dead", [0x00, 0xD7, 0xFF])
def test_pair_index_edges(ctx, O, dregs, dead):
    targets = [z80b.parse_assembly(t) for t in TARGETS]
    n = len(targets)
    rules, st = ctx.search(targets, per_target_dead=[dead] * n, dead_regs=[dregs] * n, max_cand_len=2)
    exp, checked = O.search_ext(targets, 2, [dead] * n, [dregs] * n)
    want = [(r.target_index, list(r.src[:r.src_len]), list(r.rep[:r.rep_len]), r.bytes_saved, r.cycles_saved,
             r.dead_flags, r.dead_regs) for r in exp]
    assert dev_keys(rules) == want
    assert st.checked_ref == checked
