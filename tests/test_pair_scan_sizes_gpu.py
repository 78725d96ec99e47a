"""Pairs of candidates in jobs on both sides of 4,096 targets, where the scan of
the pair index changes from a block per lane to a warp per lane: the rules of
one job are those of its targets searched in small jobs, with lanes that take
several scans (all registers dead: buckets of millions of pairs)."""
import numpy as np
import pytest

import z80b
from test_c3_gpu import dev_keys

pytestmark = pytest.mark.gpu

TEXT = ["LD B, 12h : INC C", "SLA B : SLA B : RES 0, B", "LD A, 12h : INC A : INC A", "INC B : INC B : INC B",
        "LD C, 7 : LD A, C : ADD A, A", "AND 0Fh : RLCA : RLCA"]


@pytest.mark.parametrize("n", [4095, 4096, 4097])
def test_rules_of_a_job_are_those_of_its_parts(ctx, n):
    rng = np.random.default_rng(n)
    base = [z80b.parse_assembly(t) for t in TEXT]
    pick = rng.integers(0, len(base), n)
    targets = [base[p] for p in pick]
    dead = [int(x) for x in rng.choice([0x00, 0xD7, 0xFF], n)]
    dregs = [int(x) for x in rng.choice([0x00, 0x01, 0x3F], n)]
    whole, st = ctx.search(targets, per_target_dead=dead, dead_regs=dregs, max_cand_len=2)
    parts, checked = [], 0
    for lo in range(0, n, 1365):
        hi = min(n, lo + 1365)
        rules, s = ctx.search(targets[lo:hi], per_target_dead=dead[lo:hi], dead_regs=dregs[lo:hi], max_cand_len=2)
        parts += [(k[0] + lo,) + tuple(k[1:]) for k in dev_keys(rules)]
        checked += s.checked_ref
    assert [tuple(k) for k in dev_keys(whole)] == parts
    assert st.checked_ref == checked
    assert len(parts) > 0
