"""All-hits searches over uploaded candidate lists at both sides of the size
where the QuickCheck index goes from all dead-register masks in one sort to a
sort per mask in use: the index gives what the scan over every candidate gives."""
import numpy as np
import pytest

import workloads
import z80b

pytestmark = pytest.mark.gpu


def first_op_list():
    o = workloads.ops()
    return list(z80b.pool8()) + [z80b.pack(o[n], i) for n in ("LD_BC_NN", "LD_DE_NN", "LD_HL_NN", "LD_SP_NN")
                                 for i in range(65536)]


@pytest.mark.parametrize("n_cands", [1, 65536, 65537, 266675])
def test_index_equals_scan(n_cands):
    rng = np.random.default_rng(n_cands)
    targets = workloads.to_lists(workloads.c2_subset(600, seed=11))
    dead = [int(x) for x in rng.choice([0x00, 0x28, 0xFF], size=len(targets))]
    dregs = [int(x) for x in rng.choice([0x00, 0x01, 0x30, 0x3F], size=len(targets))]
    got = []
    with z80b.Context(0) as ctx:
        ctx.load_candidates(first_op_list()[-n_cands:])
        for index in (1, 0):
            ctx.set_option(z80b.OPT_QC_INDEX, index)
            # without dead registers first: their masks are indexed by the second search
            a, sa = ctx.search(targets, dead_flags=0x28, mode=z80b.MODE_ALL)
            b, sb = ctx.search(targets, per_target_dead=dead, dead_regs=dregs, mode=z80b.MODE_ALL)
            got.append(([r.key() for r in a], [r.key() for r in b], sa.checks, sb.checks, sa.qc_survivors,
                        sb.qc_survivors))
    assert got[0] == got[1]
    assert n_cands < 266675 or len(got[0][1]) > 0  # the last 65,536 entries load SP: no target here does
