"""Bad targets in jobs large enough for the chunked upload, whose opcodes the
QuickCheck count checks: the lowest bad index is reported, wherever the fault
and in whichever chunk, and the context goes on working."""
import numpy as np
import pytest

import workloads
import z80b

pytestmark = pytest.mark.gpu
N = 70001


@pytest.mark.parametrize("bad", [[0], [40000, 66000], [N - 1], [17500, 17499]])
@pytest.mark.parametrize("index", [1, 0])
def test_lowest_bad_opcode(ctx, bad, index):
    arr = np.ascontiguousarray(workloads.c2_subset(N, seed=2))
    targets = workloads.to_lists(arr)
    broken = [list(t) for t in targets]
    for i in bad:
        broken[i] = [455, 65535]
    ctx.set_option(z80b.OPT_QC_INDEX, index)
    try:
        with pytest.raises(z80b.Z80BError) as e:
            ctx.search(broken)
        assert e.value.status == z80b.EINVAL
        assert f"target {min(bad)}: opcode > 454" in str(e.value)
        if index:
            rules, st = ctx.search(targets)
            assert st.targets == N and len(rules) > 0
    finally:
        ctx.set_option(z80b.OPT_QC_INDEX, 1)


def test_bad_registers_before_bad_opcode(ctx):
    targets = workloads.to_lists(workloads.c2_subset(N, seed=2))
    targets[50000] = [460]
    dregs = [0] * N
    dregs[49999] = 0x40
    with pytest.raises(z80b.Z80BError) as e:
        ctx.search(targets, per_target_dead=[0] * N, dead_regs=dregs)
    assert "target 49999: dead_regs" in str(e.value)
    targets[40000] = [460]
    with pytest.raises(z80b.Z80BError) as e:
        ctx.search(targets, per_target_dead=[0] * N, dead_regs=dregs)
    assert "target 40000: opcode" in str(e.value)
