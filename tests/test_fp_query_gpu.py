"""Fingerprint queries around the number of hits that one launch hands back by
itself, in sequence on one context (a query leaves its counters cleared)."""
import pytest

import z80b

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 2046, 2047, 3000])
def test_hit_counts(n):
    nop, inc = z80b.parse_assembly("NOP")[0], z80b.parse_assembly("INC A")[0]
    cands = [inc] + [nop] * n + [inc]
    with z80b.Context(0) as ctx:
        ctx.load_candidates(cands)
        fn, fi = ctx.fingerprints([[nop], [inc]], 1)
        for _ in range(2):
            assert ctx.quickcheck_gpu(fn) == list(range(1, n + 1))
            assert ctx.quickcheck_gpu(fi) == [0, n + 1]
        if n:
            with pytest.raises(z80b.Z80BError) as e:
                ctx.quickcheck_gpu(fn, cap=n - 1) if n > 1 else ctx.quickcheck_gpu(fi, cap=1)
            assert e.value.status == z80b.ECAPACITY
