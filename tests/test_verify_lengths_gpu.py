"""z80b_verify_pairs on programs of every length it takes (4 + 3 instructions is
the longest pair that is planned): its verdicts against the sweep of every
state without a plan (z80b_exhaustive_noalloc), and against the oracle where
that is quick; and around the number of pairs that go up in one copy.

The pairs share instructions, so that many are proven or have only some of
their outputs and inputs left to sweep."""
import random
import re

import pytest

import z80b
from test_zz_no_alloc import _noalloc

pytestmark = pytest.mark.gpu
REGS = "BCDEHL"


def instructions(allowed, sp):
    """Those of the 8-bit list that name no register but A and `allowed`, by opcode."""
    out = {}
    for w in z80b.pool8():
        text = z80b.disasm([w])
        ops = text.split(" ", 1)[1] if " " in text else ""
        names = re.findall(r"\b(?:BC|DE|HL|SP|[A-EHL])\b(?!h)", ops)
        if "SP" in names and not sp:
            continue
        if set("".join(n for n in names if n != "SP")) - {"A"} <= set(allowed):
            out.setdefault(w & 0xFFFF, []).append(w)
    return list(out.values())


def pair(rng, pool, tl, cl):
    """Programs of tl and cl instructions: the longer one is the shorter with instructions put in, or moved."""
    def any_one():
        return rng.choice(rng.choice(pool))
    short = [any_one() for _ in range(min(tl, cl))]
    long = list(short)
    while len(long) < max(tl, cl):
        at = rng.randrange(len(long) + 1)
        long.insert(at, rng.choice([any_one(), rng.choice(long), 0]))  # 0: NOP
    if rng.random() < 0.4:
        i, j = rng.randrange(len(long)), rng.randrange(len(long))
        long[i], long[j] = long[j], long[i]
    if rng.random() < 0.2:
        long[rng.randrange(len(long))] = any_one()
    return (long, short) if tl >= cl else (short, long)


@pytest.mark.parametrize("tl,cl", [(4, 3), (4, 2), (4, 1), (3, 3), (2, 3), (1, 3), (1, 1)])
def test_lengths_against_unplanned_sweeps(ctx, O, tl, cl):
    rng = random.Random(100 * tl + cl)
    pairs, deads = [], []
    sets = [("".join(rng.sample(REGS, k)), sp) for k in (0, 1, 1, 2, 2, 3, 4) for sp in (False, True)] + [("HL", False)]
    pools = [instructions(*s) for s in sets]
    while len(pairs) < 1200:
        p = pair(rng, rng.choice(pools), tl, cl)
        if O.exhaustive_states(*p) <= 1 << 32:
            pairs.append(p)
            deads.append(rng.choice([0x00, 0x28, 0x01, 0xD7, 0xFF]))
    st, want = _noalloc(pairs, deads)
    assert st == z80b.OK
    got = [bits >> 2 & 1 for bits, _ in ctx.verify_pairs(pairs, dead=deads, tiers=z80b.TIER_EXH)]
    bad = [(O.disasm(t), O.disasm(c), d, g, w) for (t, c), d, g, w in zip(pairs, deads, got, want) if g != w]
    assert not bad, bad[:5]
    assert 30 < sum(got) < len(got) - 30
    checked = 0
    for (t, c), d, g in zip(pairs, deads, got):
        if O.exhaustive_states(t, c) <= 1 << 18 and checked < 200:
            checked += 1
            assert g == int(O.exhaustive(t, c, d)), (O.disasm(t), O.disasm(c), d)
    assert checked == 200


@pytest.mark.parametrize("n", [1, 4096, 4097, 20000])
def test_sizes(ctx, O, n):
    rng = random.Random(n)
    pool = instructions("BC", False)
    base = [pair(rng, pool, 2, 1) for _ in range(50)]
    deads = [rng.choice([0x00, 0x28, 0xFF]) for _ in base]
    want = [int(O.quickcheck(t, c, d)) | int(O.midcheck(t, c, d)) << 1 | int(O.exhaustive(t, c, d)) << 2
            for (t, c), d in zip(base, deads)]
    got = ctx.verify_pairs([base[i % 50] for i in range(n)], dead=[deads[i % 50] for i in range(n)])
    assert got == [(want[i % 50], O.flagdiff(*base[i % 50])) for i in range(n)]
    some = ctx.verify_pairs([base[i % 50] for i in range(n)], dead=[deads[i % 50] for i in range(n)],
                            tiers=z80b.TIER_QC | z80b.TIER_MID)
    assert [b for b, _ in some] == [w & 3 for w in (want[i % 50] for i in range(n))]
    without = ctx.verify_pairs([base[i % 50] for i in range(n)], tiers=z80b.TIER_EXH)
    alive = [int(O.exhaustive(t, c, 0)) << 2 for t, c in base]
    assert [b for b, _ in without] == [alive[i % 50] for i in range(n)]
