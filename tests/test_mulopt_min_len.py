"""Constant-multiply searches that leave out the shorter lengths, at lengths
whose prefixes come from the levels of distinct states (the levels' states are
kept apart there, and every last instruction is walked): against answers found
by a walk of every sequence."""
import json
import os

import pytest

import z80b
from conftest import ROOT

DOC = json.load(open(os.path.join(ROOT, "tests", "golden", "mulopt_min_len.json")))["searches"]


def ops_of(n, length, index):
    out = []
    for _ in range(length):
        out.append(index % n)
        index //= n
    return out[::-1]


@pytest.mark.parametrize("i", range(len(DOC)))
def test_fixture_under_the_oracle(O, i):
    s = DOC[i]
    n = O.mul_pool_size(s["pool"])
    for k, length, ts, index in s["results"]:
        seq = ops_of(n, length, index)
        assert s["min_len"] <= length <= s["max_len"]
        assert sum(O.mul_tstates_pool(s["pool"], op) for op in seq) == ts
        assert all(O.mul_run_pool(s["pool"], seq, x, *s["init"]) == (x * k) & 0xFF for x in range(256)), (k, seq)


@pytest.mark.gpu
@pytest.mark.parametrize("i", range(len(DOC)))
def test_min_len_with_states(ctx, i):
    s = DOC[i]
    res, st = ctx.mul_search(s["pool"], tuple(s["init"]), s["min_len"], s["max_len"])
    assert [[r["k"], r["length"], r["tstates"], r["index"]] for r in res if r["found"]] == s["results"]
    n = len(z80b.mul_pool(s["pool"])[0])
    assert st.sequences == sum(n ** l for l in range(s["min_len"], s["max_len"] + 1))


@pytest.mark.gpu
def test_shortest_length_agrees(ctx):
    """A constant whose shortest sequence has the length that the search begins
    with gets the answer of the search from length 1 on."""
    full, _ = ctx.mul_search(z80b.MULPOOL_FAST14, (0, 0, 0), 1, 8)
    part, _ = ctx.mul_search(z80b.MULPOOL_FAST14, (0, 0, 0), 8, 8)
    same = [(a, b) for a, b in zip(full, part) if a["found"] and a["length"] == 8]
    assert len(same) > 10 and all(a == b for a, b in same)
