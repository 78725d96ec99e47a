"""The work of this library, case by case, through its C ABI and Python binding.

Every case is a call that a program using the library makes, on seeded
synthetic inputs of the workloads that the benchmark, the tests and the tools
use: searches of whole enumerations and of small jobs, uneven jobs with dead
registers and two-instruction candidates, all-hits searches, re-verification
of rules, single fingerprint queries, constant-multiply searches and served
queries.  A program keeps one context per role (candidates are uploaded once,
the two-instruction pool is built once) and hands over host arrays, so the
contexts are kept here and every pass is a whole call from host arrays to
host arrays.
"""
import ctypes
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "z80-optimizer_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import workloads  # noqa: E402
import z80b  # noqa: E402

U8P = ctypes.POINTER(ctypes.c_uint8)
U32P = ctypes.POINTER(ctypes.c_uint32)

# ------------------------------------------------------------------ cases

# kind "search": z80b_search.  `source` says where the targets come from:
#   pairs   length-2 sequences over the whole 8-bit list, in enumeration order
#           (z80opt enumerate), every one of them or a seeded sample
#   small   length-2 sequences over the reduced register/ALU pool of the small
#           configuration, its immediates drawn from the seed
#   uneven  60% length 2, 40% length 3, drawn instruction by instruction, each
#           with its own dead flags and dead registers
#   query   the served mix: lengths 2 to 4, own dead flags and registers
_LISTED = [
    # z80opt target: one sequence, is there a shorter single instruction?
    {"name": "target_one", "kind": "search", "source": "pairs", "n": 1, "cand": 1, "dead": 0x00, "mode": 0},
    # the z80qc query: one fingerprint against the uploaded first-op list
    {"name": "fingerprint_query", "kind": "quickcheck", "dead": 0x28},
    # the small configuration: every pair over the reduced pool
    {"name": "small_pool", "kind": "search", "source": "small", "n": 50000, "cand": 1, "dead": 0x00, "mode": 0},
    # the parity subset with every flag dead: full and masked pass per target
    {"name": "pairs_100k_masked", "kind": "search", "source": "pairs", "n": 100003, "cand": 1, "dead": 0xFF, "mode": 0},
    # the headline: (nearly) the whole length-2 enumeration in one job
    {"name": "pairs_9m", "kind": "search", "source": "pairs", "n": 9437183, "cand": 1, "dead": 0x00, "mode": 0},
    # gpu.SearchGPU semantics: every passing candidate, undocumented flags dead
    {"name": "all_hits_30k", "kind": "search", "source": "pairs", "n": 30011, "cand": 1, "dead": 0x28, "mode": 1},
    # a small uneven job with candidates of up to two instructions
    {"name": "uneven_200", "kind": "search", "source": "uneven", "n": 200, "cand": 2, "dead": 0x00, "mode": 0},
    # the batched uneven workload
    {"name": "uneven_40k", "kind": "search", "source": "uneven", "n": 40009, "cand": 2, "dead": 0x00, "mode": 0},
    # z80opt verify-jsonl: a rule file through all three tiers
    {"name": "verify_rules", "kind": "verify", "n": 3001, "dead": 0xFF},
    # z80opt mulopt -k: one constant over the reference's 14-op pool
    {"name": "multiply_one", "kind": "mul", "pool": 0, "nk": 1, "max_len": 6},
    # the constant-multiply workload: (nearly) every constant, 21 ops, lengths 1..9
    {"name": "multiply_all", "kind": "mul", "pool": 1, "nk": 250, "max_len": 9},
    # a burst of queries at the serving loop
    {"name": "serve_300", "kind": "serve", "n": 300},
]


def listed():
    return [dict(c) for c in _LISTED]


def _log_int(rng, lo, hi):
    return int(round(float(lo) * (float(hi) / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["pairs", "pairs", "small", "hits", "uneven", "uneven", "verify", "mul", "serve", "quickcheck"])
    dead = rng.choice([0x00, 0x28, 0xFF, rng.randrange(1, 256)])
    if kind == "pairs":
        return {"kind": "search", "source": "pairs", "n": _log_int(rng, 1, 2000000 if dead else 9400000), "cand": 1,
                "dead": dead, "mode": 0}
    if kind == "small":
        return {"kind": "search", "source": "small", "n": _log_int(rng, 100, 50000), "cand": 1, "dead": dead, "mode": 0}
    if kind == "hits":
        return {"kind": "search", "source": "pairs", "n": _log_int(rng, 1, 30000), "cand": 1, "dead": dead, "mode": 1}
    if kind == "uneven":
        return {"kind": "search", "source": "uneven", "n": _log_int(rng, 8, 40000), "cand": rng.choice([1, 2, 2]),
                "dead": 0x00, "mode": 0}
    if kind == "verify":
        return {"kind": "verify", "n": _log_int(rng, 16, 3000), "dead": dead}
    if kind == "mul":
        pool = rng.choice([0, 1, 2, 3])
        return {"kind": "mul", "pool": pool, "nk": _log_int(rng, 1, 250),
                "max_len": rng.randint(3, 8 if pool in (1, 3) else 9)}
    if kind == "serve":
        return {"kind": "serve", "n": _log_int(rng, 32, 300)}
    return {"kind": "quickcheck", "dead": rng.randrange(256)}


# ------------------------------------------------- what a program keeps

_kept = {}


def _context(role):
    """The program's context for a role, made (and warmed) once."""
    if role not in _kept:
        ctx = z80b.Context(0)
        if role == "two":
            # one query per dead-register mask: the two-instruction pool and
            # its indexes are built before the first job
            t = [[z80b.parse_assembly("LD A, 00h")[0], z80b.parse_assembly("INC B")[0],
                  z80b.parse_assembly("INC B")[0]]] * 64
            ctx.search(t, per_target_dead=[0x28] * 64, dead_regs=list(range(64)), max_cand_len=2)
        elif role == "firstop":
            ctx.load_candidates(_first_op())
        _kept[role] = ctx
    return _kept[role]


def _first_op():
    if "first_op" not in _kept:
        o = workloads.ops()
        v = list(z80b.pool8())
        for name in ("LD_BC_NN", "LD_DE_NN", "LD_HL_NN", "LD_SP_NN"):
            v += [z80b.pack(o[name], i) for i in range(65536)]
        _kept["first_op"] = v
    return _kept["first_op"]


def _server():
    if "server" not in _kept:
        _context("two")  # the pool is shared by the contexts of a device
        _kept["server"] = z80b.Server(workers=4)
    return _kept["server"]


# --------------------------------------------------------------- inputs

def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).pin_memory()


def _pairs(n, rng):
    """n length-2 targets in enumeration order, a seeded sample."""
    every = workloads.c2_targets()
    if n > len(every) // 2:
        keep = np.ones(len(every), dtype=bool)
        keep[rng.choice(len(every), size=len(every) - n, replace=False, shuffle=False)] = False
        return every[keep]
    if n > 64:
        return every[np.unique(rng.integers(0, len(every), size=n + n // 4 + 64))[:n]]
    # a program that asks about a few sequences suspects them: half of them, and the only one, have a shorter form
    sample = every[np.unique(rng.integers(0, len(every), size=4096))]
    s = _job(sample, None, None, None, {"cand": 1, "dead": 0, "mode": 0})
    s["ctx"] = _context("one")
    found = run(s)["rules"][:s["nr"].value, 13]
    half = rng.choice(found, size=(n + 1) // 2, replace=False)
    rest = rng.choice(np.setdiff1d(np.arange(len(sample)), half), size=n // 2, replace=False)
    return sample[np.sort(np.concatenate([half, rest]))]


def _queries(n, rng, lengths, weights):
    """n sequences drawn instruction by instruction, pruned ones redrawn, with dead flags and registers."""
    pool = np.array(z80b.pool8(), dtype=np.uint32)
    lens = rng.choice(lengths, size=n, p=weights).astype(np.uint8)
    out = np.zeros((n, 4), dtype=np.uint32)
    todo = np.arange(n)
    while len(todo):
        out[todo] = pool[rng.integers(0, len(pool), size=(len(todo), 4))]
        for k in range(4):
            out[todo[lens[todo] <= k], k] = 0
        todo = todo[workloads.prune_mask(out[todo], lens[todo])]
    bits = rng.integers(0, 64, size=n)
    dead = np.zeros(n, dtype=np.uint8)
    for i, f in enumerate(workloads.DOC_FLAGS):
        dead |= np.where((bits >> i) & 1, f, 0).astype(np.uint8)
    return out, lens, dead, rng.integers(0, 64, size=n).astype(np.uint8)


def _job(arr, lens, dead, dregs, case):
    """A z80b_job over host arrays (targets in pinned memory) and its output buffers."""
    n = len(arr)
    tgt = _pinned(arr)
    keep = [tgt]
    job = z80b.Job()
    job.targets = ctypes.cast(tgt.data_ptr(), U32P)
    for field, a in (("target_lens", lens), ("dead_flags", dead), ("dead_regs", dregs)):
        if a is not None:
            a = np.ascontiguousarray(a)
            keep.append(a)
            setattr(job, field, a.ctypes.data_as(U8P))
    job.n_targets, job.target_len, job.target_stride = n, arr.shape[1] if lens is None else 0, arr.shape[1]
    job.max_cand_len, job.global_dead_flags, job.mode, job.path = case["cand"], case["dead"], case["mode"], z80b.PATH_BATCHED
    # room for the rules: one pair in fifteen has one, one in five with dead flags, two in three uneven targets; an
    # all-hits search with every flag dead returns more than one per target
    cap = (4 * n if case["mode"] == z80b.MODE_ALL else n // 8 if lens is None and case["dead"] == 0 else n) + 4096
    rules = np.zeros((cap, 16), dtype=np.int32)
    return {"do": "search", "job": job, "keep": keep, "rules": rules, "cap": cap, "nr": ctypes.c_uint64(),
            "stats": z80b.Stats()}


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "search":
        if case["source"] == "uneven":
            arr, lens, dead, dregs = _queries(case["n"], rng, [2, 3], [0.6, 0.4])
            st = _job(arr, lens, dead, dregs, case)
        else:
            if case["source"] == "small":
                arr = workloads.c1_targets(int(rng.integers(1 << 30)))
                arr = arr[np.sort(rng.choice(len(arr), size=min(case["n"], len(arr)), replace=False, shuffle=False))]
            else:
                arr = _pairs(case["n"], rng)
            st = _job(arr, None, None, None, case)
        st["ctx"] = _context("two" if case["cand"] == 2 else "hits" if case["mode"] == z80b.MODE_ALL else "one")
        return st
    if kind == "quickcheck":
        ctx = _context("firstop")
        c = _first_op()[int(rng.integers(len(_first_op())))]
        fp = np.frombuffer(ctx.fingerprints([[c]], 1)[0], dtype=np.uint8).copy()
        return {"do": "quickcheck", "ctx": ctx, "fp": fp, "dead": case["dead"],
                "hits": np.zeros(len(_first_op()), dtype=np.int32), "nh": ctypes.c_uint32()}
    if kind == "verify":
        # the rules of a search, one in eight with another rule's replacement
        n = case["n"]
        s = _job(_pairs(40 * n + 200, rng), None, None, None, {"cand": 1, "dead": case["dead"], "mode": 0})
        s["ctx"] = _context("one")
        rules = run(s)["rules"][:s["nr"].value]
        rules = rules[np.sort(rng.choice(len(rules), size=min(n, len(rules)), replace=False, shuffle=False))]
        n = len(rules)
        tgt = np.ascontiguousarray(rules[:, 0:4]).view(np.uint32)
        cand = np.ascontiguousarray(rules[:, 4:8]).view(np.uint32)
        wrong = rng.random(n) < 0.125
        cand[wrong] = np.roll(cand, 1, axis=0)[wrong]
        arrays = [tgt, rules[:, 8].astype(np.uint8), cand, rules[:, 9].astype(np.uint8), rules[:, 12].astype(np.uint8)]
        return {"do": "verify", "ctx": _context("one"), "a": arrays, "n": n, "out": np.zeros(n, dtype=np.uint8),
                "flagdiff": np.zeros(n, dtype=np.uint8)}
    if kind == "mul":
        ks = np.sort(rng.choice(np.arange(2, 256), size=case["nk"], replace=False)).astype(np.int32)
        # the 21-op workload draws its initial B, C and F; the reference's pools start at zero
        init = workloads.mul_init(int(rng.integers(1 << 30))) if case["pool"] == z80b.MULPOOL_WIDE21 else (0, 0, 0)
        return {"do": "mul", "ctx": _context("one"), "pool": case["pool"], "init": init, "max_len": case["max_len"],
                "ks": ks, "out": np.zeros((len(ks), 10), dtype=np.int32)}
    n = case["n"]
    arr, lens, dead, dregs = _queries(n, rng, [1, 2, 3, 4], [0.5, 0.3, 0.15, 0.05])
    qs = (z80b.Query * n)()
    for i in range(n):
        qs[i].id = i
        qs[i].len, qs[i].dead_flags, qs[i].dead_regs = int(lens[i]), int(dead[i]), int(dregs[i])
        for k in range(4):
            qs[i].target[k] = int(arr[i, k])
    return {"do": "serve", "server": _server(), "queries": qs, "n": n, "got": (z80b.Answer * n)()}


# ----------------------------------------------------------------- passes

_ANSWER = np.dtype([("id", "<u8"), ("head", "<i4", (2,)), ("rules", "<i4", (2, 16)), ("ms", "<f8", (3,)),
                    ("batch", "<u4"), ("flags", "<u4")])


def run(s):
    L = z80b.lib()
    do = s["do"]
    if do == "search":
        ctx, st = s["ctx"], s["stats"]
        rules = s["rules"]
        ctx._check(L.z80b_search(ctx._h, ctypes.byref(s["job"]), ctypes.cast(rules.ctypes.data, ctypes.POINTER(z80b.Rule)),
                                 s["cap"], ctypes.byref(s["nr"]), ctypes.byref(st)))
        return {"rules": rules, "n_rules": s["nr"].value, "checks": st.checks, "checked_ref": st.checked_ref,
                "qc_survivors": st.qc_survivors}
    if do == "quickcheck":
        ctx = s["ctx"]
        ctx._check(L.z80b_quickcheck(ctx._h, s["fp"].ctypes.data_as(U8P), s["dead"], s["hits"].ctypes.data_as(U32P),
                                     len(s["hits"]), ctypes.byref(s["nh"])))
        return {"n": s["nh"].value, "hits": s["hits"]}
    if do == "verify":
        ctx, (tgt, tl, cand, cl, dead) = s["ctx"], s["a"]
        ctx._check(L.z80b_verify_pairs(ctx._h, tgt.ctypes.data_as(U32P), tl.ctypes.data_as(U8P), cand.ctypes.data_as(U32P),
                                       cl.ctypes.data_as(U8P), 4, s["n"], dead.ctypes.data_as(U8P), 7,
                                       s["out"].ctypes.data_as(U8P), s["flagdiff"].ctypes.data_as(U8P)))
        return {"tiers": s["out"], "flagdiff": s["flagdiff"]}
    if do == "mul":
        ctx = s["ctx"]
        b, c, f = s["init"]
        ctx._check(L.z80b_mul_search(ctx._h, s["pool"], b, c, f, 1, s["max_len"],
                                     s["ks"].ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), len(s["ks"]),
                                     ctypes.cast(s["out"].ctypes.data, ctypes.POINTER(z80b.MulResult)), None))
        return {"results": s["out"]}
    # serve: one burst, then the answers as they come
    h, n, got = s["server"]._h, s["n"], s["got"]
    if L.z80b_server_submit(h, s["queries"], n) != z80b.OK:
        raise z80b.Z80BError(z80b.EINVAL, "z80b_server_submit failed")
    have, k = 0, ctypes.c_uint32()
    while have < n:
        at = ctypes.cast(ctypes.byref(got, have * ctypes.sizeof(z80b.Answer)), ctypes.POINTER(z80b.Answer))
        if L.z80b_server_poll(h, at, n - have, ctypes.byref(k), 100) != z80b.OK:
            raise z80b.Z80BError(z80b.EINVAL, "z80b_server_poll failed")
        have += k.value
    a = np.frombuffer(got, dtype=_ANSWER)
    a = a[np.argsort(a["id"])]
    return {"status_and_rules": a["head"], "rules": a["rules"], "flags": a["flags"].astype(np.int32)}


# ------------------------------------------------------------------- work

def work(case):
    """Bytes in and out of one pass: programs and masks in, rules (or verdicts, or hits) out.  The operations are
    integer ones (emulated instructions), so no floating-point work is stated."""
    kind = case["kind"]
    if kind == "search":
        if case["source"] in ("uneven",):
            per = 16 + 3 + 40 if case["cand"] == 2 else 16 + 3 + 8
        else:
            per = 8 + (24 if case["dead"] == 0xFF else 8)
        return {"bytes": case["n"] * per, "flops": 0}
    if kind == "quickcheck":
        # the flag and A bytes alone decide nearly every candidate: one 16-byte output each
        return {"bytes": 266675 * 16 + 80, "flops": 0}
    if kind == "verify":
        return {"bytes": case["n"] * (2 * 16 + 5), "flops": 0}
    if kind == "mul":
        return {"bytes": case["nk"] * (4 + 40), "flops": 0}
    return {"bytes": case["n"] * (32 + 200), "flops": 0}


def exact(case, seed):
    """Every output is a whole number (opcodes, masks, savings, counters, indices): compared as they are."""
    return None
