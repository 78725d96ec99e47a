"""Pair planning (z80_plan.cuh): proofs by value numbers and the sweeps left
after them, compiled for the host and compared with the CPU oracle."""
import os
import subprocess

from conftest import ROOT


def test_pair_plans_against_oracle(tmp_path):
    """A pair that the planning proves passes the oracle's ExhaustiveCheck,
    and every planned sweep gives the oracle's verdict; the per-opcode flow
    tables hold under the oracle's Exec."""
    exe = tmp_path / "plan_check"
    srcs = [os.path.join(ROOT, "tests", "native", "plan_check.cpp"),
            os.path.join(ROOT, "z80-optimizer_b200", "csrc", "z80_tables.cpp"),
            os.path.join(ROOT, "oracle", "z80_oracle_isa_cpu.cpp"),
            os.path.join(ROOT, "oracle", "z80_oracle_search.cpp")]
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe)] + srcs + ["-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("OK")
