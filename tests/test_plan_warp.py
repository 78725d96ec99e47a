"""The pair plan as the kernel runs it, a lane per field (z80_plan_warp.cuh),
gives the plan of z80_plan.cuh, which the oracle is compared with."""
import os
import subprocess

from conftest import ROOT


def test_plan_by_a_warp(tmp_path):
    exe = tmp_path / "plan_warp_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", str(exe), os.path.join(ROOT, "tests", "native", "plan_warp_check.cpp"),
                    os.path.join(ROOT, "z80-optimizer_b200", "csrc", "z80_tables.cpp"), "-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.startswith("OK"), r.stdout + r.stderr
