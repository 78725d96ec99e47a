"""The engine's order of work, its behaviour when a CUDA call fails and what it
keeps: its own object files linked with a CUDA runtime that has no device
(tests/native/fake_cudart.cpp).  No GPU is needed and no kernel runs."""
import os
import subprocess

import pytest

from conftest import PKG, ROOT

NATIVE = os.path.join(ROOT, "tests", "native")
OBJS = [os.path.join(PKG, "_build", f) for f in ("z80b_kernels.o", "z80b_engine.o", "z80_tables.o", "z80b_hostapi.o",
                                                  "z80b_noalloc.o", "z80b_mulopt.o", "z80b_serve.o")]


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = tmp_path_factory.mktemp("engine") / "engine_host_check"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + os.path.join(cuda, "include"), "-o", str(out),
                    os.path.join(NATIVE, "engine_host_check.cpp"), os.path.join(NATIVE, "fake_cudart.cpp"), *OBJS,
                    "-lpthread"], check=True)
    return out


@pytest.mark.parametrize("check", ["error_reported_once", "mul_tables", "mul_no_room", "pair_pool_order", "pair_pool_retry", "chunks",
                                   "verify_events", "verify_copies", "qc_index_memory", "query_counters", "qc_index_debt", "small_graphs"])
def test_engine_host(exe, check):
    r = subprocess.run([str(exe), check], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.startswith("OK " + check), r.stdout + r.stderr


def test_bench_counts_what_comes_back(exe):
    import sys
    sys.path.insert(0, ROOT)
    import bench
    r = subprocess.run([str(exe), "sizes"], capture_output=True, text=True, timeout=600)
    assert r.stdout.split()[:4] == ["OK", "sizes", str(bench.RULE_BYTES), str(bench.REPORT_BYTES)], r.stdout
