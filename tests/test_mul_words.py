"""The constant-multiply walk's suffix tables (z80b_mul_words.h) keep, for
every effect on A, the smallest suffix that has it."""
import os
import subprocess

from conftest import ROOT


def test_suffix_tables_keep_the_smallest(tmp_path):
    exe = tmp_path / "words_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe), os.path.join(ROOT, "tests", "native", "words_check.cpp")],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.rstrip().endswith("OK words")
