"""Ranks of block-matching candidates (csrc/bm_rank.h) over cost patterns with
NaN and infinite costs, on the CPU: a gap in the ranks leaves a place of the
group's best-4 list unwritten, and the positions read from it would address the
planes anywhere."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "vapoursynth-lgcr_b200", "csrc")


def test_ranks_have_no_gap_and_no_tie(tmp_path):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "bm_rank_sweep")
    base = [cxx, "-O1", "-std=c++17", "-I", CSRC, os.path.join(HERE, "host_sanitize", "bm_rank_sweep.cpp"), "-o", exe]
    if subprocess.run(base + ["-fsanitize=address,undefined"], capture_output=True).returncode != 0:
        subprocess.run(base, check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
