"""Column-pair tables of the guided pass (geometry.cpp) against the axes they
are made from, under AddressSanitizer and UBSan where the compiler has them.
CPU only."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "vapoursynth-lgcr_b200", "csrc")


def test_pair_tables_match_their_axes(tmp_path):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "pair_sweep")
    base = [cxx, "-O1", "-std=c++17", "-ffp-contract=off", "-I", CSRC,
            os.path.join(HERE, "host_sanitize", "pair_sweep.cpp"), os.path.join(CSRC, "geometry.cpp"), "-o", exe]
    if subprocess.run(base + ["-fsanitize=address,undefined"], capture_output=True).returncode != 0:
        subprocess.run(base, check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
