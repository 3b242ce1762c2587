"""The benchmark's CPU baseline: "unavailable" stands for a missing reference
build alone, and names where it was looked for; a file that is missing later
does not turn a measured baseline into one."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402
from oracle import oracle as O  # noqa: E402


def test_a_missing_reference_build_is_named(monkeypatch):
    monkeypatch.setattr(O, "available", lambda variant: False)
    got = bench.cpu_baseline(None, None)
    assert list(got) == ["unavailable"]
    assert os.path.join("oracle", "_ref") in got["unavailable"]


def test_other_missing_files_are_not_hidden(monkeypatch):
    def missing():
        raise FileNotFoundError(2, "No such file or directory", "/proc/other")
    monkeypatch.setattr(O, "available", lambda variant: True)
    monkeypatch.setattr(bench, "run_cpu", lambda *a, **k: (12.5, 10.0, [1.0, 1.0]))
    monkeypatch.setattr(bench, "reference_scene_fps", lambda: None)
    assert bench.cpu_baseline({}, [])["value"] == 12.5
    monkeypatch.setattr(bench, "host_cpu", missing)
    with pytest.raises(FileNotFoundError, match="/proc/other"):
        bench.cpu_baseline({}, [])
