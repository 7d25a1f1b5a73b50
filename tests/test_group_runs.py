"""Runs of tile groups within a memory budget (csrc/group_runs.h), on the host."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_group_runs(tmp_path):
    exe = str(tmp_path / "group_runs_check")
    subprocess.run(["g++", "-std=c++17", "-O1", os.path.join(HERE, "group_runs_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=60).stdout
    assert out.strip().endswith("ok")
