"""The division of a single-pass launch among the SMs (launch_split.h)."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


def test_columns_are_covered_once_and_waves_are_not_wasted(tmp_path):
    cxx = shutil.which("c++") or shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "launch_split_check"
    subprocess.run([cxx, "-O2", "-std=c++17", str(HERE / "launch_split_check.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout
