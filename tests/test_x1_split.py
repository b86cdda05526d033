"""The rule that splits the x1 sweep over warps (csrc/x1_split.cuh), on the host
over all that it accepts: the items cover every cell once, their windows stay in
their rows, and no item reads the ghost cells that another one revises."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_every_split_is_sound(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "x1_split_check"
    src = os.path.join(HERE, "cpp", "x1_split_check.cpp")
    subprocess.run([cxx, "-O2", "-std=c++17", "-x", "c++", src, "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    n, faults = out.split()[-3], out.split()[-1]
    assert int(n) > 100000 and int(faults) == 0, out
