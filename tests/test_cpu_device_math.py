"""The device math headers compiled as host C++ and checked against the FP64 formulas they replace."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _run(tmp_path, name, *args):
    exe = str(tmp_path / name)
    src = os.path.join(HERE, "cpp", name + ".cpp")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fno-strict-aliasing", "-w", src, "-o", exe], check=True)
    return subprocess.run([exe, *args], check=True, capture_output=True, text=True).stdout.split()


def test_cfl_screen_bounds(tmp_path):
    """lo <= FP64 value <= hi for every state, tight for most: the screen never drops the maximum."""
    bad, n, tight = map(int, _run(tmp_path, "cfl_bounds_check"))
    assert bad == 0 and n == 320000 and tight > n // 2
