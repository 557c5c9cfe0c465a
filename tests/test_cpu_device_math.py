"""The device math headers compiled as host C++ and checked against the FP64 formulas they replace."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _run(tmp_path, name, *args, units=0):
    exe = str(tmp_path / name)
    src = os.path.join(HERE, "cpp", name + ".cpp")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fno-strict-aliasing", "-w",
                    f"-DHOST_SEED_UNITS={units}", src, "-o", exe], check=True)
    return subprocess.run([exe, *args], check=True, capture_output=True, text=True).stdout.split()


def test_cfl_screen_bounds(tmp_path):
    """lo <= FP64 value <= hi for every state, tight for most: the screen never drops the maximum."""
    bad, n, tight = map(int, _run(tmp_path, "cfl_bounds_check"))
    assert bad == 0 and n == 320000 and tight > n // 2


def test_fp64_on_the_integer_pipe(tmp_path):
    """Division, square root, min, max, comparisons and power-of-two scalings equal the CPU's FP64 bit for bit, with
    seeds off by as much as the GPU's approximations may be."""
    bad, n = map(int, _run(tmp_path, "fp64_int_check", "100000"))
    assert bad == 0 and n > 6_000_000


def test_exact_solvers_match_the_oracle(tmp_path):
    """Slopes, HLLD fluxes and edge EMFs of the exact path equal the oracle's: independent states, states equal to
    within 1e-1 .. 0, low beta, supersonic, unmagnetised, degenerate wave fans, NaN."""
    bad, n = map(int, _run(tmp_path, "exact_solvers_check", "20000"))
    assert bad == 0 and n == 7_000_000


@pytest.mark.parametrize("units", ["0", "1"])
def test_speed_screens_near_equal_speeds(tmp_path, units):
    """Fast speeds nearly equal next to equal sound and Alfven speeds, where the discriminant's error is largest, with the
    FP32 approximations exact and off by one unit in the last place: the largest is the oracle's."""
    bad, n = map(int, _run(tmp_path, "speed_screen_check", "degenerate", "400000", units))
    assert bad == 0 and n == 11 * 400_001


@pytest.mark.parametrize("units", ["0", "1"])
def test_speed_screens_at_any_scale(tmp_path, units):
    """Densities, pressures and squared fields down to the end of the FP32 range and past it, with tiny floors."""
    bad, n = map(int, _run(tmp_path, "speed_screen_check", "scales", "400000", units))
    assert bad == 0 and n == 11 * 400_000


@pytest.mark.parametrize("units", ["0", "1"])
def test_alfven_screen_of_weak_fields(tmp_path, units):
    """Alfven speeds of fields whose squares are near the end of the FP32 range."""
    bad, n = map(int, _run(tmp_path, "speed_screen_check", "weak", "1000000", units))
    assert bad == 0 and n == 11 * 1_000_000


def test_cfl_screen_bounds_with_approximate_reciprocals(tmp_path):
    """As test_cfl_screen_bounds, with reciprocals and reciprocal square roots off by two units in the last place."""
    bad, n, tight = map(int, _run(tmp_path, "cfl_bounds_check", units=2))
    assert bad == 0 and n == 320000 and tight > n // 2
