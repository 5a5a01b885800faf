"""The number ranges of the fixed-point geodesic (csrc/fixed_geodesic.cuh) on
the CPU: a build in which every product, shift and sum that loses bits of its
value, and every shift by a word's length or more (which differs between
machines), ends the program, and so does a sum of products whose cross terms
could come to more than 64 bits, over both ends of the grids' range and views
from the polar axis to the equator.  A product that wraps is off by its
format's range, and the ray by 1e-4 or far more: its final state is held to
1e-7 of long double."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TESTS = os.path.join(ROOT, "tests")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("kept") / "fixed_check")
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fsanitize=signed-integer-overflow,shift",
                    "-fsanitize-undefined-trap-on-error", "-include", os.path.join(TESTS, "fixed_kept.h"),
                    "-x", "c++", "-o", exe, os.path.join(TESTS, "fixed_check.cpp"), "-lm"], check=True)
    return exe


@pytest.mark.parametrize("inclination", [1.0, 2.0, 5.0, 10.0, 17.0, 30.0, 90.0, 160.0, 179.0])
@pytest.mark.parametrize("hslope", [0.2, 1.0, 1.4, 1.8])
def test_no_bits_are_lost(check, hslope, inclination):
    for eps, integ, spin in ((0.05, 4, 0.9375), (0.1, 2, -0.998)):
        run = subprocess.run([check, "500", str(eps), str(integ), str(spin), str(hslope), str(inclination), "40", "3"],
                             capture_output=True, text=True)
        assert run.returncode == 0, "an operation lost bits of its value"
        worst = float(run.stdout.split()[13])
        assert worst <= 1e-7, worst


@pytest.mark.parametrize("case", ["150 0.02 2 0.9999 0.37148528972428885 177.03208629875422 40 836910",
                                  "300 0.02 2 0.9999 0.2 4.903135877080161 40 577980",
                                  "300 0.02 4 0.9999 1.8 1.3047726026769095 40 364885"])
def test_no_ray_jumps(check, case):
    """Rays that wind long close to a fast hole, where the cross terms of three
    products fill more than 64 bits: no ray is more than eight times as far
    off as its double-precision counterpart (beyond 1e-13)."""
    run = subprocess.run([check, *case.split()], capture_output=True, text=True)
    assert run.returncode == 0, "an operation lost bits of its value"
    assert float(run.stdout.split()[12]) <= 8.0


@pytest.mark.parametrize("case", ["20 0.002 2 0.9375 0.3 60 40 7", "20 0.002 2 0.5 1.0 175 40 7"])
def test_rk2_roundings_do_not_add_up(check, case):
    """Thousands of midpoint steps: the root mean square error of every state
    component is at most the double-precision one (or 2^-52)."""
    run = subprocess.run([check, *case.split()], capture_output=True, text=True)
    vals = list(map(float, run.stdout.split()))
    for fixed, double in zip(vals[0:12:2], vals[1:12:2]):
        assert fixed <= max(double, 2.0 ** -52), vals


def test_symmetry_is_kept(tmp_path):
    """Exact zeros of a ray's state stay exact: the sums' starts, which make up
    for what floors lose on average, do not act where nothing is rounded."""
    exe = str(tmp_path / "symmetry")
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-x", "c++", "-o", exe,
                    os.path.join(TESTS, "fixed_symmetry_check.cpp"), "-lm"], check=True)
    steps = list(map(int, subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()))
    assert len(steps) == 54 and min(steps) > 100, steps
