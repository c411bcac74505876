"""The mixed trace's double-float arithmetic on the host (pairs_host.cpp): no further from exact values than pairs
renormalised at every operation, over the scenes' range of eyes.  No GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "artful_gb300", "csrc")
VALUES = ["invEnergy", "xi", "big", "uA", "uB", "uC", "xiA",
          "radial_x", "radial_v", "radial_first", "polar_x", "polar_v", "polar_first"]


@pytest.fixture(scope="module")
def measured(tmp_path_factory):
    cxx, cc = shutil.which("g++"), shutil.which("gcc")
    if not cxx or not cc:
        pytest.skip("no C++ compiler")
    tmp = tmp_path_factory.mktemp("pairs")
    objects = []
    for name in ("holeHost", "synthScene"):
        objects.append(str(tmp / (name + ".o")))
        subprocess.run([cc, "-std=c11", "-O2", "-ffp-contract=off", "-I" + os.path.join(ROOT, "include"), "-c",
                        os.path.join(CSRC, name + ".c"), "-o", objects[-1]], check=True)
    exe = str(tmp / "pairs")
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC,
                    os.path.join(ROOT, "tests", "pairs_host.cpp")] + objects + ["-lm", "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return {name: float(value) for name, value in (line.split() for line in out.splitlines())}


@pytest.mark.parametrize("name", VALUES)
def test_errors_are_the_renormalised_pairs(measured, name):
    """Both are measured on the same rays, so the quantiles' own noise is theirs in common; what is left of it is a
    third of a per cent or less (1 % allowed, 2 % of the 99.9 % quantile's few values).  Pairs that are never
    renormalised are 7 to 50 % off in the median and 20 to 80 % at 99.9 %, in all but the small parts' sums."""
    assert measured[name + "_count"] > 1e5
    assert measured[name + "_log2"] < -46.5
    assert measured[name + "_median"] <= 1.01
    assert measured[name + "_99"] <= 1.01
    assert measured[name + "_999"] <= 1.02


def test_kept_values_are_normalised(measured):
    assert measured["loose"] == 0


def test_the_axis_cubic_keeps_its_bits(measured):
    """a^2 - K as a pair, whether the ray's constants are pairs or float: one renormalised difference of values of
    48 and 24 bits, 2^-47 of their size."""
    assert measured["axis_log2"] <= -47.0


def test_a_double_is_its_float_and_its_rest(measured):
    assert measured["lost"] == 0
