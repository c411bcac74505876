"""The mixed trace's queue, part by part (parts_host.cpp): every ray traced once and within its slot, whatever the
frame, the launch and the heavy slots.  No GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "artful_gb300", "csrc")


def _run(tmp_path, header=None):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    csrc = CSRC
    if header is not None:
        csrc = str(tmp_path)
        (tmp_path / "lensParts.h").write_text(header)
    exe = str(tmp_path / "parts")
    subprocess.run([cxx, "-std=c++17", "-O2", "-I" + csrc, os.path.join(ROOT, "tests", "parts_host.cpp"), "-o", exe],
                   check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout
    return {name: int(value) for name, value in (line.split() for line in out.splitlines())}


def test_every_ray_is_traced_once(tmp_path):
    got = _run(tmp_path)
    assert got["checked"] > 1000000 and got["wrong"] == 0


@pytest.mark.parametrize("old,new", [
    ("(totalUnits - q.heavy) >> lanesLog2", "totalUnits >> lanesLog2"),              # parts past the last ray
    ("q.heavy + ((part - q.heavyParts) << rays)", "part << rays"),                   # light parts from the queue's start
    ("rays = split ? kHeavyRaysLog2 : lanesLog2;", "rays = lanesLog2;"),             # a heavy part of a whole slot
])
def test_a_planted_mistake_is_seen(tmp_path, old, new):
    with open(os.path.join(CSRC, "lensParts.h")) as f:
        text = f.read()
    assert old in text
    assert _run(tmp_path, text.replace(old, new))["wrong"] > 0
