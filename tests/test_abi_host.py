"""The C ABI's host code over a fake CUDA runtime (abi_host.cpp): what reaches the launches, and what failed
calls leave behind."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "artful_gb300", "csrc")


def test_host_code_over_a_fake_runtime(tmp_path):
    from artful_gb300 import build
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which(build.nvcc()) or build.nvcc()))), "include")
    if not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    exe = str(tmp_path / "abi_host")
    inc = ["-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-I" + cuda]
    objects = []
    for cc, std, source in (("g++", "-std=c++17", os.path.join(ROOT, "tests", "abi_host.cpp")),
                            ("g++", "-std=c++17", os.path.join(CSRC, "abi.cu")),
                            ("gcc", "-std=c11", os.path.join(CSRC, "holeHost.c")),
                            ("gcc", "-std=c11", os.path.join(CSRC, "synthScene.c"))):
        objects.append(str(tmp_path / (os.path.basename(source) + ".o")))
        cmd = [cc, std, "-O1", "-g"] + (["-x", "c++"] if cc == "g++" else []) + inc + ["-c", source, "-o", objects[-1]]
        built = subprocess.run(cmd, capture_output=True, text=True)
        assert built.returncode == 0, built.stderr
    built = subprocess.run(["g++"] + objects + ["-lm", "-ldl", "-o", exe], capture_output=True, text=True)
    assert built.returncode == 0, built.stderr
    run = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and "host checks failed: 0" in run.stdout, run.stdout + run.stderr
