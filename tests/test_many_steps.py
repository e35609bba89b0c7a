"""A refused cooperative launch leaves its steps to plain launches (tests/cpp/run_many_steps.cpp, with a fake of the
launch that is refused)."""
import os
import subprocess

from conftest import ROOT

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_refused_launches(tmp_path):
    exe = os.path.join(str(tmp_path), "run_many_steps")
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", f"-I{CUDA}/include",
                    f"-I{ROOT}/hippolbm_b200/csrc", os.path.join(ROOT, "tests", "cpp", "run_many_steps.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
