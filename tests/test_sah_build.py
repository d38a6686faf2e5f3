"""The host SAH build against a sweep over every bin (tests/cpp)."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_tree_is_the_one_of_the_full_sweep(tmp_path):
    exe = tmp_path / "test_sah_build"
    csrc = os.path.join(ROOT, "vk_cinematic_gb300", "csrc")
    cmd = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", csrc, "-I", "/usr/local/cuda/include",
           os.path.join(ROOT, "tests", "cpp", "test_sah_build.cpp"), os.path.join(csrc, "sah_build.cpp"),
           "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
