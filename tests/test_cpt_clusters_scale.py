"""The compute path tracer's cluster rejection (csrc/cpt_clusters.h) where floats
run out of exponent, on the CPU: no triangle of a rejected cluster is accepted."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_rejection_holds_at_the_ends_of_the_range(tmp_path):
    exe = tmp_path / "test_cpt_clusters_scale"
    cmd = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "include"),
           "-I", os.path.join(ROOT, "vk_cinematic_gb300", "csrc"), "-I", "/usr/local/cuda/include",
           os.path.join(ROOT, "tests", "cpp", "test_cpt_clusters_scale.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
