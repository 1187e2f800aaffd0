"""The task images of the per-subdomain triangular solve, walked on the host (tests/flow_harness.cpp)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_images(tmp_path):
    exe = str(tmp_path / "flow_harness")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fopenmp", "-o", exe, os.path.join(HERE, "flow_harness.cpp")], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
