"""The FP64 kernels' quotients from a reciprocal pair, on the CPU: ordinary and
infinite numerators as the IEEE division has them, and the stated distance
from a/b where a/b is all but a midpoint of two doubles."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_quotients_from_a_reciprocal_pair(tmp_path):
    exe = tmp_path / "exact_div_test"
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=gnu++17", "-O2", "-ffp-contract=off", "-isystem", cuda,
                    os.path.join(ROOT, "tests", "cpp", "exact_div_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and "exact_div ok" in r.stdout, (r.returncode, r.stdout, r.stderr)
