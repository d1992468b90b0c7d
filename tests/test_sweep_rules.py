"""Rules that choose two sweeps per pass (host arithmetic, no GPU involved)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_rules_choose_launchable_passes(tmp_path):
    exe = tmp_path / "sweep_rules_test"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror",
                    os.path.join(ROOT, "tests", "cpp", "sweep_rules_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and "sweep rules ok" in r.stdout, (r.returncode, r.stdout, r.stderr)
