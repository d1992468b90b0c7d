"""Graph captures report every error: a host test of the capture helper with
a fake of the failing runtime calls, no GPU involved.  A segment whose launch
was refused must not become a graph without that launch."""
import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_error_of_a_capture_is_reported(tmp_path):
    exe = tmp_path / "capture_test"
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-isystem", cuda,
                    os.path.join(ROOT, "tests", "cpp", "capture_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and "capture ok" in r.stdout, (r.returncode, r.stdout, r.stderr)


def test_captures_go_through_the_helper():
    """No segment is captured beside capture_graph (the loop graphs capture
    into a body of their own and test cudaGetLastError themselves)."""
    for path in glob.glob(os.path.join(ROOT, "lbm_b200", "csrc", "*.cu")):
        assert not re.search(r"cudaStreamBeginCapture\(", open(path).read()), path
