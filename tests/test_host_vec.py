"""The host's vectorised extension-field arithmetic equals the scalar operations."""
import os
import subprocess


def test_host_vectors(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src = os.path.join(root, "whirlaway_b200", "csrc")
    exe = tmp_path / "hv"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", src, os.path.join(root, "tests", "host_vec_check.cpp"),
                    os.path.join(src, "host_vec.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
