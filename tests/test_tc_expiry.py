"""After a wait for a matrix product ran out, a block starts no product and waits for the one that
may still run before it frees tensor memory: the threads' account of it, on a model of the block."""
import os
import subprocess


def test_no_product_outlives_its_block(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    exe = tmp_path / "expiry"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(root, "whirlaway_b200", "csrc"),
                    os.path.join(root, "tests", "tc_expiry_host_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
