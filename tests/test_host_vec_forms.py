"""Both forms of the host's extension-field vectors, the AVX-512 one and the scalar one, equal the
scalar operations of kb.cuh, whatever the CPU that runs the tests (a CPU without AVX-512 skips the
vector form)."""
import os
import subprocess

import pytest

FEATURES = {"avx512f", "avx512bw", "avx512dq", "avx512vl"}


def cpu_flags():
    for line in open("/proc/cpuinfo"):
        if line.startswith("flags"):
            return set(line.split())
    return set()


@pytest.mark.parametrize("check", ["host_vec_check", "host_vec_alias_check"])
@pytest.mark.parametrize("form", ["scalar", "vector"])
def test_form(tmp_path, check, form):
    if form == "vector" and not FEATURES <= cpu_flags():
        pytest.skip("this CPU has no AVX-512")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src = os.path.join(root, "whirlaway_b200", "csrc")
    exe = tmp_path / "hv"
    flags = ["-DWL_HOST_VEC_SCALAR"] if form == "scalar" else []
    subprocess.run(["g++", "-O2", "-std=c++17", *flags, "-I", src, os.path.join(root, "tests", check + ".cpp"),
                    os.path.join(src, "host_vec.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), "1" if form == "vector" else "0"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
