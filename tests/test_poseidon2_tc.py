"""The tensor-core Poseidon2-24 of the Merkle leaves.

CPU: the permutation's arithmetic, restated on the host over the same tables, equals the plain
one, and every intermediate stays in the range its exactness rests on.
GPU: proofs whose commitments have less than one tile of 128 leaf rows, exactly one, and several,
at every number of tiles a block, and through the one-absorption-per-launch path of a host
witness, equal the oracle's."""
import os
import subprocess

import numpy as np
import pytest


def test_permutation_on_host(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    exe = tmp_path / "p2tc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(root, "whirlaway_b200", "csrc"),
                    os.path.join(root, "tests", "poseidon2_tc_host_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("plan", [0, 1, 2])
@pytest.mark.parametrize("log_n,skips", [(4, 3), (5, 4), (6, 4), (9, 4)])
def test_leaf_tiles_match_oracle(oracle, wl, ctx, log_n, skips, plan):
    """2^(log_n + 2) leaf rows: 64, 128, 256 and 2048."""
    settings = wl.AirSettings(univariate_skips=skips)
    consts, inputs = oracle.workload(log_n, 21)
    wit = oracle.trace(log_n, consts, inputs)
    ref, _ = oracle.prove(log_n, consts, wit, settings.as_array())
    table = wl.AirTable(ctx, consts, log_n, settings)
    wl.tune_force("leaf", plan)
    try:
        w = wl.Witness.generate(ctx, consts, inputs, log_n)
        got = table.prove_witness(w)
        w.free()
        got_host = table.prove(wit)
    finally:
        wl.tune_force("leaf", -1)
    assert np.array_equal(got, ref)
    assert np.array_equal(got_host, ref)
