"""The sumcheck tails that start on a cluster of blocks: proofs where the launch holds one, two or three
cluster rounds before one block goes on alone, or ends while still on the cluster."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0x7F000001


# points of the a*b - c sumcheck's round 1: 512, 1024, 2048 (the launch takes all rounds), 4096
@pytest.mark.parametrize("log_n,skips", [(11, 1), (12, 1), (14, 2), (14, 1), (15, 3)])
def test_abc_cluster_tail_matches_oracle(oracle, wl, ctx, log_n, skips):
    rng = np.random.default_rng(3 * log_n + skips)
    a, b = (rng.integers(0, P, 1 << log_n, dtype=np.uint64) for _ in range(2))
    cols = [x.astype(np.uint32) for x in (a, b, a * b % P)]
    consts, _ = oracle.workload(2)
    ref = oracle.prove_abc(consts[148:296], log_n, skips, *cols)
    got, _ = wl.sumcheck_abc_prove(ctx, consts[148:296], log_n, skips, *cols)
    assert np.array_equal(got, ref)


# inner sumcheck of 2^(log_n - 1) points at first; WHIR blocks of 7 and 4 rounds on tables of
# 2^(log_n + 1), 2^(log_n - 6), ...: the block of 7 rounds starts at 2^log_n points
@pytest.mark.parametrize("log_n", [10, 11, 12, 13])
def test_pair_cluster_tails_match_oracle(oracle, wl, ctx, log_n):
    consts, inputs = oracle.workload(log_n, 47)
    wit = oracle.trace(log_n, consts, inputs)
    ref, _ = oracle.prove(log_n, consts, wit)
    assert np.array_equal(wl.AirTable(ctx, consts, log_n).prove(wit), ref)
