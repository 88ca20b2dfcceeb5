"""The last rounds of a sumcheck phase in one launch (k_abc_tail, k_pair_tail): proofs at the sizes
where the launch takes over at once, after one or more separate rounds, or holds a single round."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0x7F000001


def _abc(log_n, seed):
    rng = np.random.default_rng(seed)
    a, b = (rng.integers(0, P, 1 << log_n, dtype=np.uint64) for _ in range(2))
    return [x.astype(np.uint32) for x in (a, b, a * b % P)]


# points of round 1: 1, 2, 32, 128, 256 (one launch from the start), 512, 1024, 2048
@pytest.mark.parametrize("log_n,skips", [(2, 1), (3, 1), (10, 4), (10, 2), (11, 2), (11, 1), (12, 1), (13, 1)])
def test_abc_tail_matches_oracle(oracle, wl, ctx, log_n, skips):
    import torch
    cols = _abc(log_n, 7 * log_n + skips)
    consts, _ = oracle.workload(2)
    p16 = consts[148:296]
    ref = oracle.prove_abc(p16, log_n, skips, *cols)
    got, ms = wl.sumcheck_abc_prove(ctx, p16, log_n, skips, *cols)
    assert np.array_equal(got, ref)
    assert len(ms) == log_n - skips + 1
    dev = [torch.from_numpy(c.view(np.int32)).cuda() for c in cols]
    assert np.array_equal(wl.sumcheck_abc_prove_noalloc(p16, log_n, skips, *dev), ref)


# inner sumcheck rounds of 2^(log_n - 1) points at first: 16, 256 (one launch) and 512 (one round before it)
@pytest.mark.parametrize("log_n", [5, 9, 10])
def test_inner_tail_matches_oracle(oracle, wl, ctx, log_n):
    consts, inputs = oracle.workload(log_n, 31)
    wit = oracle.trace(log_n, consts, inputs)
    ref, _ = oracle.prove(log_n, consts, wit)
    assert np.array_equal(wl.AirTable(ctx, consts, log_n).prove(wit), ref)


@pytest.mark.parametrize("log_n,skips", [(5, 1), (12, 2), (14, 3), (13, 4)])
def test_abc_takes_any_word_for_its_residue(oracle, wl, ctx, log_n, skips):
    """The device columns are read as they are: words x and x + p are the same value, and the
    caller's columns are left as they were."""
    import torch
    cols = _abc(log_n, 90 + skips)
    consts, _ = oracle.workload(2)
    p16 = consts[148:296]
    ref = oracle.prove_abc(p16, log_n, skips, *cols)
    for every in (1, 3):
        shifted = [c.copy() for c in cols]
        for c in shifted:
            c[::every] += np.uint32(P)
        dev = [torch.from_numpy(c.view(np.int32)).cuda() for c in shifted]
        torch.cuda.synchronize()
        got, _ = wl.sumcheck_abc_prove(ctx, p16, log_n, skips, *dev, device=True)
        assert np.array_equal(got, ref)
        for d, c in zip(dev, shifted):
            assert np.array_equal(d.cpu().numpy().view(np.uint32), c)
