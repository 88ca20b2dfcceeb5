"""Eq tables around the size from which a block writes 2^12 entries: the a*b - c sumcheck's tables of
2^(log_n - skips) entries and half of that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0x7F000001


@pytest.mark.parametrize("log_n,skips", [(20, 3), (20, 2), (20, 1), (21, 1)])
def test_abc_eq_tables_match_oracle(oracle, wl, ctx, log_n, skips):
    rng = np.random.default_rng(5 * log_n + skips)
    a, b = (rng.integers(0, P, 1 << log_n, dtype=np.uint64) for _ in range(2))
    cols = [x.astype(np.uint32) for x in (a, b, a * b % P)]
    consts, _ = oracle.workload(2)
    ref = oracle.prove_abc(consts[148:296], log_n, skips, *cols)
    got, _ = wl.sumcheck_abc_prove(ctx, consts[148:296], log_n, skips, *cols)
    assert np.array_equal(got, ref)
