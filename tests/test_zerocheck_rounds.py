"""The zerocheck's round 0 over tables whose input groups are split over blocks, its later rounds on
the carried cube inputs, and the partial evaluation of short tables: proofs at the edges of the
splits against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 2^log_n / 2^skips points of round 0: 2 and 8 (a partial tile), 32 (one tile, one group a block),
# 128, 512 and 1024 (uneven splits), 2048 and 4096 (two to four groups of columns)
@pytest.mark.parametrize("log_n,skips", [(4, 3), (7, 4), (9, 4), (9, 2), (10, 3), (13, 4), (13, 3), (14, 3)])
def test_round0_splits_match_oracle(oracle, wl, ctx, log_n, skips):
    settings = wl.AirSettings(univariate_skips=skips)
    consts, inputs = oracle.workload(log_n, 5 + skips)
    wit = oracle.trace(log_n, consts, inputs)
    ref, _ = oracle.prove(log_n, consts, wit, settings.as_array())
    got = wl.AirTable(ctx, consts, log_n, settings).prove(wit)
    assert np.array_equal(got, ref)
