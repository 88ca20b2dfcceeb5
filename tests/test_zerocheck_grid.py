"""How the zerocheck's rounds >= 1 are split over blocks (k_zc_sbox): few x, one column per warp; more,
several columns per warp; many, all columns in one block. Host functions of the library, no GPU."""
import ctypes

import pytest

COLUMN_GROUPS = 37  # 148 cube inputs, four at a time
FILL = 2 * 2 * 148  # two waves of two blocks an SM


@pytest.mark.parametrize("m", range(1, 22))
def test_blocks_and_class_of_a_round(wl, m):
    lib = ctypes.CDLL(wl.LIB_PATH)
    blocks, several = lib._ZN2wl12zc_ef_blocksEi, lib._ZN2wl16zc_eval_is_denseEi
    blocks.restype, several.restype = ctypes.c_int, ctypes.c_bool
    x_blocks = max(1, (1 << (m - 1)) // 32)
    n = blocks(m)
    assert n % x_blocks == 0
    splits = n // x_blocks
    assert 1 <= splits <= COLUMN_GROUPS
    per = -(-COLUMN_GROUPS // splits)
    assert (splits - 1) * per < COLUMN_GROUPS  # no block without columns
    assert splits == 1 or (splits - 1) * x_blocks < FILL  # no more blocks than the two waves ask for
    assert several(m) == (per > 1)


def test_the_proofs_compared_with_the_oracle_take_every_split(wl):
    """2^8 rows at 4 skips only one column per warp, 2^16 rows several, 2^20 rows all in one block."""
    lib = ctypes.CDLL(wl.LIB_PATH)
    several = lib._ZN2wl16zc_eval_is_denseEi
    several.restype = ctypes.c_bool
    assert not several(8 - 4) and several(15 - 4) and several(16 - 4)
    assert lib._ZN2wl12zc_ef_blocksEi(20 - 4) == (1 << 15) // 32
