"""Plan switches whose forms are gone (include/birdwing.h names them) are
accepted and leave the plan as it is, tables and split included, at every kind
of plan; so is a tune entry's row radix."""
import numpy as np
import pytest

import birdwing_b200 as bw
from birdwing_b200 import _lib as L
from oracle import gmp_ref

pytestmark = pytest.mark.gpu

INERT = (L.BW_PLAN_RADIX8, L.BW_PLAN_RADIX16, L.BW_PLAN_COL_RADIX8, L.BW_PLAN_TMA_COLS,
         L.BW_PLAN_NO_TMA_COLS, L.BW_PLAN_SHFL_ROWS, L.BW_PLAN_K1_ONE_PRIME)


@pytest.mark.parametrize("words", [30, 900, 5000, 1 << 18])
@pytest.mark.parametrize("path,K,flags", [(32, 2, 0), (32, 3, 0), (64, 2, 0), (0, 0, 0),
                                          (64, 0, L.BW_PLAN_COEF64), (32, 0, L.BW_PLAN_COEF64),
                                          (64, 2, L.BW_PLAN_TW_SMEM),
                                          (32, 2, L.BW_PLAN_THREE_PASS)])
def test_plan_is_the_same(path, K, flags, words):
    rng = np.random.default_rng(words)
    a, b = (rng.integers(0, 1 << 32, words, dtype=np.uint64).astype(np.uint32) for _ in range(2))
    want = gmp_ref.mul(a, b)
    with bw.Plan(words, words, path, K, flags=flags) as p:
        info = p.info
    for extra in INERT + (sum(INERT),):
        with bw.Plan(words, words, path, K, flags=flags | extra) as p, bw.Context(p) as c:
            assert p.info == info, hex(extra)
            assert (c.multiply(a, b) == want).all(), hex(extra)


def test_row_radix_is_kept():
    for radix in (0, 8, 16):
        bw.set_tune_entry(64, 2, 30, False, 15, radix)
        e = [x for x in bw.tune_table() if (x["path"], x["log_n"]) == (64, 30)]
        assert e[0]["row_radix"] == radix and e[0]["log_cols"] == 15
    with pytest.raises(bw.BwError):
        bw.set_tune_entry(64, 2, 30, False, 15, 4)
