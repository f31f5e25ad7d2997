"""Plans are made on the caller's time whenever a size is new.  One of a product
that runs in one CTA, with its own tables beside the 4-step ones, costs little
more than one of the next length, which has only those."""
import time

import numpy as np
import pytest

import birdwing_b200 as bw

pytestmark = pytest.mark.gpu


def plan_us(words, K):
    us = []
    for _ in range(40):
        t = time.perf_counter()
        p = bw.Plan(words, words, 32, K)
        us.append(1e6 * (time.perf_counter() - t))
        p.close()
    return float(np.min(us))


@pytest.mark.parametrize("K,limit", [(2, 1.15), (3, 1.25)])
def test_one_cta_plan_is_not_slow(K, limit):
    plan_us(500, K)
    # 2^11 points, 2^12 points
    assert plan_us(500, K) < limit * plan_us(1000, K)
