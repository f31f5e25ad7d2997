"""Short products on the 64-bit path's integer primes: the automatic split is
exact at every length it covers and no slower than rows of four points, which
measured fastest there (a third less than a square split)."""
import time

import numpy as np
import pytest

import birdwing_b200 as bw
from oracle import gmp_ref, mt64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [2, 3])
@pytest.mark.parametrize("log_n", range(4, 12))
def test_exact(log_n, K):
    n = 1 << log_n
    for la, lb in ((n // 2, n // 2), (n // 2 + 1, n // 2), (n - 2, 3), (n // 2 - 1, 1)):
        for a, b in ((mt64.random_words_top_fast(la, la), mt64.random_words_top_fast(lb, lb)),
                     (np.full(la, 0xFFFFFFFF, np.uint32), np.full(lb, 0xFFFFFFFF, np.uint32))):
            with bw.Plan(la, lb, 64, K) as p, bw.Context(p) as c:
                assert (c.multiply(a, b) == gmp_ref.mul(a, b)).all(), (la, lb)
                if la == lb:
                    assert (c.square(a) == gmp_ref.mul(a, a)).all(), la


def product_us(words, log_cols):
    import torch
    x = torch.randint(-(1 << 31), 1 << 31, (2 * words,), dtype=torch.int32, device="cuda")
    out = torch.empty(2 * words, dtype=torch.int32, device="cuda")
    with bw.Plan(words, words, 64, 2, log_cols=log_cols) as p, bw.Context(p) as c:
        torch.cuda.synchronize()
        best = 1e9
        for _ in range(8):
            t = time.perf_counter()
            for _ in range(200):
                c.multiply_device(x.data_ptr(), words, x.data_ptr() + 4 * words, words,
                                  out.data_ptr(), 2 * words)
            c.sync()
            best = min(best, 1e6 * (time.perf_counter() - t) / 200)
    return best


@pytest.mark.parametrize("log_n", [7, 8, 9])
def test_default_split_is_not_slow(log_n):
    words = 1 << (log_n - 1)
    seen = []
    for _ in range(3):  # (single products step by 2 us)
        seen.append((product_us(words, 0), product_us(words, 2)))
        if seen[-1][0] < 1.1 * seen[-1][1]:
            return
    assert False, seen
