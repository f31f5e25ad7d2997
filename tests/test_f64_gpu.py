"""64-bit coefficients on the 64-bit path run in double-precision modular
arithmetic: two prime sets, chosen by the shorter operand's coefficients.
Products are exact against GMP at the edges of the choice, of the transform
lengths and of the coefficients' range (all words at their maximum)."""
from fractions import Fraction

import numpy as np
import pytest

import birdwing_b200 as bw
from birdwing_b200 import _lib as L
from oracle import gmp_ref, mt64

pytestmark = pytest.mark.gpu


def check(a, b, flags=0):
    with bw.Plan(a.size, b.size, L.BW_PATH_P64, 0, flags=L.BW_PLAN_COEF64 | flags) as p, \
            bw.Context(p) as c:
        assert p.info["coeff_bits"] == 64 and p.info["num_primes"] == 3
        assert (c.multiply(a, b) == gmp_ref.mul(a, b)).all(), (a.size, b.size, hex(flags))
        if a.size == b.size:
            assert (c.square(a) == gmp_ref.mul(a, a)).all(), (a.size, hex(flags))
        return p.info["primes"]


@pytest.mark.parametrize("log_n", range(4, 20))
def test_every_length_random_and_all_ones(log_n):
    # n = 2^log_n exactly filled (na + nb - 1 = n) and one word short of it
    n = 1 << log_n
    for wa, wb in ((n, n), (n + 1, n - 1), (2 * n - 2, 3)):
        ones = [np.full(w, 0xFFFFFFFF, dtype=np.uint32) for w in (wa, wb)]
        rnd = [mt64.random_words_top_fast(w, 7 * w + log_n) for w in (wa, wb)]
        check(*ones)
        check(*rnd)


def test_prime_sets_meet():
    # the shorter operand has 2^22 coefficients (first set), then 2^22 + 1
    # (second set, also in three passes); every coefficient at its maximum
    ones = np.full((1 << 23) + 1, 0xFFFFFFFF, dtype=np.uint32)
    first = check(ones[:-1], ones[:-1])
    second = check(ones, ones)
    assert first != second
    assert first[0] * first[1] * first[2] > 1 << 150
    assert second[0] * second[1] * second[2] > 1 << 155
    assert check(ones, ones, L.BW_PLAN_THREE_PASS) == second
    # the bounds on the quotients: 1 / p within 2^-58 of a double, 2 p < 2^53 / 1.2
    for ps in (first, second):
        for q in ps:
            assert abs(Fraction(1.0 / q) * q - 1) < Fraction(1, 1 << 58)
            assert (q - 1) % (1 << 32) == 0 and q.bit_length() in (51, 52)
    # unbalanced: a long transform with a short operand stays on the first set
    assert check(mt64.random_words_top_fast((1 << 24) + 3, 5), ones[:7]) == first
