"""Each arithmetic of 64-bit coefficients on the 64-bit path at small sizes.
Left to itself a plan takes 58-bit integer primes only above 2^28 words a side
and the second double-precision set above 2^23; here they are asked for, in two
and three passes, with fixed and any-length columns, against GMP, and the rule
that picks them is looked at where it changes."""
import ctypes

import numpy as np
import pytest

import birdwing_b200 as bw
from birdwing_b200 import _lib as L
from oracle import gmp_ref, mt64

pytestmark = pytest.mark.gpu

C64 = L.BW_PLAN_COEF64
INT, SECOND = 0, 2


class ArithPlan(bw.Plan):
    def __init__(self, la, lb, arith, flags=0):
        fn = bw.lib.bw_plan_create_arith
        fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t, ctypes.c_size_t,
                       ctypes.c_int, ctypes.c_uint, ctypes.c_int]
        h = ctypes.c_void_p()
        self._h = None
        bw._lib.check(fn(ctypes.byref(h), 64, la, lb, 0, C64 | flags, arith))
        self._h = h
        info = L.bw_plan_info()
        bw._lib.check(bw.lib.bw_plan_get_info(h, ctypes.byref(info)))
        self.info = {"log_n": info.log_n, "log_cols": info.log_cols,
                     "bits": int(info.primes[0]).bit_length()}


def operands(la, lb):
    """Random words, and the largest coefficients in every place."""
    yield (mt64.random_words_top_fast(la, la + 1), mt64.random_words_top_fast(lb, lb + 2))
    yield (np.full(la, 0xFFFFFFFF, dtype=np.uint32), np.full(lb, 0xFFFFFFFF, dtype=np.uint32))


@pytest.mark.parametrize("arith,bits", [(INT, 58), (SECOND, 52)])
@pytest.mark.parametrize("flags", [0, L.BW_PLAN_THREE_PASS, L.BW_PLAN_TW_SMEM,
                                   L.BW_PLAN_THREE_PASS | L.BW_PLAN_TW_SMEM])
@pytest.mark.parametrize("la,lb", [(1, 1), (5, 7), (32, 32), (511, 514), (4096, 4095),
                                   (30001, 1200), (70001, 65536), (1 << 18, 1 << 18),
                                   ((1 << 19) + 1, 1 << 19)])
def test_forced_arithmetic_exact(la, lb, flags, arith, bits):
    with ArithPlan(la, lb, arith, flags) as p, bw.Context(p) as c:
        assert p.info["bits"] == bits
        for a, b in operands(la, lb):
            assert (c.multiply(a, b) == gmp_ref.mul(a, b)).all()
            if la == lb:
                assert (c.square(a) == gmp_ref.mul(a, a)).all()
        for chunks in (1, 4):
            c.set_copy_chunks(chunks)
            assert (c.multiply(a, b) == gmp_ref.mul(a, b)).all()


@pytest.mark.parametrize("arith", [INT, SECOND])
@pytest.mark.parametrize("log_c", range(5, 14))
def test_forced_arithmetic_splits_exact(log_c, arith):
    words = 1 << 16  # n = 2^16
    a, b = next(operands(words, words))
    want = gmp_ref.mul(a, b)
    with ArithPlan(words, words, arith, log_c << 8) as p, bw.Context(p) as c:
        assert (p.info["log_n"], p.info["log_cols"]) == (16, log_c)
        assert (c.multiply(a, b) == want).all()


def test_where_the_rule_changes():
    for words, bits in ((1 << 23, 51), ((1 << 23) + 1, 52), (1 << 28, 52), ((1 << 28) + 1, 58)):
        with bw.Plan(words, words, 64) as p:
            assert [q.bit_length() for q in p.info["primes"]] == [bits] * 3, words
    for arith in (1, 3):  # a set that does not hold the product is refused
        with pytest.raises(bw.BwError):
            ArithPlan((1 << 23) + 1, (1 << 23) + 1, arith)


@pytest.mark.parametrize("words,log_c", [(1 << 24, 13), ((1 << 24) + 9, 0), ((1 << 24) + 9, 13),
                                         (1 << 26, 0), (1 << 26, 13)])
def test_second_set_long_products(words, log_c):
    # transforms of 2^24 to 2^26 points, three passes and (log_c) two; checked
    # modulo three random odd 61-bit numbers
    a, b = next(operands(words, words - 3))
    with bw.Plan(words, words - 3, 64, log_cols=log_c) as p, bw.Context(p) as c:
        assert p.info["primes"][0].bit_length() == 52
        r = p.info["log_n"] - p.info["log_cols"]
        assert (p.info["log_rows"] == r) == (log_c != 0)
        out = c.multiply(a, b)
    A, B, C = (int.from_bytes(x.tobytes(), "little") for x in (a, b, out))
    rng = np.random.default_rng(words)
    for m in (int(rng.integers(1 << 60, 1 << 61)) | 1 for _ in range(3)):
        assert C % m == (A % m) * (B % m) % m, (words, log_c)
