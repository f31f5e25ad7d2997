"""The transform passes with compile-time lengths: every row length and column
length they are instantiated for, at narrow and wide column tiles, on the
32-bit path (16- and 64-bit coefficients) and the 64-bit path's
double-precision arithmetic, exact against GMP; lengths outside the range run
the general passes and give the same products."""
import numpy as np
import pytest

import birdwing_b200 as bw
from birdwing_b200 import _lib as L
from oracle import gmp_ref, mt64

pytestmark = pytest.mark.gpu

# (log2 rows, log2 columns): each row length, each column length with few and
# with many columns, and lengths just outside the instantiated range
SPLITS = ([(7, c) for c in range(4, 14)] + [(r, 6) for r in range(4, 14)] +
          [(r, 12) for r in (5, 6, 8, 9, 10)] + [(5, 13), (6, 13), (3, 9), (12, 9)])
# path, primes, plan flags, coefficients per 64-bit pair of words
FORMS = [(32, 2, 0, 4), (32, 3, 0, 4), (32, 6, L.BW_PLAN_COEF64, 1),
         (64, 3, L.BW_PLAN_COEF64, 1)]


@pytest.mark.parametrize("log_r,log_c", SPLITS)
@pytest.mark.parametrize("path,K,flags,per", FORMS)
def test_split_exact(log_r, log_c, path, K, flags, per):
    n = 1 << (log_r + log_c)
    # words of a product that fills the transform
    total = n // 2 if per == 4 else 2 * n
    for la, lb in ((total // 2, total // 2), (total // 2 + 3, total // 2 - 7),
                   (total - 9, 5)):
        a = mt64.random_words_top_fast(la, 3 * la + log_r)
        b = mt64.random_words_top_fast(lb, 5 * lb + log_c)
        if lb == total // 2:
            a[: la // 2] = 0xFFFFFFFF
        with bw.Plan(la, lb, path, K, log_cols=log_c, flags=flags) as p, bw.Context(p) as c:
            assert (p.info["log_rows"], p.info["log_cols"]) == (log_r, log_c)
            assert (c.multiply(a, b) == gmp_ref.mul(a, b)).all(), (la, lb)
            if la == lb:
                assert (c.square(a) == gmp_ref.mul(a, a)).all(), la


@pytest.mark.parametrize("path,K,flags", [f[:3] for f in FORMS])
def test_operand_offsets_exact(path, K, flags):
    # operands at odd word offsets of a device buffer (8-byte loads of 64-bit
    # coefficients need an even one) and an output at an odd offset
    import torch
    la, lb = 30001, 26215
    a = mt64.random_words_top_fast(la, 9)
    b = mt64.random_words_top_fast(lb, 10)
    want = gmp_ref.mul(a, b)
    buf = torch.from_numpy(np.concatenate([[7], a, b]).astype(np.uint32).view(np.int32)).cuda()
    dc = torch.empty(la + lb + 1, dtype=torch.int32, device="cuda")
    with bw.Plan(la, lb, path, K, flags=flags) as p, bw.Context(p) as c:
        for _ in range(2):
            dc.fill_(-1)
            torch.cuda.synchronize()
            c.multiply_device(buf.data_ptr() + 4, la, buf.data_ptr() + 4 * (1 + la), lb,
                              dc.data_ptr() + 4, la + lb)
            c.sync()
            got = dc.cpu().numpy().view(np.uint32)
            assert got[0] == 0xFFFFFFFF and (got[1:] == want).all()


@pytest.mark.parametrize("path,K,flags", [f[:3] for f in FORMS])
def test_carry_fix_between_products(path, K, flags):
    # products whose tiles generate and propagate carries (all-ones operands,
    # all-ones times 2^(32 m) + 1) alternate with random ones on one context:
    # the fix pass runs, leaves no trace, and is skipped again
    import torch
    m = 30000
    rng = np.random.default_rng(77)
    ones = np.full(m, 0xFFFFFFFF, dtype=np.uint32)
    sparse = np.zeros(m, dtype=np.uint32)
    sparse[0] = sparse[m - 1] = 1
    rnd = [rng.integers(0, 1 << 32, m, dtype=np.uint64).astype(np.uint32) for _ in range(2)]
    da = torch.empty(m, dtype=torch.int32, device="cuda")
    db = torch.empty(m, dtype=torch.int32, device="cuda")
    dc = torch.empty(2 * m, dtype=torch.int32, device="cuda")
    with bw.Plan(m, m, path, K, flags=flags) as p, bw.Context(p) as c:
        for a, b in ((ones, sparse), (rnd[0], rnd[1]), (ones, ones.copy()), (rnd[1], rnd[0]),
                     (sparse, ones)):
            want = gmp_ref.mul(a, b)
            da.copy_(torch.from_numpy(a.view(np.int32)))
            db.copy_(torch.from_numpy(b.view(np.int32)))
            torch.cuda.synchronize()
            c.multiply_device(da.data_ptr(), m, db.data_ptr(), m, dc.data_ptr(), 2 * m)
            c.sync()
            assert (dc.cpu().numpy().view(np.uint32) == want).all()
            assert (c.multiply(a, b) == want).all()
