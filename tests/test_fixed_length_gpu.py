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
SPLITS = ([(7, c) for c in range(4, 14)] + [(r, 6) for r in range(2, 14)] +
          [(r, 12) for r in (5, 6, 8, 9, 10)] + [(5, 13), (6, 13), (3, 9), (12, 9), (3, 7), (4, 7), (3, 12)])
# path, primes, plan flags, coefficients per pair of words
FORMS = [(32, 2, 0, 4), (32, 3, 0, 4), (32, 6, L.BW_PLAN_COEF64, 1), (64, 2, 0, 2), (64, 3, 0, 2),
         (64, 3, L.BW_PLAN_COEF64, 1)]


@pytest.mark.parametrize("log_r,log_c", SPLITS)
@pytest.mark.parametrize("path,K,flags,per", FORMS)
def test_split_exact(log_r, log_c, path, K, flags, per):
    n = 1 << (log_r + log_c)
    # words of a product that fills the transform
    total = 2 * n // per
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


@pytest.mark.parametrize("K", [2, 3])
@pytest.mark.parametrize("log_n", range(4, 14))
def test_one_cta_products_exact(log_n, K):
    # products of up to 2^11 points run in one CTA, 2^12 and more do not; every
    # length filled exactly (the final carry lands past the last coefficient),
    # one word short, and squared; alone, with stage times and in a batch
    import torch
    total = 1 << (log_n - 1)
    cases = {(max(1, total // 2), max(1, total // 2)), (max(1, total - 2), 2), (total, 1),
             (max(1, total // 2 + 1), max(1, total // 2 - 2))}
    items = []
    for la, lb in sorted(cases):
        a = mt64.random_words_top_fast(la, 3 * la + log_n)
        b = mt64.random_words_top_fast(lb, 5 * lb + log_n)
        for x, y in ((a, b), (np.full(la, 0xFFFFFFFF, np.uint32), np.full(lb, 0xFFFFFFFF, np.uint32))):
            items.append((x, y))
            want = gmp_ref.mul(x, y)
            with bw.Plan(la, lb, L.BW_PATH_P32, K) as p, bw.Context(p) as c:
                assert (c.multiply(x, y) == want).all(), (la, lb)
                assert (c.multiply(x, y, timing=True)[0] == want).all(), (la, lb)
                da = torch.from_numpy(x.view(np.int32)).cuda()
                db = torch.from_numpy(y.view(np.int32)).cuda()
                dc = torch.full((la + lb + 1,), -1, dtype=torch.int32, device="cuda")
                torch.cuda.synchronize()
                c.multiply_device(da.data_ptr(), la, db.data_ptr(), lb, dc.data_ptr() + 4, la + lb)
                c.sync()
                got = dc.cpu().numpy().view(np.uint32)
                assert got[0] == 0xFFFFFFFF and (got[1:] == want).all(), (la, lb)
                if la == lb:
                    assert (c.square(x) == gmp_ref.mul(x, x)).all()
    with bw.Batch(num_primes=K) as bt:
        outs = [(x, y, bt.add(x, y, path=path)) for x, y in items for path in (32, 64)]
        outs += [(x, x, bt.add(x, x, path=path)) for x, _ in items for path in (32, 64)]
        bt.run()
        for x, y, got in outs:
            assert (got == gmp_ref.mul(x, y)).all(), (x.size, y.size)


@pytest.mark.parametrize("path", [32, 64])
@pytest.mark.parametrize("log_n", range(10, 18))
def test_group_splits_exact(log_n, path):
    # batched 4-step products over the splits the group passes are
    # instantiated for, with ragged sizes and squarings in one bucket
    per = 2 if path == 32 else 1
    total = (1 << log_n) // per
    rng = np.random.default_rng(log_n)
    shapes = [(total // 2, total // 2), (total // 2 + 7, total // 2 - 9), (total - 3, 3)]
    ops = [tuple(rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32) for n in s)
           for s in shapes]
    ops.append((np.full(total // 2, 0xFFFFFFFF, np.uint32),) * 2)
    want = [gmp_ref.mul(a, b) for a, b in ops]
    for log_c in sorted({5, 7, 10, 13, log_n - 3, log_n - 4}):
        if not 3 <= log_n - log_c <= 13 or log_c < 5 or log_c > 13:
            continue
        bw.set_tune_entry(path, 2, log_n, 0, log_c)
        try:
            with bw.Batch() as bt:
                outs = [bt.add(a, b, path=path) for a, b in ops]
                bt.run()
        finally:
            bw.set_tune_entry(path, 2, log_n, log_n <= 12, 0)
        for w, got in zip(want, outs):
            assert (w == got).all(), (log_n, log_c)


@pytest.mark.parametrize("log_r2", range(2, 12))
@pytest.mark.parametrize("path,K,flags", [(32, 2, 0), (64, 3, L.BW_PLAN_COEF64)])
def test_middle_lengths_exact(log_r2, path, K, flags):
    # three passes at every middle length (below 2^5: the any-length pass), by
    # way of the row length: n = R * R2 * C with R = R2 or 2 R2
    for extra in (0, 1):
        log_c = max(5, 12 - log_r2)
        log_n = 2 * log_r2 + extra + log_c
        if log_n > 25:
            continue
        total = (1 << log_n) // 2 if path == 32 else 2 << log_n
        if total > 1 << 23:
            continue
        la, lb = total // 2 + 5, total // 2 - 9
        a = mt64.random_words_top_fast(la, la)
        b = mt64.random_words_top_fast(lb, lb)
        a[: la // 2] = 0xFFFFFFFF
        with bw.Plan(la, lb, path, K, log_cols=log_c, flags=flags | L.BW_PLAN_THREE_PASS) as p, \
                bw.Context(p) as c:
            assert p.info["log_n"] - p.info["log_rows"] - p.info["log_cols"] == log_r2
            assert (c.multiply(a, b) == gmp_ref.mul(a, b)).all(), (la, lb)
        with bw.Plan(la, la, path, K, flags=flags | L.BW_PLAN_THREE_PASS) as p, bw.Context(p) as c:
            assert (c.square(a) == gmp_ref.mul(a, a)).all(), la


@pytest.mark.parametrize("path,K,flags", [f[:3] for f in FORMS])
def test_any_length_passes_exact(path, K, flags):
    # the passes for any length, which BW_PLAN_TW_SMEM selects for the columns
    # (two and three passes), beside the fixed-length rows
    rng = np.random.default_rng(97)
    for la, lb in ((3001, 2500), (70001, 65536)):
        a, b = (rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32) for n in (la, lb))
        want = gmp_ref.mul(a, b)
        for fl in (L.BW_PLAN_TW_SMEM, L.BW_PLAN_TW_SMEM | L.BW_PLAN_THREE_PASS,
                   L.BW_PLAN_TW_SMEM | L.BW_PLAN_WIDE_COLS):
            with bw.Plan(la, lb, path, K, flags=flags | fl) as p, bw.Context(p) as c:
                assert (c.multiply(a, b) == want).all(), (la, lb, hex(fl))
