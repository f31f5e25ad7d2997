"""Long carry chains: all-ones operands make every tile of the product's low
half pass a carry on.  Broken at chosen words, exact against GMP; and a product
of such operands costs no more than twice one of random words -- the carry fix
rewrites each word at most once, less than the product's own traffic."""
import numpy as np
import pytest

import birdwing_b200 as bw
from birdwing_b200 import _lib as L
from oracle import gmp_ref

pytestmark = pytest.mark.gpu

TILE = 2048


def ones(n):
    return np.full(n, 0xFFFFFFFF, dtype=np.uint32)


@pytest.mark.parametrize("path,K,flags", [(32, 2, 0), (64, 2, 0), (64, 3, L.BW_PLAN_COEF64)])
@pytest.mark.parametrize("words", [TILE // 2 + 1, 40 * TILE + 5, 400 * TILE])
def test_broken_chains_exact(words, path, K, flags):
    # one tile and two, one CTA of the fix, several; the chain broken in the
    # first tile, at a tile's edge, inside the run of another CTA
    breaks = sorted({0, 1, words // 2, words - 1, min(words - 1, TILE),
                     min(words - 1, 64 * TILE - 1), min(words - 1, 130 * TILE + 17)})
    with bw.Plan(words, words, path, K, flags=flags) as p, bw.Context(p) as c:
        for at in breaks:
            a = ones(words)
            a[at] = 0x7FFFFFFF
            assert (c.multiply(a, ones(words)) == gmp_ref.mul(a, ones(words))).all(), at
        # a power of two minus one, times a number with one high word
        b = np.zeros(words, dtype=np.uint32)
        b[0], b[-1] = 1, 0x80000000
        assert (c.multiply(ones(words), b) == gmp_ref.mul(ones(words), b)).all()


@pytest.mark.parametrize("path", [32, 64])
def test_broken_chains_in_groups_exact(path):
    words = 100 * TILE
    ops = []
    for i in range(8):  # 1600 tiles: the words pass and the fix
        a, b = ones(words - i), ones(words)
        if i:
            a[(i * 37 * TILE + i) % words - 8] = 5
        ops.append((a, b))
    with bw.Batch() as bt:
        outs = [bt.add(a, b, path=path) for a, b in ops]
        for _ in range(2):
            for o in outs:
                o[:] = 0
            bt.run()
            for (a, b), o in zip(ops, outs):
                assert (o == gmp_ref.mul(a, b)).all(), a.size


def product_ms(a, b, path):
    import torch
    n = a.size
    d = [torch.from_numpy(x.view(np.int32)).cuda() for x in (a, b)]
    out = torch.empty(2 * n, dtype=torch.int32, device="cuda")
    with bw.Plan(n, n, path) as p, bw.Context(p) as c:
        torch.cuda.synchronize()
        s = torch.cuda.ExternalStream(c.stream)
        best = 1e9
        for _ in range(8):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record(s)
            for _ in range(4):
                c.multiply_device(d[0].data_ptr(), n, d[1].data_ptr(), n, out.data_ptr(), 2 * n)
            e1.record(s)
            c.sync()
            best = min(best, e0.elapsed_time(e1) / 4)
    return best


def group_ms(ops, path):
    with bw.Batch() as bt:
        for a, b in ops:
            bt.add(a, b, path=path)
        bt.run()
        return min(bt.run(2, timing=True)["total_ms"] for _ in range(8))


@pytest.mark.parametrize("path", [32, 64])
def test_long_chains_are_not_slow(path):
    rng = np.random.default_rng(3)
    n = 1 << 20
    rnd = [rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32) for _ in range(2)]
    assert product_ms(ones(n), ones(n), path) < 2 * product_ms(*rnd, path)
    m = 1 << 22
    rnd = [rng.integers(0, 1 << 32, m, dtype=np.uint64).astype(np.uint32) for _ in range(2)]
    assert group_ms([(ones(m), ones(m))], path) < 2 * group_ms([rnd], path)
