"""BW_ECHECK.  On products with 64-bit coefficients no prime is redundant,
so the product's words are checked against the operands' modulo 2^32 - 1.  One
residue in the wrong place (data only: a valid residue copied from its
neighbour) is reported however little room the primes leave, in every form of
the carry and of the column passes, and the next product is right again."""
import numpy as np
import pytest

import birdwing_b200 as bw
from birdwing_b200 import _lib as L
from oracle import gmp_ref

pytestmark = pytest.mark.gpu

C64 = L.BW_PLAN_COEF64


def operands(la, lb, kind="random"):
    rng = np.random.default_rng(la + lb)
    a, b = (rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32) for n in (la, lb))
    if kind == "ones":  # carry chains through every tile of the low half
        a[:] = 0xFFFFFFFF
        b[:] = 0xFFFFFFFF
    return a, b


def device_product(c, a, b):
    import torch
    d = [torch.from_numpy(x.view(np.int32)).cuda() for x in (a, b)]
    out = torch.empty(a.size + b.size, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    c.multiply_device(d[0].data_ptr(), a.size, d[1].data_ptr(), b.size, out.data_ptr(),
                      out.numel())
    c.sync()
    return out.cpu().numpy().view(np.uint32)


def check_reports(c, call, want, spots):
    assert (call() == want).all()
    for at in spots:
        bw._lib.check(bw.lib.bw_ctx_inject_residue_fault(c._h, 1, at))
        with pytest.raises(bw.BwError) as e:
            call()
        assert e.value.code == L.BW_ECHECK, at
        bw._lib.check(bw.lib.bw_ctx_inject_residue_fault(c._h, 0, 0))
        assert (call() == want).all(), at


# words of each operand; 2^23 leave the first double-precision set 2% of room
@pytest.mark.parametrize("path,words,flags", [
    (64, 1 << 23, 0), (32, 1 << 20, C64), (64, 40001, C64), (32, 40001, C64), (64, 300, C64),
    (32, 300, C64), (64, 70001, C64 | L.BW_PLAN_TW_SMEM), (32, 70001, C64 | L.BW_PLAN_TW_SMEM),
    (64, 70001, C64 | L.BW_PLAN_THREE_PASS), (64, 70001, C64 | L.BW_PLAN_THREE_PASS | L.BW_PLAN_TW_SMEM)])
def test_one_wrong_residue_is_reported(path, words, flags):
    a, b = operands(words, words - 1)
    want = gmp_ref.mul(a, b)
    with bw.Plan(words, words - 1, path, flags=flags) as p, bw.Context(p) as c:
        assert p.info["coeff_bits"] == 64
        spots = (0, 5, words // 2, words - 2)
        check_reports(c, lambda: device_product(c, a, b), want, spots)
        for chunks in (1, 8):
            c.set_copy_chunks(chunks)
            check_reports(c, lambda: c.multiply(a, b), want, spots[:2])
        c.set_copy_chunks(1)
        c.multiply(a, b, timing=True)
    with bw.Plan(words, words, path, flags=flags) as p, bw.Context(p) as c:
        check_reports(c, lambda: c.square(a), gmp_ref.mul(a, a), spots[:2])


@pytest.mark.parametrize("path", [32, 64])
@pytest.mark.parametrize("la,lb", [(5, 5), (1024, 1024), (1025, 1023), (60000, 777), (1 << 18, 1 << 18)])
def test_carry_chains_pass_the_check(la, lb, path):
    # all-ones operands: the fix rewrites tiles, and its changes are counted
    # (residues in the wrong place are reported all the same)
    a, b = operands(la, lb, "ones")
    b[lb // 2] = 12345
    want = gmp_ref.mul(a, b)
    with bw.Plan(la, lb, path, flags=C64) as p, bw.Context(p) as c:
        # (where the coefficients still rise: neighbours differ)
        spots = (1, 101) if lb > 300 else (1,)
        for chunks in (1, 4):
            c.set_copy_chunks(chunks)
            check_reports(c, lambda: c.multiply(a, b), want, spots)
        check_reports(c, lambda: device_product(c, a, b), want, spots)


@pytest.mark.parametrize("K", [2, 3])
@pytest.mark.parametrize("words", [3000, 100000])
def test_groups_report_a_wrong_residue(words, K):
    # the 64-bit path's groups: with two primes by the coefficient's bound (a
    # wrong one passes with probability n 2^-37), with three by the third.
    # 64 products, one at a time: by the bound 2^96 alone some would pass.
    rng = np.random.default_rng(words)
    a, b = (np.zeros(words, dtype=np.uint32) for _ in range(2))
    with bw.Batch(num_primes=K) as bt:
        out = bt.add(a, b, path=64)
        for on in [1] * 64 + [0]:
            a[:] = rng.integers(0, 1 << 32, words, dtype=np.uint64)
            b[:] = rng.integers(0, 1 << 32, words, dtype=np.uint64)
            bw._lib.check(bw.lib.bw_batch_inject_residue_fault(bt._h, on))
            if on:
                with pytest.raises(bw.BwError) as e:
                    bt.run()
                assert e.value.code == L.BW_ECHECK
            else:
                bt.run()
                assert (out == gmp_ref.mul(a, b)).all()


def test_context_made_beside_a_busy_default_stream():
    # the carry state and the sums are clear before the first product, whatever
    # is queued on the default stream when the context is made
    import torch
    n = 1 << 16
    a, b = operands(n, n, "ones")
    want = torch.from_numpy(gmp_ref.mul(a, b).view(np.int32)).cuda()
    d = [torch.from_numpy(x.view(np.int32)).cuda() for x in (a, b)]
    out = torch.empty(2 * n, dtype=torch.int32, device="cuda")
    with bw.Plan(n, n, 64, flags=C64) as p:
        torch.cuda.synchronize()
        for _ in range(5):
            torch.cuda._sleep(4_000_000)  # about 2 ms
            with bw.Context(p) as c:
                for _ in range(200):
                    c.multiply_device(d[0].data_ptr(), n, d[1].data_ptr(), n, out.data_ptr(),
                                      2 * n)
                c.sync()
            torch.cuda.synchronize()
            assert torch.equal(out, want)
