"""Default transform shapes and the one-launch short transforms.

Sizes around every change of shape (one launch up to 2^12 points; 4-, 32- and
64-point columns; the row lengths of 2^19 to 2^21 points), as whole products,
squarings, windows, polynomials mod n (cyclic lengths shorter than an operand
included) and integer polynomials, alone and in a planned batch.  Exact, so
there is no tolerance.
"""
import numpy as np
import pytest

import flint_b200 as FB
import oracle as O

pytestmark = pytest.mark.gpu


def _dev(torch, a):
    return torch.from_numpy(a.view(np.int64)).cuda()


SIZES = [(1 << k, 1) for k in (9, 12, 13, 14, 18)] + [(1 << k, 2) for k in (9, 10, 11, 12, 13, 14, 15, 17, 18, 19, 20)] + \
        [(255, 258), (4000, 97), (7000, 1190), (16000, 300), (300000, 200000), (600000, 400000)]


@pytest.mark.parametrize("an,bn", SIZES)
def test_products_and_squares(ctx, an, bn):
    torch = pytest.importorskip("torch")
    a, b = O.rand_limbs(an, an), O.rand_limbs(bn + 7, bn)
    da, db = _dev(torch, a), _dev(torch, b)
    s = torch.cuda.current_stream().cuda_stream
    z = torch.full((an + bn,), -1, dtype=torch.int64, device="cuda")
    w = torch.full((2 * bn,), -1, dtype=torch.int64, device="cuda")
    ctx.mpn_mul_device(z.data_ptr(), da.data_ptr(), an, db.data_ptr(), bn, s)
    ctx.mpn_mul_device(w.data_ptr(), db.data_ptr(), bn, db.data_ptr(), bn, s)
    torch.cuda.synchronize()
    assert (z.cpu().numpy().view(np.uint64) == O.gmp_mpn_mul(a, b)).all()
    assert (w.cpu().numpy().view(np.uint64) == O.gmp_mpn_mul(b, b)).all()


@pytest.mark.parametrize("n", [(1 << 61) + 15, 65537])
@pytest.mark.parametrize("an,bn,zl,zh", [(700, 300, 0, 999), (700, 300, 299, 700), (3000, 1500, 1499, 3000),
                                         (4096, 4096, 2000, 6000), (9000, 5000, 4999, 9000)])
def test_nmod_windows(ctx, an, bn, zl, zh, n):
    a, b = O.rand_below(an, an, n), O.rand_below(bn, bn, n)
    assert (ctx.nmod_poly_mul_mid(zl, zh, a, b, n) == O.port_nmod_mul_mid(zl, zh, a, b, n)).all()


@pytest.mark.parametrize("an,bn", [(2000, 300), (1100, 1050)])
def test_nmod_division_folds(ctx, an, bn):
    """The remainder is a cyclic product whose operands wrap around."""
    n = (1 << 50) + 55
    a, b = O.rand_below(1, an, n), O.rand_below(2, bn, n)
    b[-1] = 1
    q, r = ctx.nmod_poly_divrem(a, b, n)
    wq, wr = O.nmod_divrem_python([int(v) for v in a], [int(v) for v in b], n)
    assert [int(v) for v in q] == wq and [int(v) for v in r] == wr


@pytest.mark.parametrize("an,bn,bits", [(100, 60, 60), (300, 200, 200), (128, 128, 1000)])
def test_integer_polynomials(ctx, an, bn, bits):
    a, b = O.rand_fmpz_raw(an, an, bits), O.rand_fmpz_raw(bn + 1, bn, bits)
    z = ctx.fmpz_poly_mul_mid(0, an + bn - 1, a, b)
    assert O.raw_to_ints(z) == O.fmpz_poly_mul_python(O.raw_to_ints(a), O.raw_to_ints(b))


def test_batch_of_short_products(ctx):
    """Enough products of one short length that its threads own sixteen words."""
    torch = pytest.importorskip("torch")
    sizes = [(300 + 3 * k, 150 + k) for k in range(40)] + [(2500, 1400)] * 40 + [(9000, 7000)] * 3 + [(70000, 40000)] * 2
    A = [O.rand_limbs(10 + k, s[0]) for k, s in enumerate(sizes)]
    B = [O.rand_limbs(900 + k, s[1]) for k, s in enumerate(sizes)]
    dA, dB = [_dev(torch, x) for x in A], [_dev(torch, x) for x in B]
    Z = [torch.full((sum(s),), -1, dtype=torch.int64, device="cuda") for s in sizes]
    reqs = [(z.data_ptr(), a.data_ptr(), s[0], b.data_ptr(), s[1]) for z, a, b, s in zip(Z, dA, dB, sizes)]
    st = torch.cuda.current_stream().cuda_stream
    with FB.MpnBatch(ctx, reqs) as batch:
        batch.run(st)
        batch.check(st)
    for a, b, z in zip(A, B, Z):
        assert (z.cpu().numpy().view(np.uint64) == O.gmp_mpn_mul(a, b)).all()
