"""Columns of 2^9 to 2^11 points over 2^13-point rows, where single products reach them.

Squarings on 2^22 to 2^24 points (the inverse columns that carry the scale), a
product of two operands on 2^24 (the forward columns that start from the limbs),
and windows whose cyclic length is shorter than an operand, which wraps around
there and takes the column kernels' general load.  Compared with GMP on every
limb, so there is no tolerance.
"""
import numpy as np
import pytest

import flint_b200 as FB
import oracle as O

pytestmark = pytest.mark.gpu


def _product(ctx, a, b):
    torch = pytest.importorskip("torch")
    da = torch.from_numpy(a.view(np.int64)).cuda()
    db = da if b is a else torch.from_numpy(b.view(np.int64)).cuda()
    z = torch.full((len(a) + len(b),), -1, dtype=torch.int64, device="cuda")
    ctx.mpn_mul_device(z.data_ptr(), da.data_ptr(), len(a), db.data_ptr(), len(b))
    torch.cuda.synchronize()
    return z.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("n,logM", [(1900003, 22), (3800001, 23), (7500000, 24)])
def test_squarings(ctx, n, logM):
    assert FB.mpn_mul_transform_points(n, n, square=True) == 1 << logM
    a = O.rand_limbs(logM, n)
    assert (_product(ctx, a, a) == O.gmp_mpn_mul(a, a)).all()


def test_two_operands(ctx):
    an, bn = 7500000, 7400001
    assert FB.mpn_mul_transform_points(an, bn) == 1 << 24 and not FB.mpn_mul_split_plan(an, bn)
    a, b = O.rand_limbs(1, an), O.rand_limbs(2, bn)
    assert (_product(ctx, a, b) == O.gmp_mpn_mul(a, b)).all()


@pytest.mark.parametrize("logM", [22, 23, 24])
def test_windows_shorter_than_an_operand(ctx, logM):
    M = 1 << logM
    an, bn = M + 5001, 2003
    lo, hi = 10000, M - 9                      # needs M points: L + 3 - lo and hi below M
    a, b = O.rand_limbs(logM, an), O.rand_limbs(logM + 50, bn)
    want = O.gmp_mpn_mul(a, b)
    assert 2 < int(want[lo - 1]) < (1 << 64) - 4   # no carry into the window is in doubt
    assert (ctx.mpn_mul_range(lo, hi, a, b) == want[lo:hi]).all()
    assert (ctx.mpn_mul_range(lo, hi, b, a) == want[lo:hi]).all()
