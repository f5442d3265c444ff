"""The row pass whose five lowest levels are byte-matrix products.

Items of 2^13 words take it, for rows of 2^9 to 2^13 points: every row length
with five and six primes, products and squarings, values that drive the byte
sums to their extremes (all-ones limbs, zeros), the chunks of a split product
(b's spectrum given) and ring products whose last item is ragged.  Integers
are compared exactly, so there is no tolerance.
"""
import numpy as np
import pytest

import flint_b200 as FB
import oracle as O

pytestmark = pytest.mark.gpu


def _dev(torch, a):
    return torch.from_numpy(a.view(np.int64)).cuda()


def _mul(torch, ctx, a, b, cfg):
    da = _dev(torch, a)
    db = da if b is a else _dev(torch, b)
    z = torch.full((len(a) + len(b),), -1, dtype=torch.int64, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    if cfg is None:
        ctx.mpn_mul_device(z.data_ptr(), da.data_ptr(), len(a), db.data_ptr(), len(b), s)
    else:
        ctx.mpn_mul_device_config(z.data_ptr(), da.data_ptr(), len(a), db.data_ptr(), len(b), cfg, s)
    torch.cuda.synchronize()
    return z.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("np_", [5, 6])
@pytest.mark.parametrize("logC", [9, 10, 11, 12, 13])
def test_row_lengths(ctx, logC, np_):
    torch = pytest.importorskip("torch")
    an, bn = 300001, 200003                       # 2^19 points
    cfg = FB.MulConfig(FB.ROUTE_NTT, np_, 0, logC, 0)
    a, b = O.rand_limbs(logC, an), O.rand_limbs(logC + 100, bn)
    assert (_mul(torch, ctx, a, b, cfg) == O.gmp_mpn_mul(a, b)).all()
    assert (_mul(torch, ctx, b, b, cfg) == O.gmp_mpn_mul(b, b)).all()


@pytest.mark.parametrize("kind", ["ones", "sparse", "one_limb"])
def test_extreme_values(ctx, kind):
    torch = pytest.importorskip("torch")
    a = O.rand_limbs(5, 300001)
    b = np.full(200003, (1 << 64) - 1, dtype=np.uint64)
    if kind == "ones":
        a[:] = (1 << 64) - 1
    elif kind == "sparse":
        a[1:-1] = 0
        b[5:-3] = 0
    else:
        a[:] = 0
        a[-1] = 1
    assert (_mul(torch, ctx, a, b, None) == O.gmp_mpn_mul(a, b)).all()


def test_split_chunks(ctx):
    torch = pytest.importorskip("torch")
    an, bn = 5000000, 300000
    assert FB.mpn_mul_split_plan(an, bn)
    a, b = O.rand_limbs(1, an), O.rand_limbs(2, bn)
    assert (_mul(torch, ctx, a, b, None) == O.gmp_mpn_mul(a, b)).all()


@pytest.mark.parametrize("m", [512, 1024, 4096])
def test_ragged_ring_batches(ctx, m):
    torch = pytest.importorskip("torch")
    N = 40 * m
    n = N // 64
    count = (1 << 13) // m + 1                    # the second item holds one row
    R = FB.Mulmod2expp1(ctx, N, m)
    x = np.concatenate([O.neg_operand(10 + i, n) for i in range(count)])
    y = np.concatenate([O.neg_operand(90 + i, n) for i in range(count)])
    z = torch.full((count * (n + 1),), -1, dtype=torch.int64, device="cuda")
    dx, dy = _dev(torch, x), _dev(torch, y)
    R.batch_device(z.data_ptr(), dx.data_ptr(), dy.data_ptr(), count, None, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    z = z.cpu().numpy().view(np.uint64).reshape(count, n + 1)
    for i in range(count):
        s = slice(i * (n + 1), (i + 1) * (n + 1))
        assert (z[i] == O.negmul_python(x[s], y[s], N)).all()
