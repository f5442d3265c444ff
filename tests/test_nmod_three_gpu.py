"""Windows of polynomial products mod n on 3 2^k-point cyclic transforms.

A window that such a length keeps free of aliasing takes it: every prime count,
whole products and middle windows whose aliases end just outside, squarings,
the boundary to the power of two on both sides, and an operand longer than the
transform (which stays on the power of two).  Compared with the restated
reference on every coefficient, so there is no tolerance.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

M = 3 << 18


@pytest.mark.parametrize("n", [3, 1000003, (1 << 31) - 1, (1 << 50) + 55, (1 << 61) + 15, (1 << 64) - 59])
def test_prime_counts(ctx, n):
    an, bn = 300001, 250000
    a, b = O.rand_below(an, an, n), O.rand_below(bn, bn, n)
    zn = an + bn - 1
    assert (ctx.nmod_poly_mul_mid(0, zn, a, b, n) == O.port_nmod_mul_mid(0, zn, a, b, n)).all()
    assert (ctx.nmod_poly_mul_mid(1, 2 * bn - 1, b, b, n) == O.port_nmod_mul_mid(1, 2 * bn - 1, b, b, n)).all()


@pytest.mark.parametrize("an,bn,zl,zh", [
    (M - 1000, 1001, 0, M),                        # product of exactly M coefficients
    (M // 2 + 200000, M // 2 + 100000, 299999, M),  # wraps: aliases end at coefficient zl - 1
    (M // 2 + 200000, M // 2 + 100000, 400000, 700000),
    (M // 2 + 1, M // 2 + 1, 0, M + 1),            # one coefficient too many: 2^20 points
    (M + 5000, 3000, 8000, M),                     # an operand longer than M
])
def test_windows(ctx, an, bn, zl, zh):
    n = (1 << 61) + 15
    a, b = O.rand_below(an, an, n), O.rand_below(bn + 1, bn, n)
    assert (ctx.nmod_poly_mul_mid(zl, zh, a, b, n) == O.port_nmod_mul_mid(zl, zh, a, b, n)).all()
