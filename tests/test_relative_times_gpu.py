"""Calls that do less work, or the same work by a given shape, are no slower.

Each test compares two calls timed in turn on one device, the best of several
runs each, and passes if any of a few attempts is inside its bound; the bounds
lie midway between the ratio that the placement or shape it guards gives and the
ratio without it (both in the test's comment).
"""
import pytest

import flint_b200 as FB

pytestmark = pytest.mark.gpu

ATTEMPTS = 5


def _limbs(torch, *shape):
    return torch.randint(-(1 << 62), 1 << 62, shape, dtype=torch.int64, device="cuda")


def _best(torch, fn, stream, reps):
    best = float("inf")
    for _ in range(5):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        with torch.cuda.stream(stream):
            e0.record()
            for _ in range(reps):
                fn()
            e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return best


def _ratio_below(torch, f, g, bound, reps=30):
    """time(f) / time(g) < bound in at least one of a few attempts."""
    stream = torch.cuda.Stream()
    seen = []
    for _ in range(ATTEMPTS):
        ratio = _best(torch, lambda: f(stream.cuda_stream), stream, reps) / \
            _best(torch, lambda: g(stream.cuda_stream), stream, reps)
        seen.append(ratio)
        if ratio < bound:
            return
    raise AssertionError("ratios %s, bound %s" % (seen, bound))


def _ring(torch, ctx, N, count):
    C = FB.Mulmod2expp1(ctx, N)
    n = N // 64
    x, y, z = (_limbs(torch, count, n + 1) for _ in range(3))
    x[:, n] = 0
    y[:, n] = 0
    return C, x, y, z


@pytest.mark.parametrize("count", [50, 64])
def test_ring_products_by_kept_transforms(ctx, count):
    """A product by a kept transform does less than a whole one: 1.00-1.02
    (with finishing CTAs placed beside the inverse rows 1.40-1.48)."""
    torch = pytest.importorskip("torch")
    C, x, y, z = _ring(torch, ctx, 1 << 20, count)
    F = torch.empty(C.transformed_size(count), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    C.transform_device(F.data_ptr(), y.data_ptr(), count)
    torch.cuda.synchronize()
    _ratio_below(torch, lambda s: C.mul_cached_device(z.data_ptr(), x.data_ptr(), F.data_ptr(), count, None, s),
                 lambda s: C.batch_device(z.data_ptr(), x.data_ptr(), y.data_ptr(), count, None, s), 1.2)


@pytest.mark.parametrize("N,count,bound", [(12288, 500, 1.38), (196608, 64, 1.19)])
def test_ring_products_in_small_numbers(ctx, N, count, bound):
    """Twice as many products where the GPU is far from full: 1.24 and 1.06 of
    the time (with row CTAs placed beside the splitting ones 1.52 and 1.31)."""
    torch = pytest.importorskip("torch")
    C, x, y, z = _ring(torch, ctx, N, count)
    torch.cuda.synchronize()
    run = lambda c: lambda s: C.batch_device(z.data_ptr(), x.data_ptr(), y.data_ptr(), c, None, s)
    _ratio_below(torch, run(count), run(count // 2), bound)


def _batch(torch, ctx, n, count, configs=None):
    a, z = _limbs(torch, 2 * n * count), _limbs(torch, 2 * n * count)
    reqs = [(z.data_ptr() + 16 * n * i, a.data_ptr() + 16 * n * i, n, a.data_ptr() + 16 * n * i + 8 * n, n)
            for i in range(count)]
    B = FB.MpnBatch(ctx, reqs, configs=configs)
    B.keep = a, z
    return B


@pytest.mark.parametrize("logM,count", [(15, 1), (15, 4), (16, 1), (17, 2)])
def test_batches_of_few_products(ctx, logM, count):
    """A class too small to fill the GPU is as fast as with rows of the longest
    32-point columns: 0.99-1.08 (with the full classes' rows 1.13-1.24)."""
    torch = pytest.importorskip("torch")
    n = 1 << (logM - 1)
    plain = _batch(torch, ctx, n, count)
    fixed = _batch(torch, ctx, n, count, [FB.MulConfig(FB.ROUTE_NTT, 0, 0, logM - 5, 0)] * count)
    torch.cuda.synchronize()
    _ratio_below(torch, lambda s: plain.run(s), lambda s: fixed.run(s), 1.10)


def test_configured_short_rows(ctx):
    """2^15 points in rows of 2^7 against rows of 2^9: 1.18 (with inverse columns
    placed beside the rows 1.45)."""
    torch = pytest.importorskip("torch")
    n = 1 << 14
    a, b, z = _limbs(torch, n), _limbs(torch, n), _limbs(torch, 2 * n)
    torch.cuda.synchronize()
    run = lambda c: lambda s: ctx.mpn_mul_device_config(z.data_ptr(), a.data_ptr(), n, b.data_ptr(), n,
                                                        FB.MulConfig(FB.ROUTE_NTT, 0, 0, c, 0), s)
    _ratio_below(torch, run(7), run(9), 1.30, reps=100)


def test_squares_modulo_a_small_prime(ctx):
    """A square mod 3 on one prime against one mod 1000003 on two, 2^20 coefficients
    on 3 2^19 points: 0.71 (with inverse columns placed beside the rows 0.79)."""
    torch = pytest.importorskip("torch")
    n = 1 << 19
    a = torch.randint(0, 3, (n,), dtype=torch.int64, device="cuda")
    z = torch.empty(2 * n + 1001, dtype=torch.int64, device="cuda")
    m = n + 500                                    # a product of 2^20 + 999 coefficients
    a = torch.cat([a, a[:500]])
    torch.cuda.synchronize()
    run = lambda p: lambda s: ctx.nmod_poly_mul_mid_device(z.data_ptr(), 0, 2 * m - 1, a.data_ptr(), m, a.data_ptr(), m,
                                                           p, s)
    _ratio_below(torch, run(3), run(1000003), 0.75, reps=100)
