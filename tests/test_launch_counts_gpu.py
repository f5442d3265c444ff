"""Launch counts are the kernels a call issues.

One launch for a transform of 2^9 to 2^12 points and the recombination behind
it; split, rows and recombination for the other one-row transforms, columns
besides for longer ones; for a host product a column launch for each operand, a's
early rows where it has them, and the recombination in the chunks of its download
(four, or one a 512-limb tile where the product has fewer); the short operand's
transform and three launches a chunk for a split product.  A batch's count is the
sum over its classes.
"""
import numpy as np
import pytest

import flint_b200 as FB
import oracle as O

pytestmark = pytest.mark.gpu


def _limbs(torch, n):
    return torch.randint(-(1 << 62), 1 << 62, (n,), dtype=torch.int64, device="cuda")


@pytest.mark.parametrize("an,bn,cfg,want", [
    (16, 16, None, 3), (100, 100, None, 3), (250, 250, None, 2), (2048, 2048, None, 2),
    (2048, 2048, FB.MulConfig(0, 0, 0, 0, FB.FLAG_ROWS32), 3), (4096, 4096, None, 4), (65536, 65536, None, 4),
    (4096, 4096, FB.MulConfig(0, 0, 0, 13, 0), 3), (700001, 650003, None, 4),
    (100, 100, FB.MulConfig(FB.ROUTE_BASECASE, 0, 0, 0, 0), 2)])
def test_device_products(ctx, an, bn, cfg, want):
    torch = pytest.importorskip("torch")
    a, b, z = _limbs(torch, an), _limbs(torch, bn), _limbs(torch, an + bn)
    if cfg is None:
        ctx.mpn_mul_device(z.data_ptr(), a.data_ptr(), an, b.data_ptr(), bn)
    else:
        ctx.mpn_mul_device_config(z.data_ptr(), a.data_ptr(), an, b.data_ptr(), bn, cfg)
    torch.cuda.synchronize()
    assert ctx.last_launches == want


def test_split_product(ctx):
    torch = pytest.importorskip("torch")
    an, bn = 5000000, 300000
    Lc = FB.mpn_mul_split_plan(an, bn)
    chunks = -(-an // ((1 << Lc) - bn + 1))
    a, b, z = _limbs(torch, an), _limbs(torch, bn), _limbs(torch, an + bn)
    ctx.mpn_mul_device(z.data_ptr(), a.data_ptr(), an, b.data_ptr(), bn)
    torch.cuda.synchronize()
    assert ctx.last_launches == 2 + 3 * chunks + 1


@pytest.mark.parametrize("n,want", [(300, 1 + 2), (50000, 3 + 1 + 4), (1 << 19, 3 + 2 + 4)])
def test_host_products(ctx, n, want):
    a, b = O.rand_limbs(1, n), O.rand_limbs(2, n)
    ctx.mpn_mul(a, b)
    assert ctx.last_launches == want


def test_polynomials(ctx):
    for n, want in ((20, 3), (700, 2), (9000, 4), (300000, 4)):
        a = O.rand_below(n, n, 1000003)
        ctx.nmod_poly_mul_mid(0, 2 * n - 1, a, a, 1000003)
        assert ctx.last_launches == want, n
    for n, want in ((10, 3), (500, 2), (9000, 4)):
        a = O.rand_fmpz_raw(n, n, 50)
        ctx.fmpz_poly_mul_mid(0, 2 * n - 1, a, a)
        assert ctx.last_launches == want, n


def test_batch_is_the_sum_of_its_classes(ctx):
    torch = pytest.importorskip("torch")
    want = {16: 3, 128: 3, 256: 2, 512: 2, 1024: 2, 2048: 2, 4096: 3, 8192: 4, 40000: 4}
    sizes = [n for n in want for _ in range(2)]
    a, z = _limbs(torch, 2 * sum(sizes)), _limbs(torch, 2 * sum(sizes))
    reqs, off = [], 0
    for n in sizes:
        reqs.append((z.data_ptr() + 8 * off, a.data_ptr() + 8 * off, n, a.data_ptr() + 8 * (off + n), n))
        off += 2 * n
    with FB.MpnBatch(ctx, reqs) as B:
        B.run(torch.cuda.current_stream().cuda_stream)
        B.check(torch.cuda.current_stream().cuda_stream)
        assert B.classes == len(want)
        assert B.launches == sum(want.values())
    host = z.cpu().numpy().view(np.uint64)
    assert host.any()
