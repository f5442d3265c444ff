"""Chains of products whose kernels start before their predecessors end.

The kernels of a short product run as programmatic dependents of one another
and of the product before them on the stream.  Each product of a chain here
reads what the one before it wrote and shares its scratch, so a kernel that
did not wait for its predecessor would show; sizes straddle the launch rules
(narrow column tiles, 2^20 points, 3 2^k lengths).  Every value is compared
with GMP, so there is no tolerance.
"""
import numpy as np
import pytest

import flint_b200 as FB
import oracle as O

pytestmark = pytest.mark.gpu


def _dev(torch, a):
    return torch.from_numpy(a.view(np.int64)).cuda()


@pytest.mark.parametrize("n", [1, 17, 700, 4096, 8193, 40000, 131072, 131073, 300000, 524288, 600000])
def test_chain_reads_predecessors_output(ctx, n):
    """x <- low n limbs of x y, four times on one stream, then a squaring."""
    torch = pytest.importorskip("torch")
    x, y = O.rand_limbs(n + 1, n), O.rand_limbs(n + 2, n)
    dx, dy = _dev(torch, x), _dev(torch, y)
    bufs = [torch.full((2 * n,), -1, dtype=torch.int64, device="cuda") for _ in range(2)]
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    src = dx
    for k in range(4):
        z = bufs[k & 1]
        ctx.mpn_mul_device(z.data_ptr(), src.data_ptr(), n, dy.data_ptr(), n, s.cuda_stream)
        src = z
    w = bufs[0]
    ctx.mpn_mul_device(w.data_ptr(), src.data_ptr(), n, src.data_ptr(), n, s.cuda_stream)
    s.synchronize()
    want = x
    for _ in range(4):
        z = O.gmp_mpn_mul(want, y)
        want = z[:n]
    assert (bufs[1].cpu().numpy().view(np.uint64) == z).all()
    assert (w.cpu().numpy().view(np.uint64) == O.gmp_mpn_mul(want, want)).all()


@pytest.mark.parametrize("n", [700, 40000, 131072])
def test_captured_products_replay(n):
    """Two dependent allocation-free products captured in a CUDA graph and
    replayed on new values."""
    torch = pytest.importorskip("torch")
    dx, dy = _dev(torch, O.rand_limbs(n + 1, n)), _dev(torch, O.rand_limbs(n + 2, n))
    z, w = (torch.empty(2 * n, dtype=torch.int64, device="cuda") for _ in range(2))
    mul = FB.lib().gpu_mpn_mul_device_noalloc

    def call():
        s = torch.cuda.current_stream().cuda_stream
        assert mul(z.data_ptr(), dx.data_ptr(), n, dy.data_ptr(), n, s) == FB.OK
        assert mul(w.data_ptr(), z.data_ptr(), n, dy.data_ptr(), n, s) == FB.OK

    call()                      # the one-time set-up is outside the capture
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    for r in range(3):
        x = O.rand_limbs(n + 10 + r, n)
        y = O.rand_limbs(n + 20 + r, n)
        dx.copy_(_dev(torch, x))
        dy.copy_(_dev(torch, y))
        g.replay()
        torch.cuda.synchronize()
        zz = O.gmp_mpn_mul(x, y)
        assert (z.cpu().numpy().view(np.uint64) == zz).all()
        assert (w.cpu().numpy().view(np.uint64) == O.gmp_mpn_mul(zz[:n], y)).all()
