"""CRT recombination at its coefficient bound.

(B^n - 1)^2 has the largest coefficients an n-limb product can have, n (B - 1)^2
(at n = 2^24 the quotient k's margin is smallest), the longest carry chain, and a
closed form: limbs 1, 0 .. 0, B - 2, B - 1 .. B - 1.  Exact, so there is no
tolerance; n = 1 and n around the kernel's 512-limb tiles are included.
"""
import pytest

import flint_b200 as FB

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,np_", [(1, 5), (511, 5), (513, 5), (1 << 24, 5), (1, 6), (513, 6), (1 << 20, 6)])
def test_all_ones_square(ctx, n, np_):
    torch = pytest.importorskip("torch")
    a = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    b = a.clone()                                    # a product, then a squaring
    cfg = FB.MulConfig(FB.ROUTE_NTT, np_, 0, 0, 0)
    s = torch.cuda.current_stream().cuda_stream
    want = torch.full((2 * n,), -1, dtype=torch.int64, device="cuda")
    want[:n] = 0
    want[0] = 1
    want[n] = -2
    for other in (a, b):
        z = torch.zeros(2 * n, dtype=torch.int64, device="cuda")
        ctx.mpn_mul_device_config(z.data_ptr(), a.data_ptr(), n, other.data_ptr(), n, cfg, s)
        torch.cuda.synchronize()
        assert torch.equal(z, want)
