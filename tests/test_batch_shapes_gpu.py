"""Planned batches on both sides of the class sizes where the row length changes.

Classes of 2^14 to 2^18 points take the short rows of a full GPU or, with fewer
products, a single product's rows; a configured request with the same key and
promoted ones share the plan.  Compared with GMP on every limb.
"""
import numpy as np
import pytest

import flint_b200 as FB
import oracle as O

pytestmark = pytest.mark.gpu


def _check(ctx, sizes, configs=None, **opts):
    torch = pytest.importorskip("torch")
    a = [O.rand_limbs(3 * i + 1, an) for i, (an, _) in enumerate(sizes)]
    b = [O.rand_limbs(3 * i + 2, bn) for i, (_, bn) in enumerate(sizes)]
    da = [torch.from_numpy(x.view(np.int64)).cuda() for x in a]
    db = [torch.from_numpy(x.view(np.int64)).cuda() for x in b]
    z = [torch.full((an + bn,), -1, dtype=torch.int64, device="cuda") for an, bn in sizes]
    reqs = [(z[i].data_ptr(), da[i].data_ptr(), an, db[i].data_ptr(), bn) for i, (an, bn) in enumerate(sizes)]
    s = torch.cuda.current_stream().cuda_stream
    with FB.MpnBatch(ctx, reqs, configs=configs, **opts) as B:
        for _ in range(2):
            B.run(s)
        B.check(s)
    for i in range(len(sizes)):
        assert (z[i].cpu().numpy().view(np.uint64) == O.gmp_mpn_mul(a[i], b[i])).all(), i


@pytest.mark.parametrize("logM,count", [(14, 1), (14, 7), (14, 8), (15, 1), (15, 14), (15, 15), (16, 7), (16, 8),
                                        (17, 3), (17, 4), (18, 1), (18, 2)])
def test_class_sizes(ctx, logM, count):
    n = 1 << (logM - 1)
    _check(ctx, [(n - 3 * i, n - 7 * i) if i else (n, n) for i in range(count)])


def test_mixed_with_configured_and_promoted(ctx):
    sizes = [(40000, 20000)] * 3 + [(8000, 8000)] * 2 + [(16000, 300)] * 3
    cfg = lambda c, np_=0: FB.MulConfig(FB.ROUTE_NTT, np_, 0, c, 0)
    configs = [cfg(0), cfg(9), cfg(0, 6), cfg(0), cfg(9), cfg(0), cfg(0), cfg(11)]
    _check(ctx, sizes, configs)
    _check(ctx, sizes, configs, promote_small=4)
    _check(ctx, sizes, promote_small=6, max_streams=1, use_graph=False)


@pytest.mark.parametrize("logM", [14, 15, 16, 17])
def test_narrow_column_tiles(ctx, logM):
    """Columns of 2^5 to 2^8 points in classes small enough for narrow tiles."""
    n = 1 << (logM - 1)
    _check(ctx, [(n, n), (n - 5, n - 1000)], [FB.MulConfig(FB.ROUTE_NTT, 0, 0, 9, 0)] * 2)
