"""Every host entry point reports the context's error flag, and clears it.

A kernel whose bounded wait gives up sets the flag and finishes with wrong
values, so a host call that does not read it returns them as a success and
leaves the flag to fail some unrelated call later.  The flag is planted from the
host as such a kernel would set it (valid inputs never do); the call after
the report must be exact.
"""
import numpy as np
import pytest

import flint_b200 as FB
import oracle as O

pytestmark = pytest.mark.gpu

MOD = (1 << 61) + 15


def _nmod(ctx):
    a, b = O.rand_below(1, 3000, MOD), O.rand_below(2, 2000, MOD)
    return (lambda: ctx.nmod_poly_mul_mid(100, 4500, a, b, MOD)), O.port_nmod_mul_mid(100, 4500, a, b, MOD)


def _fmpz(ctx):
    a, b = O.rand_fmpz_raw(3, 200, 120), O.rand_fmpz_raw(4, 150, 120)
    want = O.fmpz_poly_mul_python(O.raw_to_ints(a), O.raw_to_ints(b))
    return (lambda: O.raw_to_ints(ctx.fmpz_poly_mul_mid(0, 349, a, b))), want


def _ring(ctx):
    N = 47104
    C = FB.Mulmod2expp1(ctx, N)
    x, y = O.neg_operand(5, N // 64), O.neg_operand(6, N // 64)
    return (lambda: C.mul(x, y)), O.negmul_python(x, y, N)


def _divrem(ctx):
    a, b = O.rand_below(7, 900, 101), O.rand_below(8, 400, 101)
    b[-1] = 1
    return (lambda: ctx.nmod_poly_divrem(a, b, 101)[0]), O.nmod_divrem_python(a, b, 101)[0]


@pytest.mark.parametrize("case", [_nmod, _fmpz, _ring, _divrem])
def test_host_call_reports_and_clears(ctx, case):
    call, want = case(ctx)
    FB._check(FB.lib().gpu_test_set_device_error(ctx.ptr))
    with pytest.raises(FB.GpuFftSmallError) as e:
        call()
    assert e.value.code == FB.ETIMEOUT
    assert np.array_equal(np.asarray(call(), dtype=object), np.asarray(want, dtype=object))


def test_device_calls_have_a_check(ctx):
    torch = pytest.importorskip("torch")
    s = torch.cuda.current_stream().cuda_stream
    a = O.rand_below(9, 5000, MOD)
    d = torch.from_numpy(a.view(np.int64)).cuda()
    z = torch.empty(9999, dtype=torch.int64, device="cuda")
    ctx.nmod_poly_mul_mid_device(z.data_ptr(), 0, 9999, d.data_ptr(), 5000, d.data_ptr(), 5000, MOD, s)
    ctx.check(s)
    assert (z.cpu().numpy().view(np.uint64) == O.port_nmod_mul_mid(0, 9999, a, a, MOD)).all()
    FB._check(FB.lib().gpu_test_set_device_error(ctx.ptr))
    with pytest.raises(FB.GpuFftSmallError) as e:
        ctx.check(s)
    assert e.value.code == FB.ETIMEOUT
    ctx.check(s)


@pytest.mark.parametrize("bits,code,words", [(1, "ETIMEOUT", ["carry"]), (2, "ETIMEOUT", ["row pass", "matrix product"]),
                                             (3, "ETIMEOUT", ["row pass", "carry"]), (4, "ECUDA", ["row pass", "aligned"])])
def test_message_names_the_kernel(ctx, bits, code, words):
    """The row pass's errors are not reported as the carry look-back's."""
    FB._check(FB.lib().gpu_test_set_device_error_bits(ctx.ptr, bits))
    with pytest.raises(FB.GpuFftSmallError) as e:
        ctx.mpn_mul(O.rand_limbs(1, 100), O.rand_limbs(2, 100))
    assert e.value.code == getattr(FB, code)
    assert all(w in str(e.value) for w in words)
    assert ("carry" in str(e.value)) == bool(bits & 1)
    ctx.check()


def test_error_of_an_earlier_device_call_is_not_lost():
    """A host call that launches no kernel which can set the flag skips reading it,
    but not after a device-pointer call on another stream, whose kernels may end
    after any number of reads."""
    torch = pytest.importorskip("torch")
    with FB.MpnCtx() as c:
        s = torch.cuda.Stream()
        a = torch.randint(-(1 << 62), 1 << 62, (100,), dtype=torch.int64, device="cuda")
        z = torch.empty(200, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        c.mpn_mul_device(z.data_ptr(), a.data_ptr(), 100, a.data_ptr(), 100, s.cuda_stream)
        x = O.rand_below(1, 50, MOD)
        want = O.port_nmod_mul_mid(0, 99, x, x, MOD)
        for _ in range(2):
            assert (c.nmod_poly_mul_mid(0, 99, x, x, MOD) == want).all()
        s.synchronize()
        FB._check(FB.lib().gpu_test_set_device_error_bits(c.ptr, 1 + 256))
        c2 = FB.lib().gpu_mpn_ctx_check
        with pytest.raises(FB.GpuFftSmallError):
            c.nmod_poly_mul_mid(0, 99, x, x, MOD)
        assert (c.nmod_poly_mul_mid(0, 99, x, x, MOD) == want).all()
        assert c2(c.ptr, None) == FB.OK
