"""The device forms of the exponential delay and of the clock advance give
the bits of the definitions they replace.

* exp_delay: the integer draw's exponent and mantissa are split before the
  scaling and the logarithm's quotient is a Markstein division; every one of
  the 2^24 draws is compared with the host's form (tolerance: none).
* GELU: its sigmoid's reciprocal is an approximation and a Newton step; a
  grid of 2^24 floats over the exponents where the sigmoid is neither 0 nor
  1, and the clamped ends, are compared with the host's form (none).
* The reciprocal itself: every float of [1, 2^126] against the double
  quotient rounded to float (none; 53 bits rounded to 24 is the quotient
  rounded once).
* time_add: one float addition instead of a double sum rounded to float, in
  numpy and in the device's form.
"""
import numpy as np
import pytest

import oracle


@pytest.mark.gpu
def test_exp_delay_of_every_draw_equals_the_host():
    import torch
    from cusmc_b200 import _native
    from cusmc_b200._native import check, lib
    x = np.arange(1 << 24, dtype=np.uint32) << np.uint32(8)
    inv = np.ones(x.size, dtype=np.float32)
    got = torch.empty(x.size, dtype=torch.float32, device="cuda")
    xd, invd = torch.from_numpy(x.view(np.int32)).cuda(), torch.from_numpy(inv).cuda()
    check(lib().csmc_numeric_eval(_native.NUM_EXP_DELAY, xd.data_ptr(), invd.data_ptr(), x.size, got.data_ptr(), None))
    torch.cuda.synchronize()
    want = oracle.numeric(_native.NUM_EXP_DELAY, x, inv)
    assert np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.gpu
def test_gelu_over_a_dense_grid_equals_the_host():
    import torch
    from cusmc_b200 import _native
    from cusmc_b200._native import check, lib
    step = np.arange(1 << 22, dtype=np.uint32) * np.uint32(37)
    x = np.concatenate([(np.uint32(0x3c000000) + step % np.uint32(0x05000000)).view(np.float32),
                        -(np.uint32(0x3c000000) + step % np.uint32(0x05000000)).view(np.float32),
                        np.linspace(-12.0, 12.0, 1 << 23, dtype=np.float32),
                        np.array([0.0, -0.0, 50.0, -50.0, 1e9, -1e9, 3e38, -3e38], np.float32)])
    for fn in (_native.NUM_GELU_F32, _native.NUM_GELU_GRAD_F32):
        got = torch.empty(x.size, dtype=torch.float32, device="cuda")
        xd = torch.from_numpy(x).cuda()
        check(lib().csmc_numeric_eval(fn, xd.data_ptr(), None, x.size, got.data_ptr(), None))
        torch.cuda.synchronize()
        want = oracle.numeric(fn, x)
        same = got.cpu().numpy().view(np.uint32) == want.view(np.uint32)
        assert np.all(same | (np.isnan(want) & np.isnan(got.cpu().numpy())))


def test_float_sum_equals_the_double_sum_rounded_to_float():
    """Random floats over all exponents (subnormal results, cancellation,
    exponent gaps around the 24- and 53-bit limits, overflow)."""
    rng = np.random.default_rng(5)
    n = 4_000_000
    a = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32).view(np.float32)
    gap = rng.integers(-60, 61, n)
    m = (1.0 + rng.integers(0, 2**23, n) * 2.0 ** -23) * rng.choice([-1.0, 1.0], n)
    with np.errstate(all="ignore"):
        b = np.where(np.isfinite(a), np.ldexp(m, np.frexp(a)[1] + gap), 1.0).astype(np.float32)
        ok = np.isfinite(a) & np.isfinite(b)
        a, b = a[ok], b[ok]
        once = a + b
        twice = (a.astype(np.float64) + b.astype(np.float64)).astype(np.float32)
    assert np.array_equal(once.view(np.uint32), twice.view(np.uint32))


@pytest.mark.gpu
def test_reciprocal_of_every_float_from_one_to_2_126_equals_the_quotient():
    import torch
    from cusmc_b200 import _native
    from cusmc_b200._native import check, lib
    mantissas = torch.arange(1 << 23, dtype=torch.int32, device="cuda")
    got = torch.empty(1 << 23, dtype=torch.float32, device="cuda")
    for e in range(127):  # (at the last exponent 2^126 alone)
        x = (mantissas if e < 126 else torch.zeros_like(mantissas)).add((e + 127) << 23).view(torch.float32)
        check(lib().csmc_numeric_eval(_native.NUM_RCP_F32, x.data_ptr(), None, x.numel(), got.data_ptr(), None))
        want = (1.0 / x.double()).float()
        assert torch.equal(got.view(torch.int32), want.view(torch.int32)), e


@pytest.mark.gpu
def test_device_time_add_equals_the_double_sum_rounded_to_float():
    import torch
    from cusmc_b200 import _native
    from cusmc_b200._native import check, lib
    rng = np.random.default_rng(6)
    n = 4_000_000
    a = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32).view(np.float32)
    m = (1.0 + rng.integers(0, 2**23, n) * 2.0 ** -23) * rng.choice([-1.0, 1.0], n)
    with np.errstate(all="ignore"):
        b = np.where(np.isfinite(a), np.ldexp(m, np.frexp(a)[1] + rng.integers(-60, 61, n)), 1.0).astype(np.float32)
        ok = np.isfinite(a) & np.isfinite(b)
        a, b = a[ok], b[ok]
        want = (a.astype(np.float64) + b.astype(np.float64)).astype(np.float32)
    ad, bd = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    got = torch.empty(a.size, dtype=torch.float32, device="cuda")
    check(lib().csmc_numeric_eval(_native.NUM_TIME_ADD, ad.data_ptr(), bd.data_ptr(), a.size, got.data_ptr(), None))
    assert np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))
