"""dB scaling on the device at the sizes where its kernels change (one CTA up
to 32 768 values, two kernels above) and at every alignment of the buffers,
against the rule in float64.

Tolerance: |y| stays below 800 dB here, and log10f (2 ulp), the division (half
an ulp) and the product (half an ulp) are off by at most 3 * 2^-23 of it, so
3e-4 dB; values near 0 dB carry the division's 2^-24 through the logarithm,
under 1e-6 dB."""

import numpy as np
import pytest

import metalmom_b200 as M

pytestmark = pytest.mark.gpu

TOL = 3e-4
SIZES = [1, 3, 4, 5, 1023, 32767, 32768, 32769, 4 * 303104 + 2, 5000003]


def _expected(x, mult, amin, ref, top_db):
    x = x.astype(np.float64)
    with np.errstate(all="ignore"):
        y = mult * np.log10(np.where(x >= np.float32(amin), x, np.float64(np.float32(amin))) / ref)
        if top_db is None:
            return y
        top = np.fmax.reduce(y, initial=-np.inf)
        return np.where(y >= top - top_db, y, top - top_db)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("shift_in,shift_out", [(0, 0), (1, 0), (0, 3), (2, 2)])
def test_db_device_sizes_and_alignments(n, shift_in, shift_out):
    import torch
    rng = np.random.default_rng(n + shift_in)
    x = np.exp(4.0 * rng.standard_normal(n)).astype(np.float32)
    x[rng.random(n) < 0.1] = 0.0
    buf = torch.full((n + 8,), -7.0, device="cuda")
    out = torch.full((n + 8,), -7.0, device="cuda")
    xin, y = buf[shift_in:shift_in + n], out[shift_out:shift_out + n]
    xin.copy_(torch.from_numpy(x))
    for fn, mult, amin in ((M.power_to_db_device, 10.0, 1e-10), (M.amplitude_to_db_device, 20.0, 1e-5)):
        for ref, top_db in ((1.0, 80.0), (np.max, 80.0), (2.5, None), (np.max, None), (0.5, 30.0)):
            r = float(max(x.max(), 0.0)) if ref is np.max else ref
            if r == 0.0:
                continue
            out.fill_(-7.0)
            fn(xin, ref=ref, amin=amin, top_db=top_db, out=y)
            got = out.cpu().numpy()
            np.testing.assert_allclose(got[shift_out:shift_out + n], _expected(x, mult, amin, r, top_db), rtol=0, atol=TOL)
            assert (got[:shift_out] == -7.0).all() and (got[shift_out + n:] == -7.0).all()
    M.power_to_db_device(xin, out=xin)
    np.testing.assert_allclose(buf.cpu().numpy()[shift_in:shift_in + n], _expected(x, 10.0, 1e-10, 1.0, 80.0), rtol=0,
                               atol=TOL)


@pytest.mark.parametrize("n", [1000, 200001])
def test_db_device_special_values(n):
    """NaN and infinite inputs, an amin that is not positive (the pass-by-pass
    form), a reference that is not positive."""
    import torch
    rng = np.random.default_rng(n)
    base = np.exp(rng.standard_normal(n)).astype(np.float32)
    for bad in (np.nan, np.inf, -np.inf, -3.0):
        x = base.copy()
        x[n // 2] = bad
        d = torch.from_numpy(x).cuda()
        for amin, ref, top_db in ((1e-10, 1.0, 80.0), (0.0, 1.0, 80.0), (-1.0, 2.0, 80.0), (1e-10, -1.0, 80.0),
                                  (1e-10, 1.0, None), (1e-10, np.inf, 80.0)):
            got = M.power_to_db_device(d, ref=ref, amin=amin, top_db=top_db).cpu().numpy()
            exp = _expected(x, 10.0, amin, np.float64(ref), top_db)
            assert (np.isnan(got) == np.isnan(exp)).all(), (bad, amin, ref)
            fin = np.isfinite(exp)
            assert (got[~fin & ~np.isnan(exp)] == exp[~fin & ~np.isnan(exp)]).all()
            np.testing.assert_allclose(got[fin], exp[fin], rtol=0, atol=TOL)
    x = base.copy()
    x[1] = np.nan
    got = M.power_to_db_device(torch.from_numpy(x).cuda(), ref=np.max, top_db=None).cpu().numpy()
    assert np.isnan(got).all()


@pytest.mark.parametrize("n", [7, 32768, 100003])
@pytest.mark.parametrize("scale", [2.0 ** -58, 1e-9, 1.0, 2.0 ** 40, 2.0 ** 59, 2.0 ** 61, 1e38])
def test_db_device_accuracy_by_magnitude(n, scale):
    """Both forms of the logarithm (values inside [2^-60, 2^60] and beyond) to a
    few roundings.  Per 10 dB of `mult`: the quotient's 2^-24 is 2.6e-7 dB, the
    logarithm of the mantissa (at most 1.51 dB) takes three roundings of 2^-24,
    2.7e-7 dB (log10f: 2 ulp of y), and the sums and product two of y."""
    import torch
    rng = np.random.default_rng(n)
    x = (scale * np.exp2(rng.uniform(-1.0, 1.0, n))).astype(np.float32)
    x[::3] = (scale * (1.0 + np.float64(2.0 ** -23) * rng.integers(-40, 40, len(x[::3])))).astype(np.float32)
    d = torch.from_numpy(x).cuda()
    for fn, mult in ((M.power_to_db_device, 10.0), (M.amplitude_to_db_device, 20.0)):
        for amin in (1e-30, float(np.float32(scale))):
            for ref in (1.0, np.max, float(np.float32(scale * 0.7))):
                r = float(max(x.max(), np.float32(amin))) if ref is np.max else ref
                y = fn(d, ref=ref, amin=amin, top_db=100.0).cpu().numpy().astype(np.float64)
                e = _expected(x, mult, amin, np.float64(r), 100.0)
                assert (np.abs(y - e) <= 1e-6 * mult / 10 + 2.0 ** -21 * np.abs(e)).all()
