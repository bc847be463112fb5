"""The table-driven power and logarithm of the relative-permeability kernels on the device against extended
precision, over all 128 intervals of the logarithm's table, both sides of x = 1, exponents of either sign up to 1000,
and on both sides of each hand-over to the library's function.
Bounds. The power for |y| <= 6: half an ulp, the exponential's table 0.01, the logarithm's error 6 2^-61 (0.03 ulp),
and the degree-4 polynomial beyond its range R = 1.36e-3 by y lo <= 6 2^-15, where its Chebyshev remainder 2.3e-18
has grown by T5(1.14) = 6.9 (0.15 ulp): 0.7. Elsewhere the library's 2 ulp. The logarithm hi + lo: the rounding of
m c - 1 at 2^-61, of the table 2^-97 and of the polynomial 2^-66: 2^-60.5."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble


def _pow(pkg, x, y):
    import torch
    x, y = np.broadcast_arrays(np.asarray(x, np.float64), np.asarray(y, np.float64))
    d = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (x, y)]
    out = [torch.full((x.size,), 7.0, dtype=torch.float64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    rc = pkg.load().dpf_debug_pow64(x.size, *[ctypes.c_void_p(t.data_ptr()) for t in d + out])
    assert rc == 0
    return [t.cpu().numpy() for t in out]


def _intervals(rng, n, exponents):
    """n significands in each of the 128 intervals, their ends among them, times powers of two."""
    j = np.repeat(np.arange(128), n)
    m = 1.0 + (j + rng.random(j.size)) / 128
    m[::n] = 1.0 + j[::n] / 128
    m[1::n] = np.nextafter(1.0 + (j[1::n] + 1) / 128, 0)
    return m * 2.0 ** rng.choice(exponents, j.size)


def _ulps(got, want):
    """Error in units in the last place of the exact value (subnormal results: of the smallest subnormal)."""
    with np.errstate(all="ignore"):
        e = np.maximum(np.floor(np.log2(np.abs(want))), LD(-1022))
        return np.abs((got.astype(LD) - want) / LD(2.0) ** (e - 52))


@pytest.mark.parametrize("ymax", [0.05, 0.9, 3.0, 5.999, 6.01, 8.0, 16.0, 40.0, 100.0, 1000.0])
@pytest.mark.parametrize("exponents", [[0], [-1], [-1, 0], range(-30, 30), range(-990, 990)])
def test_power(gpu_lib, ymax, exponents):
    rng = np.random.default_rng(int(10 * ymax))
    x = _intervals(rng, 400, np.array(exponents))
    near = np.exp(rng.uniform(-0.02, 0.02, 20000) / max(ymax / 40, 1.0))
    x = np.concatenate([x, near, 1.0 + np.arange(-40, 41) * 2.0 ** -52])
    y = ymax * rng.uniform(0.7, 1.0, x.size) * rng.choice([-1.0, 1.0], x.size)
    p = _pow(gpu_lib, x, y)[0]
    with np.errstate(all="ignore"):
        want = np.power(x.astype(LD), y.astype(LD))
        ok = (want < LD(1.79e308)) & (want > LD(1e-320))
        table = (np.abs(y) <= 6) & (np.abs(y * np.log(x)) < 699.9)
    assert np.all(_ulps(p[ok], want[ok]) <= np.where(table, 0.7, 2.0)[ok])


def test_limits(gpu_lib):
    """Zero, subnormal, infinite and NaN bases, results that overflow or underflow, infinite and NaN exponents."""
    x = np.array([0.0, 5e-324, 1e-310, 2.0 ** -1001, 2.0 ** -999, 2.0 ** 999, 2.0 ** 1001, np.inf, np.nan, 1.0, 2.0])
    y = np.array([-1000.0, -7.0, -6.0, -1.0, -0.5, 0.0, 0.5, 1.0, 6.0, 7.0, 1000.0, np.inf, -np.inf, np.nan])
    X, Y = (v.ravel() for v in np.meshgrid(x, y))
    p, hi, lo = _pow(gpu_lib, X, Y)
    with np.errstate(all="ignore"):
        want = np.power(X.astype(LD), Y.astype(LD))
        w64 = want.astype(np.float64)
        log = np.log(X)
    for k in range(X.size):
        if np.isnan(w64[k]):
            assert np.isnan(p[k]), (X[k], Y[k])
        elif np.isinf(w64[k]) or w64[k] == 0:
            assert p[k] == w64[k], (X[k], Y[k])
        else:
            assert _ulps(p[k:k + 1], want[k:k + 1])[0] <= 2.0, (X[k], Y[k])
    np.testing.assert_allclose(hi + lo, log, rtol=2 * 2.0 ** -52, atol=0)


def test_logarithm(gpu_lib):
    rng = np.random.default_rng(9)
    x = np.concatenate([_intervals(rng, 400, [0]), _intervals(rng, 400, [-1]), _intervals(rng, 400, range(-990, 990)),
                        1.0 + np.arange(-40, 41) * 2.0 ** -52])
    _, hi, lo = _pow(gpu_lib, x, 1.0)
    want = np.log(x.astype(LD))  # a long double of 64 bits adds its own rounding
    assert np.all(np.abs((hi.astype(LD) + lo.astype(LD)) - want) <= 2.0 ** -60.5 + 2 * np.finfo(LD).eps * np.abs(want))
