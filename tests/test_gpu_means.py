"""Face conductances from logK and their pullback against extended precision: the table-driven exponential
and the division of dpf_means.cuh over their whole range. Bounds: an exponential is within 0.54 ulp, a product,
sum or quotient within half an ulp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def _case(pkg, ns, lim, seed=0):
    coords, nb, aol, _ = pkg.regulargrid3d((0.0, 0.0, 0.0), (1.0, 1.0, 1.0), ns)
    rng = np.random.default_rng(seed)
    logK = rng.uniform(-lim, lim, coords.shape[1])
    return nb, aol, logK, rng.standard_normal(len(nb))


@pytest.mark.parametrize("general", [False, True])
@pytest.mark.parametrize("mean", ["geometric", "harmonic"])
@pytest.mark.parametrize("ns,lim", [((33, 17, 9), 0.01), ((33, 17, 9), 12.0), ((40, 1, 7), 160.0), ((2, 50, 1), 690.0)])
def test_means_and_pullback(gpu_lib, ns, lim, mean, general):
    nb, aol, logK, dKs = _case(gpu_lib, ns, lim)
    P = gpu_lib.GroundwaterProblem(nb, aol, np.array([0]), N=len(logK), general=general)
    assert P.structured != general
    a, b = nb[:, 0], nb[:, 1]
    with np.errstate(all="ignore"):
        k = np.exp(logK.astype(np.longdouble) / (2 if mean == "geometric" else 1))
        s = 1.0 if mean == "geometric" else k[a] + k[b]
        K = k[a] * k[b] if mean == "geometric" else 2 * k[a] * k[b] / s
        ga, gb = (K / 2, K / 2) if mean == "geometric" else (2 * k[a] * (k[b] / s) ** 2, 2 * k[b] * (k[a] / s) ** 2)
    got = P.logk_to_faces(logK, mean)
    assert np.all(np.abs(got - K) <= 2.1 * EPS * K + 5e-324)
    g = P.logk_to_faces_vjp(logK, dKs, mean)
    want, size = np.zeros(len(logK), np.longdouble), np.zeros(len(logK), np.longdouble)
    for i, w in ((a, ga * dKs), (b, gb * dKs)):
        np.add.at(want, i, w)
        np.add.at(size, i, np.abs(w))
    assert np.all(np.abs(g - want) <= 12 * EPS * size + 1e-300)


@pytest.mark.parametrize("general", [False, True])
def test_limits(gpu_lib, general):
    """Cell values beyond the reduced range: overflow, underflow, subnormals, infinities and NaN."""
    v = np.array([0.0, -0.0, 699.99, 700.0, 709.7, 710.0, -699.99, -700.0, -740.0, -746.0, np.inf, -np.inf, np.nan,
                  1399.9, 1400.0, 1419.0, -1399.9, -1400.0, 1e300, -1e300, 5e-324])
    n = len(v)
    nb = np.stack([np.arange(n), np.arange(n) + n], 1)   # each value beside a 1: K = exp(v / 2), 2 K / (1 + K)
    logK = np.concatenate([v, np.zeros(n)])
    if not general:
        coords, nb, aol, _ = gpu_lib.regulargrid3d((0.0, 0.0, 0.0), (1.0, 1.0, 1.0), (2, n, 1))
        faces = np.nonzero(nb[:, 1] - nb[:, 0] == n)[0]
    else:
        aol, faces = np.ones(n), np.arange(n)
    P = gpu_lib.GroundwaterProblem(nb, aol, np.array([0]), N=2 * n, general=general)
    with np.errstate(all="ignore"):
        np.testing.assert_allclose(P.logk_to_faces(logK, "geometric")[faces], np.exp(v / 2), rtol=4 * EPS, atol=1e-323)
        k = np.exp(v)
        np.testing.assert_allclose(P.logk_to_faces(logK, "harmonic")[faces], 2 * (k / (k + 1)), rtol=6 * EPS, atol=1e-323)


@pytest.mark.parametrize("where", ["host", "device", "overlap", "offset"])
def test_arrays_in_place(gpu_lib, where):
    """Inputs on the host, on the device, overlapping the output and at an address between two doubles: the same."""
    import ctypes
    import torch
    nb, aol, logK, dKs = _case(gpu_lib, (9, 8, 7), 3.0)
    n, F = len(logK), len(nb)
    P = gpu_lib.GroundwaterProblem(nb, aol, np.array([0]), N=n)
    want_K, want_g = P.logk_to_faces(logK), P.logk_to_faces_vjp(logK, dKs)
    if where == "host":
        got_K, got_g = P.logk_to_faces(logK.copy()), P.logk_to_faces_vjp(logK.copy(), dKs.copy())
    else:
        raw = torch.zeros(8 * (3 * F + 2 * n) + 64, dtype=torch.uint8, device="cuda")
        off = 4 if where == "offset" else 0

        def put(at, v):
            raw[at:at + 8 * len(v)] = torch.from_numpy(v.view(np.uint8).copy()).cuda()
            torch.cuda.synchronize()
            return raw.data_ptr() + at

        def get(at, m):
            torch.cuda.synchronize()
            return raw[at:at + 8 * m].cpu().numpy().view(np.float64)

        lk, dk, K = off, 8 * n + 16 + off, 8 * (n + F) + 32
        g = 8 * (n + 2 * F) + 48
        if where == "overlap":
            K, g = lk, dk + 8 * 5
        _f = lambda name, *a: gpu_lib._check(P._lib, P._h, getattr(P._lib, name)(P._h, *a))
        _f("dpf_logk_to_faces", ctypes.c_void_p(put(lk, logK)), 0, ctypes.c_void_p(raw.data_ptr() + K))
        got_K = get(K, F)
        _f("dpf_logk_to_faces_vjp", ctypes.c_void_p(put(lk, logK)), 0, ctypes.c_void_p(put(dk, dKs)),
           ctypes.c_void_p(raw.data_ptr() + g))
        got_g = get(g, n)
    assert np.array_equal(got_K, want_K) and np.array_equal(got_g, want_g)


@pytest.mark.parametrize("general", [False, True])
def test_pullback_of_cells_far_apart(gpu_lib, general):
    """Geometric means of cells up to 1300 e-folds apart: K is moderate, but either cell's value times dK overflows or
    vanishes. Also with a cell value that is 0 or subnormal, and a K that is. Twelve roundings as above."""
    # in an order in which no two neighbouring rows of the grid have an infinite K
    v = np.array([[-1200.0, 1199.0, 1e100], [1200.0, -1199.0, 1e-100], [-1300.0, 1299.0, -3e200], [1300.0, -1310.0, 2e-200],
                  [-1400.0, 1380.0, 1e300], [-700.0, -720.0, 1e200], [-1500.0, 1400.0, 1e10], [0.3, 0.4, 1e-300],
                  [-1430.0, 1400.0, 1e5]])
    m = len(v)
    logK = np.concatenate([v[:, 0], v[:, 1]])
    if general:
        nb, aol = np.stack([np.arange(m), np.arange(m) + m], 1), np.ones(m)
        faces = np.arange(m)
    else:
        _, nb, aol, _ = gpu_lib.regulargrid3d((0.0, 0.0, 0.0), (1.0, 1.0, 1.0), (2, m, 1))
        faces = np.nonzero(nb[:, 1] - nb[:, 0] == m)[0]
    dKs = np.zeros(len(nb))
    dKs[faces] = v[:, 2]
    P = gpu_lib.GroundwaterProblem(nb, aol, np.array([0]), N=2 * m, general=general)
    g = P.logk_to_faces_vjp(logK, dKs, "geometric")
    k = np.exp(v[:, :2] / 2)                          # as the cells' values, 0 and subnormal ones among them
    with np.errstate(all="ignore"):
        want = 0.5 * k[:, 0].astype(np.longdouble) * k[:, 1] * v[:, 2]
        sub = 2.0 ** -1074 * np.where(k < 1e-300, 1.0, 0.0).max(1) / np.maximum(k.min(1), 1e-323)  # rounding of exp itself
    for got in (g[:m], g[m:]):
        assert np.all(np.abs(got - want) <= (12 * EPS + 2 * sub) * np.abs(want) + 1e-300)
