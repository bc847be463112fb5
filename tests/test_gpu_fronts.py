"""The direct solver's fronts at the sizes where they can go wrong: fronts on both sides of the one-block
limit (76 rows), steps of exactly 16 own columns and with remainders, one-cell-wide and empty separators,
meshes in several components with isolated cells, a graph that cannot be halved. Against the oracle
(CG to 1e-14); heads 1e-11 and tangents 1e-9, the tolerances of the direct solver's other tests."""
import numpy as np
import pytest

from helpers import rel, steady_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [(16, 1, 1), (17, 1, 1), (2, 8, 1), (33, 3, 1), (38, 38, 1), (39, 38, 1), (16, 16, 16),
                                (17, 16, 15), (9, 130, 2), (100, 100, 1)])
def test_regular_fronts(gpu_lib, orc, ns):
    c = steady_case(gpu_lib, ns, sigma=1.5, seed=sum(ns), ndir=2, nq=3)
    delta = np.random.default_rng(6).standard_normal(c["N"])
    O = orc.Problem(c["N"], c["nb"], c["aol"], c["dn"])
    want = (O.steady(c["Ks"], c["dh"], c["Qs"], reltol=1e-14),) + tuple(O.adjoint(c["dh"], delta, reltol=1e-14))
    P = gpu_lib.GroundwaterProblem(c["nb"], c["aol"], c["dn"], N=c["N"], solver="cholesky")
    assert P.structured
    for _ in range(2):  # the second pass factors into used panels and pools
        got = (P.forward(c["Ks"], c["dh"], c["Qs"]),) + tuple(P.adjoint(delta))
        assert P.stats["iterations"] == 0 and P.stats["relres"] < 1e-12
        assert rel(got[0], want[0]) < 1e-11
        for g, w in zip(got[1:], want[1:]):
            assert rel(g, w) < 1e-9


def _mesh(kind):
    """Faces of three grids without connection (one of them a single cell), or of a star, or of a complete graph."""
    if kind == "components":
        parts, at = [], 0
        for nx, ny in ((23, 19), (1, 1), (40, 7)):
            i = at + np.arange(nx * ny).reshape(nx, ny)
            parts += [np.stack([i[:-1].ravel(), i[1:].ravel()], 1), np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1)]
            at += nx * ny
        return at, np.concatenate(parts), np.array([0, 23 * 19, 23 * 19 + 1, 5])
    if kind == "star":
        return 120, np.stack([np.zeros(119, np.int64), np.arange(1, 120)], 1), np.array([7])
    i, j = np.triu_indices(90, 1)
    return 90, np.stack([i, j], 1), np.array([3, 50])


@pytest.mark.parametrize("kind", ["components", "star", "complete"])
def test_mesh_fronts(gpu_lib, orc, kind):
    n, nb, dn = _mesh(kind)
    rng = np.random.default_rng(8)
    aol, Ks = rng.uniform(0.5, 2.0, len(nb)), np.exp(-9.0 + rng.standard_normal(len(nb)))
    dh, Qs, delta = np.zeros(n), np.zeros(n), rng.standard_normal(n)
    dh[dn] = rng.uniform(0, 1, len(dn))
    Qs[rng.choice(np.setdiff1d(np.arange(n), dn), 3, replace=False)] = [1e-4, 5e-5, -2e-5]
    P = gpu_lib.GroundwaterProblem(nb, aol, dn, N=n, general=True, solver="cholesky")
    got = (P.forward(Ks, dh, Qs),) + tuple(P.adjoint(delta))
    assert P.stats["iterations"] == 0 and P.stats["relres"] < 1e-12
    O = orc.Problem(n, nb, aol, dn)
    want = (O.steady(Ks, dh, Qs, reltol=1e-14),) + tuple(O.adjoint(dh, delta, reltol=1e-14))
    assert rel(got[0], want[0]) < 1e-11
    for g, w in zip(got[1:], want[1:]):
        assert rel(g, w) < 1e-9


def test_band_fronts(gpu_lib, orc):
    """A graph without small separators, with the memory for its band but not for its dissection: the fronts of the band
    order, 64 rows each with a remainder. Tolerances as above."""
    from test_direct_fronts import two_sets
    n, nb = two_sets(205, 0.3)
    rng = np.random.default_rng(8)
    aol, Ks = rng.uniform(0.5, 2.0, len(nb)), np.exp(-9.0 + rng.standard_normal(len(nb)))
    dn = np.array([3, 250])
    dh, Qs, delta = np.zeros(n), np.zeros(n), rng.standard_normal(n)
    dh[dn] = rng.uniform(0, 1, len(dn))
    Qs[[7, 100, 300]] = [1e-4, 5e-5, -2e-5]
    P = gpu_lib.GroundwaterProblem(nb, aol, dn, N=n, general=True, solver="cholesky")
    assert gpu_lib.load().dpf_debug_direct_memory(P._h, 3300000) == 0
    O = orc.Problem(n, nb, aol, dn)
    want = (O.steady(Ks, dh, Qs, reltol=1e-14),) + tuple(O.adjoint(dh, delta, reltol=1e-14))
    for _ in range(2):
        got = (P.forward(Ks, dh, Qs),) + tuple(P.adjoint(delta))
        assert P.stats["iterations"] == 0 and P.stats["relres"] < 1e-12
        assert rel(got[0], want[0]) < 1e-11
        for g, w in zip(got[1:], want[1:]):
            assert rel(g, w) < 1e-9
