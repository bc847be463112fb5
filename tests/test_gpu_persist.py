"""The one-launch solve (the persistent kernel) against the oracle and against the separate kernels
(use_graphs = 0), at the sizes where its parts meet: grids of a single level (up to 64 cells), levels on
both sides of the one-block tail's limits (512 cells in FP64, 2048 in FP32), one-cell-thick and odd axes,
every parity of the smoothing degree, and batches with fewer and with more problems than shares.
Tolerances: heads 1e-8 and gradients 1e-6 of the oracle's, and 1e-10 / 1e-8 between the two paths (their
V-cycles agree to rounding, and both solve to 1e-12)."""
import numpy as np
import pytest

from helpers import rel, steady_case

pytestmark = pytest.mark.gpu


def _solve(pkg, cases, **opt):
    B = pkg.GroundwaterBatch([c["ns"] for c in cases], [c["mins"] for c in cases], [c["maxs"] for c in cases],
                             [c["dn"] for c in cases], reltol=1e-12, **opt)
    cat = lambda k: np.concatenate([c[k] for c in cases])
    obs = [np.arange(0, c["N"], 3) for c in cases]
    h, g = B.solve_grad_logk(cat("logK"), cat("dh"), cat("Qs"), obs)
    return B, obs, np.asarray(h), np.asarray(g)


def _check(pkg, orc, cases, **opt):
    B, obs, h, g = _solve(pkg, cases, **opt)
    B0, _, h0, g0 = _solve(pkg, cases, use_graphs=0, **opt)
    assert B.launch_count < B0.launch_count  # one launch per solve
    off = B.cell_offsets
    for k, c in enumerate(cases):
        s = slice(off[k], off[k + 1])
        O = orc.Problem(c["N"], c["nb"], c["aol"], c["dn"])
        ho = O.steady(orc.logk_to_faces(c["nb"], c["logK"]), c["dh"], c["Qs"], reltol=1e-14)
        d = np.zeros(c["N"])
        np.add.at(d, obs[k], 2 * ho[obs[k]])
        go = orc.logk_to_faces_vjp(c["nb"], c["logK"], O.adjoint(c["dh"], d, reltol=1e-14)[0])
        assert rel(h[s], ho) < 1e-8 and rel(g[s], go) < 1e-6, k
        assert rel(h[s], h0[s]) < 1e-10 and rel(g[s], g0[s]) < 1e-8, k


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ns", [(4, 4, 4), (5, 13, 1), (1, 1, 70), (16, 16, 16), (17, 16, 16), (33, 9, 7),
                                (26, 25, 26), (51, 2, 43)])
def test_one_grid(gpu_lib, orc, ns, precision):
    _check(gpu_lib, orc, [steady_case(gpu_lib, ns, ell=4.0, sigma=1.0, seed=sum(ns), ndir=2, nq=2)], precision=precision)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("degree", [1, 3, 4])
def test_smoothing_degrees(gpu_lib, orc, degree, precision):
    _check(gpu_lib, orc, [steady_case(gpu_lib, (21, 18, 9), sigma=1.0, seed=3, ndir=1, nq=2)], precision=precision,
           cheb_degree=degree)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shapes", [[(4, 4, 3), (20, 17, 9), (40, 6, 5)], [(3, 3, 3), (5, 4, 3)],
                                    [(6, 5, 4)] * 90 + [(24, 20, 10)]])
def test_batches(gpu_lib, orc, shapes, precision):
    cases = [steady_case(gpu_lib, ns, sigma=1.0, seed=k % 7, ndir=1 + k % 2, nq=2) for k, ns in enumerate(shapes)]
    _check(gpu_lib, orc, cases, precision=precision)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nprob", [24, 25, 48, 49, 96, 97, 152])
def test_sums_of_many_problems(gpu_lib, orc, nprob, precision):
    """Both sides of every change in the number of lanes that add up a problem's slots (32 down to 4). Problems of
    different sizes and positions, so that a sum with another problem's slots would show."""
    shapes = [((7, 5, 3), (6, 6, 4), (5, 4, 8))[k % 3] for k in range(nprob)]
    cases = [steady_case(gpu_lib, ns, sigma=1.0, seed=k, ndir=1 + k % 2, nq=2) for k, ns in enumerate(shapes)]
    _check(gpu_lib, orc, cases, precision=precision)


@pytest.mark.parametrize("shapes,streams,precision,one_launch", [
    ([(5, 5, 4)] * 150 + [(100, 100, 20)], 0, "fp64", False),     # one share would hold 13 even ones
    ([(5, 5, 4)] * 150 + [(100, 100, 20)], 0, "mixed", False),
    ([(30, 30, 10)] * 77, 0, "fp64", False),                      # twice the even share
    ([(30, 30, 10)] * 77, 0, "mixed", False),
    ([(30, 30, 10)] * 76, 0, "fp64", True),
    ([(12, 10, 6)] * 4, 2, "fp64", False),                        # small parts: each would fill the GPU in turn
    ([(12, 10, 6)] * 4, 2, "mixed", False),
    ([(120, 120, 10)] * 4, 2, "fp64", True),                      # large ones: one-launch solves on two streams
    ([(120, 120, 10)] * 4, 3, "fp64", False),
])
def test_form_of_a_batch(gpu_lib, shapes, streams, precision, one_launch):
    """Batches whose shares or parts the one-launch solve would leave waiting take the separate kernels (some
    hundred launches); either form, also from several host threads and streams, gives the host-driven loop's result.
    Both solve to 1e-12; tolerances as above."""
    cases = [steady_case(gpu_lib, ns, sigma=1.0, seed=k % 5, ndir=1 + k % 2, nq=2) for k, ns in enumerate(shapes)]
    B, obs, h, g = _solve(gpu_lib, cases, precision=precision, streams=streams)
    launches = B.launch_count
    assert (launches < 60 * max(streams, 1)) == one_launch
    B0, _, h0, g0 = _solve(gpu_lib, cases, use_graphs=0, precision=precision)
    off = B.cell_offsets
    cat = lambda k: np.concatenate([c[k] for c in cases])
    for _ in range(3):
        for k in range(len(cases)):
            s = slice(off[k], off[k + 1])
            assert rel(h[s], h0[s]) < 1e-10 and rel(g[s], g0[s]) < 1e-8, k
        h, g = (np.asarray(v) for v in B.solve_grad_logk(cat("logK"), cat("dh"), cat("Qs"), obs))


def _mesh(kind):
    """(cells, faces, Dirichlet cells): a shuffled grid, a random tree, or pairs of cells beside a Dirichlet one
    (nothing to coarsen)."""
    rng = np.random.default_rng(len(kind))
    if kind.startswith("grid"):
        nx, ny = (7, 6) if kind == "grid42" else (23, 23) if kind == "grid529" else (70, 51)
        i = np.arange(nx * ny).reshape(nx, ny)
        nb = np.concatenate([np.stack([i[:-1].ravel(), i[1:].ravel()], 1), np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1)])
        return nx * ny, nb[rng.permutation(len(nb))], np.array([0, nx * ny - 1])
    if kind == "tree":
        k = np.arange(1, 900)
        return 900, np.stack([(rng.random(899) * k).astype(np.int64), k], 1), np.array([0, 17])
    k = np.arange(200)
    return 300, np.stack([k, 200 + k // 2], 1), np.arange(200, 300)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kind,degree", [("grid42", 0), ("grid529", 0), ("grid529", 1), ("grid3570", 2), ("grid3570", 4),
                                         ("tree", 0), ("pairs", 0)])
def test_face_lists(gpu_lib, orc, kind, degree, precision):
    n, nb, dn = _mesh(kind)
    rng = np.random.default_rng(5)
    aol, Ks = rng.uniform(0.5, 2.0, len(nb)), np.exp(-9.0 + rng.standard_normal(len(nb)))
    dh, Qs, delta = np.zeros(n), np.zeros(n), rng.standard_normal(n)
    dh[dn] = rng.uniform(0, 1, len(dn))
    Qs[rng.choice(np.setdiff1d(np.arange(n), dn), 3, replace=False)] = [1e-4, 5e-5, -2e-5]
    P = gpu_lib.GroundwaterProblem(nb, aol, dn, N=n, general=True, precision=precision, reltol=1e-12, cheb_degree=degree)
    O = orc.Problem(n, nb, aol, dn)
    want = (O.steady(Ks, dh, Qs, reltol=1e-14),) + tuple(O.adjoint(dh, delta, reltol=1e-14))
    got = (P.forward(Ks, dh, Qs),) + tuple(P.adjoint(delta))
    assert rel(got[0], want[0]) < 1e-8
    for g, w in zip(got[1:], want[1:]):
        assert rel(g, w) < 1e-6


def _launches(pkg, n, nb, dn, **opt):
    rng = np.random.default_rng(5)
    P = pkg.GroundwaterProblem(nb, rng.uniform(0.5, 2.0, len(nb)), dn, N=n, general=True, **opt)
    Qs = np.zeros(n)
    Qs[np.setdiff1d(np.arange(min(n, 1000)), dn)[3]] = 1e-4
    l0 = P.launch_count
    P.forward(np.exp(-9.0 + rng.standard_normal(len(nb))), np.zeros(n), Qs)
    launches = P.launch_count - l0
    P.close()
    return launches


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kind", ["grid42", "grid529", "grid3570", "tree", "pairs"])
def test_face_lists_take_one_launch(gpu_lib, kind, precision):
    """The meshes of the tests around this one are solved by the one-launch kernel."""
    n, nb, dn = _mesh(kind)
    one, many = (_launches(gpu_lib, n, nb, dn, precision=precision, reltol=1e-12, use_graphs=g) for g in (1, 0))
    assert one < many and one < 60


def test_large_mixed_face_list_takes_separate_launches(gpu_lib):
    """Above 5 Mi cells the separate kernels are the faster ones: the same launches as with the loop on the host."""
    nx, ny = 2300, 2290
    i = np.arange(nx * ny).reshape(nx, ny)
    nb = np.concatenate([np.stack([i[:-1].ravel(), i[1:].ravel()], 1), np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1)])
    opt = {"precision": "mixed", "maxiter": 2, "max_outer": 1}
    assert i.size > 5 << 20
    with pytest.warns(RuntimeWarning, match="did not reach its tolerance"):
        assert len({_launches(gpu_lib, i.size, nb, np.array([0, i.size - 1]), use_graphs=g, **opt) for g in (1, 0)}) == 1


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("degree", [1, 2, 3])
def test_face_lists_levels_of_both_kinds(gpu_lib, degree, precision):
    """90k cells: the finest level has more rows than half the threads of the GPU, the next ones fewer, the last ones
    run in one block. Against the separate launches; both stop at 1e-12 of the right-hand side."""
    i = np.arange(300 * 300).reshape(300, 300)
    nb = np.concatenate([np.stack([i[:-1].ravel(), i[1:].ravel()], 1), np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1)])
    n, rng = i.size, np.random.default_rng(2)
    aol, Ks = rng.uniform(0.5, 2.0, len(nb)), np.exp(-9.0 + rng.standard_normal(len(nb)))
    dn = np.concatenate([i[0], i[-1]])
    dh, Qs = np.zeros(n), np.zeros(n)
    dh[i[0]] = 1.0
    Qs[i[100, 100]] = 1e-4
    out = []
    for graphs in (1, 0):
        P = gpu_lib.GroundwaterProblem(nb, aol, dn, N=n, general=True, precision=precision, reltol=1e-12, cheb_degree=degree,
                                       use_graphs=graphs)
        out.append((P.forward(Ks, dh, Qs),) + tuple(P.adjoint(np.ones(n))))
    for got, want in zip(*out):
        assert rel(got, want) < 1e-8


@pytest.mark.parametrize("ns", [(1, 1, 2), (1, 1, 64), (1, 64, 1), (64, 1, 1), (7, 7, 1), (4, 4, 4), (2, 32, 1), (32, 1, 2), (3, 3, 7)])
def test_coarsest_inverse(gpu_lib, orc, ns):
    """Grids that are their own coarsest level: preconditioned with an exact inverse CG ends after one iteration, or two
    should rounding (n eps cond, below 1e-10 here) leave more than the 1e-12 asked for."""
    coords, nb, aol, _ = gpu_lib.regulargrid3d((0.0, 0.0, 0.0), (9.0, 8.0, 7.0), ns)
    n, rng = coords.shape[1], np.random.default_rng(4)
    Ks = np.exp(rng.standard_normal(len(nb)))
    dh, Qs = np.zeros(n), rng.standard_normal(n)
    dn = np.array([n // 2])
    Qs[dn] = 0.0
    P = gpu_lib.GroundwaterProblem.regular3d((0.0, 0.0, 0.0), (9.0, 8.0, 7.0), ns, dn, precision="fp64", reltol=1e-12)
    h = P.forward(Ks, dh, Qs)
    assert P.stats["iterations"] <= 2
    assert rel(h, orc.Problem(n, nb, aol, dn).steady(Ks, dh, Qs, reltol=1e-14)) < 1e-9
