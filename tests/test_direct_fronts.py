"""Which fronts the direct solver takes (host code, no GPU): a system that its band admits is never refused for the shape
of its nested dissection."""
import ctypes

import numpy as np
import pytest

REFUSED, DISSECTION, BAND = 0, 1, 2


def csr(n, nb):
    nb = np.unique(np.sort(nb[nb[:, 0] != nb[:, 1]], axis=1), axis=0)
    i = np.concatenate([nb[:, 0], nb[:, 1]])
    j = np.concatenate([nb[:, 1], nb[:, 0]])
    order = np.lexsort((j, i))
    return np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]).astype(np.int32), j[order].astype(np.int32)


def two_sets(a, share, seed=1):
    """2 a cells in two sets, couplings only between the sets (each with the given probability): no small separator."""
    m = np.random.default_rng(seed).random((a, a)) < share
    m[np.arange(a), np.arange(a)] = True
    i, j = np.nonzero(m)
    return 2 * a, np.stack([i, a + j], 1)


def grid(nx, ny):
    i = np.arange(nx * ny).reshape(nx, ny)
    return nx * ny, np.concatenate([np.stack([i[:-1].ravel(), i[1:].ravel()], 1), np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1)])


@pytest.fixture(scope="module")
def fronts(pkg):
    import __graft_entry__ as g
    g._load_build_module().build()
    lib = pkg.load()

    def ask(n, nb, free):
        rp, ci = csr(n, nb)
        form, rows, size = ctypes.c_int(-9), ctypes.c_int64(), ctypes.c_double()
        rc = lib.dpf_debug_direct_fronts(n, rp.ctypes.data, ci.ctypes.data, int(free), ctypes.byref(form), ctypes.byref(rows),
                                         ctypes.byref(size))
        return rc, form.value, rows.value, size.value
    return ask


def test_dissection_of_a_grid(fronts):
    rc, form, rows, size = fronts(*grid(300, 300), 64 << 30)
    assert (rc, form) == (0, DISSECTION) and rows < 600 and size < 0.3 * 8 * 90000 * 301


@pytest.mark.parametrize("a,share,free", [(200, 0.3, 3.2e6), (2000, 0.05, 4e8), (4000, 0.05, 5e9)])
def test_graph_without_small_separators(fronts, a, share, free):
    """The band fits half the memory given, the dissection's update matrices do not fit all of it."""
    n, nb = two_sets(a, share)
    rc, form, rows, size = fronts(n, nb, 1e12)
    assert (rc, form) == (0, DISSECTION) and size > free
    rc, form, rows, size = fronts(n, nb, free)
    assert (rc, form) == (0, BAND) and rows <= n and size <= 0.9 * free


@pytest.mark.parametrize("hub", [0, 1000])
def test_hub(fronts, hub):
    """A grid with a cell that is coupled to a thousand others (a well), beside enough memory for its band only just."""
    n, nb = grid(100, 100)
    far = np.random.default_rng(3).choice(n, hub, replace=False)
    nb = np.concatenate([nb, np.stack([np.full(hub, n), far], 1)]) if hub else nb
    for free in (64e9, 2.4e9):
        rc, form, rows, size = fronts(n + (hub > 0), nb, free)
        assert rc == 0 and form in (DISSECTION, BAND) and size <= 0.9 * free


def test_refused_and_malformed(fronts):
    n, nb = grid(300, 300)
    assert fronts(n, nb, 1e6)[:2] == (0, REFUSED)      # its band of 216 MB is above half of that
    assert fronts(n, nb, -1)[0] == 1                   # DPF_BAD_INPUT
    assert fronts(1, np.zeros((0, 2), np.int64), 1e9)[:2] == (0, DISSECTION)
