"""The work that users of the groundwater library have it do, as cases to be timed.

A case is a dict of plain values with a "kind":

* "dropin"    `groundwater_steadystate` on host arrays, as the reference's callers use it
* "steady"    forward and pullback from face conductances on one handle (`forward`, `adjoint`)
* "grad"      `solve_grad_logk`: heads and d/dlogK of many realizations in one batch
* "transient" backward Euler and its checkpointed adjoint
* "mesh"      `solve_grad_logk` on a fracture network's face list (no regular grid)
* "richards"  steady Richards and its pullback
* "direct"    forward and pullback with the direct solver (the reference's cholesky_solver)
* "faces"     face conductances from logK and their pullback

Arrays live on the GPU except in "dropin". `exact` restates each path in plain torch with 64-bit numbers.
"""
import functools
import math

import numpy as np
import torch

import __graft_entry__ as entry

PKG = entry.load_package()
F64 = torch.float64


# ------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # a small 3-D model (a laptop-sized example) called as DPFEHM's own callers do: host arrays in, heads out
        {"name": "dropin_6k", "kind": "dropin", "nx": 31, "ny": 29, "nz": 7, "tol": 1e-12},
        # one model of 50x50x5 cells, default (FP64) options, forward and pullback: latency and launches count
        {"name": "steady_12k_fp64", "kind": "steady", "nx": 50, "ny": 50, "nz": 5, "prec": "fp64", "tol": 1e-12},
        # the reference's 3-D steady-state example (100x100x10), default options
        {"name": "steady_100k_fp64", "kind": "steady", "nx": 100, "ny": 100, "nz": 10, "prec": "fp64", "tol": 1e-12},
        # one 1M-cell realization with default options: heads and the gradient of an objective at 100 cells
        {"name": "grad_1m_fp64", "kind": "grad", "sizes": "200x200x25", "batch": 1, "sigma": 2.0, "prec": "fp64",
         "mean": "geometric", "streams": 0, "tol": 1e-12},
        # an ensemble of 64 realizations of the 100x100x10 model in mixed precision
        {"name": "grad_100k_x64_mixed", "kind": "grad", "sizes": "100x100x10", "batch": 64, "sigma": 1.0,
         "prec": "mixed", "mean": "geometric", "streams": 0, "tol": 1e-10},
        # models of uneven size (one of them odd) in one batch, harmonic face means
        {"name": "grad_uneven_x24_mixed", "kind": "grad", "sizes": "50x50x5,100x100x10,151x149x11,200x200x20",
         "batch": 24, "sigma": 1.3, "prec": "mixed", "mean": "harmonic", "streams": 0, "tol": 1e-10},
        # the benchmark's ensemble: 32 realizations of 1M cells, as two concurrent parts
        {"name": "grad_1m_x32_mixed", "kind": "grad", "sizes": "200x200x25", "batch": 32, "sigma": 2.0,
         "prec": "mixed", "mean": "geometric", "streams": 2, "tol": 1e-10},
        # a transient calibration pass: 20 steps on 800k cells, heads kept every 5th step, and the adjoint
        {"name": "transient_800k_mixed", "kind": "transient", "nx": 200, "ny": 200, "nz": 20, "nsteps": 20,
         "every": 5, "prec": "mixed", "tol": 1e-12},
        # a fracture network of about 815k cells read as a face list
        {"name": "mesh_815k_mixed", "kind": "mesh", "nfrac": 2000, "h": 0.5, "prec": "mixed", "tol": 1e-12},
        # an unsaturated column of 200k cells (steady Richards and its pullback), default options
        {"name": "richards_200k_fp64", "kind": "richards", "nx": 100, "ny": 100, "nz": 20, "prec": "fp64",
         "tol": 1e-12},
        # the direct solver on a 2-D grid of 500x500 cells
        {"name": "direct_500x500", "kind": "direct", "nx": 500, "ny": 500, "nz": 1},
        # the caller's conductance step on 8 realizations of 1M cells, and its pullback
        {"name": "faces_1m_x8", "kind": "faces", "nx": 200, "ny": 200, "nz": 25, "batch": 8, "mean": "geometric"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, lo, hi):
    """A flat 3-D grid of lo..hi cells (log-uniform): nz of 3..25 layers, nx and ny within a factor of 1.5."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    nz = rng.randint(3, 25)
    side = math.sqrt(n / nz)
    r = rng.uniform(0.8, 1.25)
    return max(4, int(side * r)), max(4, int(side / r)), nz


def draw(rng):
    kind = rng.choice(["dropin", "steady", "steady", "grad", "grad", "grad", "transient", "mesh", "richards",
                       "direct", "faces"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "dropin":
        nx, ny, nz = _shape(rng, 1000, 100000)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "tol": 1e-12}
    if kind == "steady":
        nx, ny, nz = _shape(rng, 3000, 1000000)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "prec": prec, "tol": 1e-12 if prec == "fp64" else 1e-10}
    if kind == "grad":
        shapes = [_shape(rng, 10000, 1000000) for _ in range(rng.choice([1, 1, 3]))]
        cells = sum(a * b * c for a, b, c in shapes) / len(shapes)
        batch = _log_int(rng, 1, max(1.0, min(64.0, (4e6 if prec == "fp64" else 24e6) / cells)))
        batch = max(batch, len(shapes))
        return {"kind": kind, "sizes": ",".join("%dx%dx%d" % s for s in shapes), "batch": batch,
                "sigma": round(rng.uniform(0.5, 2.0), 2), "prec": prec, "mean": rng.choice(["geometric", "harmonic"]),
                "streams": rng.choice([0, 0, 2]) if batch >= 4 else 0, "tol": 1e-12 if prec == "fp64" else 1e-10}
    if kind == "transient":
        nx, ny, nz = _shape(rng, 10000, 800000)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "nsteps": rng.randint(5, 20), "every": rng.randint(1, 6),
                "prec": prec, "tol": 1e-12}
    if kind == "mesh":
        return {"kind": kind, "nfrac": rng.randint(500, 1500), "h": round(rng.uniform(0.6, 1.5), 2), "prec": prec,
                "tol": 1e-12}
    if kind == "richards":
        nx, ny, nz = _shape(rng, 4000, 200000)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "prec": prec, "tol": 1e-12}
    if kind == "direct":
        if rng.random() < 0.5:
            return {"kind": kind, "nx": _log_int(rng, 20, 500), "ny": _log_int(rng, 20, 500), "nz": 1}
        return {"kind": kind, "nx": rng.randint(8, 36), "ny": rng.randint(8, 36), "nz": rng.randint(4, 36)}
    nx, ny, nz = _shape(rng, 10000, 1000000)
    return {"kind": "faces", "nx": nx, "ny": ny, "nz": nz, "batch": _log_int(rng, 1, 8),
            "mean": rng.choice(["geometric", "harmonic"])}


def _grids(case):
    shapes = [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split(",")]
    return [shapes[p % len(shapes)] for p in range(case["batch"])]


def _ns(case):
    return case["nx"], case["ny"], case["nz"]


def _extent(ns, spacing=0.5):
    return tuple(spacing * max(n - 1, 1) for n in ns)


def _nfaces(ns):
    nx, ny, nz = ns
    return 3 * nx * ny * nz - nx * ny - nx * nz - ny * nz


def work(case):
    """Inputs read once and outputs written once; operations only where a count is inherent to the method."""
    k = case["kind"]
    if k == "grad":
        n = sum(a * b * c for a, b, c in _grids(case))
        return {"bytes": 8.0 * 5 * n, "flops": 0.0}          # logK, dh, Q in; h, g out
    if k == "mesh":
        n = 90.0 * case["nfrac"] / case["h"] ** 2            # about this many cells
        return {"bytes": 8.0 * 5 * n, "flops": 0.0}
    ns = _ns(case)
    n, f = ns[0] * ns[1] * ns[2], _nfaces(ns)
    if k == "dropin":
        return {"bytes": 8.0 * (f + 3 * n), "flops": 0.0}    # Ks, dh, Q in; h out
    if k == "faces":
        return {"bytes": 8.0 * case["batch"] * (3 * n + 2 * f), "flops": 0.0}
    if k == "transient":
        return {"bytes": 8.0 * (2 * f + 8 * n), "flops": 0.0}
    if k == "richards":
        return {"bytes": 8.0 * (6 * f + 8 * n), "flops": 0.0}
    return {"bytes": 8.0 * (2 * f + 6 * n), "flops": 0.0}    # steady, direct: Ks, dh, Q, delta in; h and tangents out


# ------------------------------------------------------------------------------------------ inputs
def _dev():
    return torch.device("cuda")


def _field(ns, mins, maxs, ell, sigma, seed):
    """A seeded Matern log-conductivity field with mean -9 (flat, z fastest), on the GPU."""
    return PKG.fields.volume_logk_torch(ns, mins, maxs, ell, sigma, -9.0, seed, device=_dev())


@functools.lru_cache(maxsize=4)
def _faces(ns):
    """(a, b, direction) of the faces of a regular grid in the reference's order: per cell +x, +y, +z where in range."""
    nx, ny, nz = ns
    i = np.arange(nx * ny * nz)
    iz, iy, ix = i % nz, i // nz % ny, i // (nz * ny)
    ok = np.stack([ix < nx - 1, iy < ny - 1, iz < nz - 1], axis=1)
    b = np.stack([i + ny * nz, i + nz, i + 1], axis=1)
    a = np.repeat(i[:, None], 3, axis=1)
    d = np.broadcast_to(np.arange(3), ok.shape)
    return a[ok], b[ok], d[ok]


def _gpu(x):
    return torch.as_tensor(x, device=_dev())


def _aol(ns, maxs):
    d = [maxs[k] / (ns[k] - 1) if ns[k] > 1 else 1.0 for k in range(3)]
    return d[1] * d[2] / d[0], d[0] * d[2] / d[1], d[0] * d[1] / d[2]


def _sources(n, rng, count):
    q = np.zeros(n)
    q[rng.choice(n, count, replace=False)] = rng.uniform(1e-5, 1e-4, count)
    return q


def _steady_inputs(case, seed):
    """Grid, Dirichlet cells, face conductances, heads, sources and cotangent of one regular grid."""
    ns = _ns(case)
    n, maxs = ns[0] * ns[1] * ns[2], _extent(ns)
    rng = np.random.default_rng([seed, n])
    if case["kind"] == "direct":  # the reference's comparison: heads held at 1 and 0 on two opposite faces
        face = ns[1] * ns[2]
        dn = np.concatenate([np.arange(face), np.arange(n - face, n)])
        dh = np.zeros(n)
        dh[:face] = 1.0
    else:
        dn = np.sort(rng.choice(n, 4, replace=False))
        dh = np.zeros(n)
        dh[dn] = rng.uniform(0.0, 1.0, 4)
    q = _sources(n, rng, 3)
    q[dn] = 0.0
    delta = np.zeros(n)
    delta[rng.choice(n, min(100, n // 4), replace=False)] = rng.standard_normal(min(100, n // 4))
    logk = _field(ns, (0.0, 0.0, 0.0), maxs, 0.3 * max(maxs), 1.0, seed)
    a, b, d = _faces(ns)
    ks = torch.exp(0.5 * (logk[_gpu(a)] + logk[_gpu(b)]))
    return {"ns": ns, "n": n, "maxs": maxs, "dn": dn, "dh": _gpu(dh), "Q": _gpu(q), "delta": _gpu(delta), "Ks": ks}


def _grad_inputs(case, seed):
    grids = _grids(case)
    rng = np.random.default_rng([seed, len(grids)])
    out = {"grids": grids, "maxs": [_extent(g) for g in grids], "dn": [], "obs": [], "logK": [], "dh": [], "Q": []}
    for p, g in enumerate(grids):
        n = g[0] * g[1] * g[2]
        if case["sigma"] == 2.0:  # the benchmark's problem: one source in the first cell, head 0 in the last
            dn, q = np.array([n - 1]), np.zeros(n)
            q[0] = 1e-4
        else:
            dn = np.sort(rng.choice(n, 1 + int(rng.integers(4)), replace=False))
            q = _sources(n, rng, 1 + int(rng.integers(4)))
        mx = out["maxs"][p]
        out["dn"].append(dn)
        out["obs"].append(rng.choice(n, 100, replace=False))
        out["logK"].append(_field(g, (0.0, 0.0, 0.0), mx, 0.2 * max(mx), case["sigma"], 1000 * seed + p))
        out["dh"].append(torch.zeros(n, dtype=F64, device=_dev()))
        out["Q"].append(_gpu(q))
    return out


def _transient_inputs(case, seed):
    ns = _ns(case)
    n, maxs = ns[0] * ns[1] * ns[2], _extent(ns)
    rng = np.random.default_rng([seed, n])
    face = ns[1] * ns[2]
    free = n - face
    q = np.zeros(n)
    q[rng.choice(free, 4, replace=False)] = 1e-3
    logk = _field(ns, (0.0, 0.0, 0.0), maxs, 0.3 * max(maxs), 1.5, seed)
    a, b, d = _faces(ns)
    return {"ns": ns, "n": n, "maxs": maxs, "dn": np.arange(free, n), "obs": rng.choice(free, 50, replace=False),
            "Q": _gpu(q), "Ks": torch.exp(0.5 * (logk[_gpu(a)] + logk[_gpu(b)])),
            "zero": torch.zeros(n, dtype=F64, device=_dev()), "Ss": torch.full((n,), 1e-5, dtype=F64, device=_dev()),
            "w": _gpu(rng.uniform(0.5, 1.5, 50)), "dt": 3600.0}


@functools.lru_cache(maxsize=2)
def _network(nfrac, h):
    c, vol, nb, areas, lengths, fr = PKG.grid.fracture_network(nfrac, 100.0, h, 3, smin=4.0)
    return c, vol, nb, areas / lengths, fr


def _mesh_inputs(case, seed):
    c, vol, nb, aol, fr = _network(case["nfrac"], case["h"])
    n, x = c.shape[1], c[0]
    rng = np.random.default_rng([seed, n])
    dn = np.nonzero((x < 5.0) | (x > 95.0))[0]
    dh = np.where(x < 5.0, 1.0, 0.0)
    q = np.zeros(n)
    q[rng.choice(np.nonzero((x > 30) & (x < 70))[0], 2, replace=False)] = 1e-6
    logk = rng.normal(-9.0, 1.0, int(fr.max()) + 1)[fr]
    return {"n": n, "nb": nb, "aol": aol, "vol": vol, "dn": dn, "dh": _gpu(dh), "Q": _gpu(q), "logK": _gpu(logk),
            "obs": rng.choice(np.setdiff1d(np.arange(n), dn), 100, replace=False)}


def _richards_inputs(case, seed):
    ns = _ns(case)
    n, maxs = ns[0] * ns[1] * ns[2], _extent(ns)
    rng = np.random.default_rng([seed, n])
    a, b, d = _faces(ns)
    f = len(a)
    iz = np.arange(n) % ns[2]
    dn = np.nonzero(iz == ns[2] - 1)[0]  # the top layer, held at psi = -2 m
    dpsi = np.where(iz == ns[2] - 1, -2.0, 0.0)
    logk = _field(ns, (0.0, 0.0, 0.0), maxs, 0.3 * max(maxs), 1.0, seed)
    q = np.zeros(n)
    q[0] = 1e-6
    delta = np.zeros(n)
    delta[rng.choice(n - len(dn), 100, replace=True)] = rng.standard_normal(100)
    delta[dn] = 0.0
    return {"ns": ns, "n": n, "maxs": maxs, "dn": dn, "psi0": torch.full((n,), -2.0, dtype=F64, device=_dev()),
            "Ks": torch.exp(0.5 * (logk[_gpu(a)] + logk[_gpu(b)])), "dpsi": _gpu(dpsi),
            "z": _gpu(iz * (maxs[2] / max(ns[2] - 1, 1))), "al": _gpu(0.375 * np.exp(0.1 * rng.standard_normal(f))),
            "N": _gpu(1.25 + 0.05 * rng.uniform(0, 1, f)), "Q": _gpu(q), "delta": _gpu(delta)}


def _faces_inputs(case, seed):
    ns, nb = _ns(case), case["batch"]
    maxs = _extent(ns)
    g = torch.Generator(device=_dev())
    g.manual_seed(seed)
    lk = torch.cat([_field(ns, (0.0, 0.0, 0.0), maxs, 0.2 * max(maxs), 1.0, 1000 * seed + p) for p in range(nb)])
    return {"ns": ns, "maxs": maxs, "batch": nb, "logK": lk,
            "dKs": torch.randn(nb * _nfaces(ns), dtype=F64, device=_dev(), generator=g)}


def prepare(case, seed):
    kind, o = case["kind"], (0.0, 0.0, 0.0)
    if kind == "dropin":
        s = _steady_inputs(case, seed)
        a, b, d = _faces(s["ns"])
        s["nb"] = np.stack([a, b], axis=1)
        s["aol"] = np.array(_aol(s["ns"], s["maxs"]))[d]
        for k in ("Ks", "dh", "Q"):
            s[k] = s[k].cpu().numpy()
        s.update(kind=kind, tol=case["tol"])
        return s
    if kind in ("steady", "direct"):
        s = _steady_inputs(case, seed)
        opt = {"solver": "cholesky", "precision": "fp64"} if kind == "direct" else {"precision": case["prec"],
                                                                                 "reltol": case["tol"]}
        s["P"] = PKG.GroundwaterProblem.regular3d(o, s["maxs"], s["ns"], s["dn"], **opt)
    elif kind == "grad":
        s = _grad_inputs(case, seed)
        for k in ("logK", "dh", "Q"):
            s[k] = torch.cat(s[k])
        s["P"] = PKG.GroundwaterBatch(s["grids"], [o] * len(s["grids"]), s["maxs"], s["dn"], precision=case["prec"],
                                      reltol=case["tol"], streams=case["streams"])
        s["mean"] = case["mean"]
    elif kind == "transient":
        s = _transient_inputs(case, seed)
        s["P"] = PKG.GroundwaterProblem.regular3d(o, s["maxs"], s["ns"], s["dn"], precision=case["prec"],
                                                  reltol=case["tol"])
        s.update(nsteps=case["nsteps"], every=case["every"])
    elif kind == "mesh":
        s = _mesh_inputs(case, seed)
        s["P"] = PKG.GroundwaterProblem(s["nb"], s["aol"], s["dn"], N=s["n"], volumes=s["vol"], reltol=case["tol"],
                                        precision=case["prec"], coarse_scale=2.0)
    elif kind == "richards":
        s = _richards_inputs(case, seed)
        a, b, d = _faces(s["ns"])
        s["P"] = PKG.GroundwaterProblem(np.stack([a, b], axis=1), np.array(_aol(s["ns"], s["maxs"]))[d], s["dn"],
                                        N=s["n"], general=True, reltol=case["tol"], precision=case["prec"])
        s["tol"] = case["tol"]
    else:
        s = _faces_inputs(case, seed)
        n = s["ns"][0] * s["ns"][1] * s["ns"][2]
        s["P"] = PKG.GroundwaterBatch([s["ns"]] * s["batch"], [o] * s["batch"], [s["maxs"]] * s["batch"],
                                      [[n - 1]] * s["batch"])
        s["mean"] = case["mean"]
    s["kind"] = kind
    return s


# ------------------------------------------------------------------------------------------ one pass
def run(s):
    kind, P = s["kind"], s.get("P")
    if kind == "dropin":
        return PKG.groundwater_steadystate(s["Ks"], s["nb"], s["aol"], s["dn"], s["dh"], s["Q"], reltol=s["tol"])
    if kind in ("steady", "direct"):
        h = P.forward(s["Ks"], s["dh"], s["Q"])
        return (h,) + tuple(P.adjoint(s["delta"]))
    if kind == "grad":
        return P.solve_grad_logk(s["logK"], s["dh"], s["Q"], s["obs"], mean=s["mean"])
    if kind == "transient":
        h = P.transient_forward(s["Ks"], s["zero"], s["Q"], s["Ss"], s["dt"], s["nsteps"], s["zero"],
                                checkpoint_every=s["every"])
        return (h,) + tuple(P.transient_adjoint(s["obs"], weights=s["w"]))
    if kind == "mesh":
        return P.solve_grad_logk(s["logK"], s["dh"], s["Q"], s["obs"])
    if kind == "richards":
        psi = P.richards_steady(s["psi0"], s["Ks"], s["dpsi"], s["z"], s["al"], s["N"], s["Q"], s["tol"], 300)
        return (psi,) + tuple(P.richards_adjoint(s["delta"], s["tol"], 300))
    return P.logk_to_faces(s["logK"], s["mean"]), P.logk_to_faces_vjp(s["logK"], s["dKs"], s["mean"])


# ------------------------------------------------------------------------------- the same in plain torch
class _Grid:
    """Flux-form operators of B regular grids of one size and their solution by conjugate gradients with a
    multigrid preconditioner (2x2x2 aggregates, damped Jacobi), all in 64 bits: A x = leak x + sum c (x - x_nb)
    over free cells, the identity on Dirichlet cells. Tensors are (B, nx, ny, nz)."""

    def __init__(self, c, leak, fixed):
        free = ~fixed
        c = [ci * (a & b) for ci, (a, b) in zip(c, _pairs(free))]
        self.free = free
        self.lv = []
        leak = torch.where(free, leak, torch.zeros_like(leak))
        while True:
            dg = leak.clone()
            for ci, (lo, hi) in zip(c, _pairs(dg)):
                lo += ci
                hi += ci
            inv = torch.where(dg > 0, 1.0 / torch.where(dg > 0, dg, torch.ones_like(dg)), torch.zeros_like(dg))
            self.lv.append((c, leak, inv))
            if leak[0].numel() <= 64:
                break
            c, leak = _coarsen(c, leak)
        c, leak, inv = self.lv[-1]
        n = leak[0].numel()
        eye = torch.eye(n, dtype=F64, device=leak.device).reshape((n, 1) + leak.shape[1:])
        A = _apply(c, leak, eye.expand((n,) + leak.shape)).reshape(n, leak.shape[0], n).permute(1, 2, 0)
        A = A + torch.diag_embed((inv.reshape(leak.shape[0], n) == 0).to(F64))
        self.inv = torch.linalg.inv(A)

    def _cycle(self, l, r):
        c, leak, inv = self.lv[l]
        if l == len(self.lv) - 1:
            return torch.einsum("bij,bj->bi", self.inv, r.reshape(r.shape[0], -1)).reshape(r.shape)
        x = 0.7 * inv * r
        x = x + 0.7 * inv * (r - _apply(c, leak, x))
        e = self._cycle(l + 1, _sum2(r - _apply(c, leak, x)))
        x = x + 1.8 * _spread2(e, x.shape) * (inv > 0)  # identity rows stay 0
        for _ in range(2):
            x = x + 0.7 * inv * (r - _apply(c, leak, x))
        return x

    def precondition(self, r):
        return self._cycle(0, r)

    def solve(self, b, x=None):
        """x with A x = b on the free cells (0 on the others), to the rounding floor of b - A x."""
        c, leak, _ = self.lv[0]
        dot = lambda u, v: (u * v).flatten(1).sum(1)[:, None, None, None]  # noqa: E731
        b = torch.where(self.free, b, torch.zeros_like(b))
        x = torch.zeros_like(b) if x is None else x.clone()
        best = None
        for _ in range(4):  # each round starts from the true residual
            r = b - _apply(c, leak, x)
            rr = dot(r, r)
            if best is not None and bool((rr > 0.25 * best).all()):
                break
            best = rr
            p, rz_old, r_old, small, k = None, None, None, rr, 0
            for _ in range(400):
                z = self._cycle(0, r)
                rz = dot(r, z)
                if p is None:
                    p = z
                else:  # the flexible form: the preconditioner need not be exactly symmetric
                    p = z + (rz - dot(r_old, z)) / torch.where(rz_old == 0, torch.ones_like(rz_old), rz_old) * p
                q = _apply(c, leak, p)
                pq = dot(p, q)
                al = torch.where(pq > 0, rz / torch.where(pq > 0, pq, torch.ones_like(pq)), torch.zeros_like(pq))
                x = x + al * p
                r_old, rz_old = r, rz
                r = r - al * q
                rr = dot(r, r)
                if bool((rr <= 1e-30 * dot(b, b)).all()):
                    break
                k = 0 if bool((rr < 0.5 * small).any()) else k + 1
                small = torch.minimum(small, rr)
                if k > 25:
                    break
        return x


def _pairs(x):
    return [(x[..., :-1, :, :], x[..., 1:, :, :]), (x[..., :-1, :], x[..., 1:, :]), (x[..., :-1], x[..., 1:])]


def _apply(c, leak, x):
    y = leak * x
    for ci, (xa, xb), (ya, yb) in zip(c, _pairs(x), _pairs(y)):
        f = ci * (xa - xb)
        ya += f
        yb -= f
    return y


def _sum2(x, axes=(-3, -2, -1)):
    for ax in axes:
        n = x.shape[ax]
        if n % 2 and n > 1:
            shape = list(x.shape)
            shape[ax] = 1
            x = torch.cat([x, x.new_zeros(shape)], ax)
        if n > 1:
            x = x.unflatten(ax % x.dim(), ((n + 1) // 2, 2)).sum((ax % x.dim()) + 1)
    return x


def _spread2(e, shape):
    for ax in (-3, -2, -1):
        if shape[ax] > 1:
            e = e.repeat_interleave(2, ax % e.dim()).narrow(ax % e.dim(), 0, shape[ax])
    return e


def _coarsen(c, leak):
    out = []
    for k, ci in enumerate(c):
        ax = k - 3
        n = leak.shape[ax]
        keep = ci.index_select(ax % ci.dim(), torch.arange(1, max(n - 1, 1), 2, device=ci.device)) if n > 1 else ci
        out.append(_sum2(keep, [a for a in (-3, -2, -1) if a != ax]))
    return out, _sum2(leak)


def _split_faces(ns, v):
    """A face list's values as the three directions' tensors (nx-1, ny, nz), (nx, ny-1, nz), (nx, ny, nz-1)."""
    nx, ny, nz = ns
    d = _gpu(_faces(ns)[2])
    return [v[d == 0].reshape(nx - 1, ny, nz), v[d == 1].reshape(nx, ny - 1, nz), v[d == 2].reshape(nx, ny, nz - 1)]


def _join_faces(ns, parts):
    d = _gpu(_faces(ns)[2])
    out = torch.empty(d.numel(), dtype=F64, device=_dev())
    for k in range(3):
        out[d == k] = parts[k].reshape(-1)
    return out


class _Steady:
    """The steady (or shifted) problem on B equal grids from the three directions' conductances K, (B, ...)."""

    def __init__(self, ns, maxs, K, dn, shift=None):
        self.ns, self.aol = ns, _aol(ns, maxs)
        B = K[0].shape[0]
        fixed = torch.zeros((B,) + tuple(ns), dtype=torch.bool, device=_dev())
        for p in range(B):
            fixed[p].view(-1)[_gpu(np.asarray(dn[p]))] = True
        self.fixed = fixed
        self.c = [K[k] * self.aol[k] for k in range(3)]
        self.leak = torch.zeros(fixed.shape, dtype=F64, device=_dev())
        for ci, (fa, fb), (la, lb) in zip(self.c, _pairs(fixed), _pairs(self.leak)):
            la += ci * fb
            lb += ci * fa
        if shift is not None:
            self.leak = self.leak + shift
        self.grid = _Grid(self.c, self.leak, fixed)

    def rhs(self, dh, Q):
        """Q plus the flow from Dirichlet neighbours, at free cells."""
        g = torch.where(self.fixed, dh, torch.zeros_like(dh))
        b = Q.clone()
        for ci, (ga, gb), (ba, bb) in zip(self.c, _pairs(g), _pairs(b)):
            ba += ci * gb
            bb += ci * ga
        return b

    def forward(self, dh, Q):
        return torch.where(self.fixed, dh, self.grid.solve(self.rhs(dh, Q)))

    def tangents(self, h, lam):
        """(dKs per direction, ddirichleths without delta, dQs) for the adjoint solution lam (0 at Dirichlet cells)."""
        dK = [-a * (ha - hb) * (la - lb) for a, (ha, hb), (la, lb) in zip(self.aol, _pairs(h), _pairs(lam))]
        ddh = torch.zeros_like(h)
        for ci, (la, lb), (da, db) in zip(self.c, _pairs(lam), _pairs(ddh)):
            da += ci * lb
            db += ci * la
        return dK, torch.where(self.fixed, ddh, torch.zeros_like(ddh)), lam


def _exact_steady(case, seed):
    s = _steady_inputs(case, seed)
    ns = s["ns"]
    sh = (1,) + tuple(ns)
    S = _Steady(ns, s["maxs"], [k[None] for k in _split_faces(ns, s["Ks"])], [s["dn"]])
    h = S.forward(s["dh"].reshape(sh), s["Q"].reshape(sh))
    if case["kind"] == "dropin":
        return h.reshape(-1)
    delta = s["delta"].reshape(sh)
    dK, ddh, dQ = S.tangents(h, S.grid.solve(delta))
    ddh = torch.where(S.fixed, ddh + delta, ddh)
    return h.reshape(-1), _join_faces(ns, [k[0] for k in dK]), ddh.reshape(-1), dQ.reshape(-1)


def _mean_faces(kc, mean):
    """Face conductances from logK and their derivatives by the logK of either end, per direction."""
    out = []
    for a, b in _pairs(kc):
        if mean == "geometric":
            K = torch.exp(0.5 * (a + b))
            out.append((K, 0.5 * K, 0.5 * K))
        else:
            ea, eb = torch.exp(a), torch.exp(b)
            K = 2.0 * ea * eb / (ea + eb)
            out.append((K, 0.5 * K * K / ea, 0.5 * K * K / eb))
    return out


def _exact_grad(case, seed):
    s = _grad_inputs(case, seed)
    hs, gs = [None] * len(s["grids"]), [None] * len(s["grids"])
    for ns in sorted(set(s["grids"])):
        every = [p for p, g in enumerate(s["grids"]) if g == ns]
        step = max(1, int(4e6 // (ns[0] * ns[1] * ns[2])))
        for at in range(0, len(every), step):
            ps = every[at:at + step]
            lk = torch.stack([s["logK"][p].reshape(ns) for p in ps])
            K = _mean_faces(lk, case["mean"])
            S = _Steady(ns, s["maxs"][ps[0]], [k[0] for k in K], [s["dn"][p] for p in ps])
            h = S.forward(torch.stack([s["dh"][p].reshape(ns) for p in ps]),
                          torch.stack([s["Q"][p].reshape(ns) for p in ps]))
            delta = torch.zeros_like(h)
            for k, p in enumerate(ps):
                o = _gpu(s["obs"][p])
                delta[k].view(-1)[o] = 2.0 * h[k].reshape(-1)[o]
            dK, _, _ = S.tangents(h, S.grid.solve(delta))
            g = torch.zeros_like(h)
            for dk, (_, ka, kb), (ga, gb) in zip(dK, K, _pairs(g)):
                ga += ka * dk
                gb += kb * dk
            for k, p in enumerate(ps):
                hs[p], gs[p] = h[k].reshape(-1), g[k].reshape(-1)
    return torch.cat(hs), torch.cat(gs)


def _exact_transient(case, seed):
    s = _transient_inputs(case, seed)
    ns, T = s["ns"], case["nsteps"]
    sh = (1,) + tuple(ns)
    d = [s["maxs"][k] / (ns[k] - 1) for k in range(3)]
    shift = s["Ss"].reshape(sh) * (d[0] * d[1] * d[2]) / s["dt"]
    S = _Steady(ns, s["maxs"], [k[None] for k in _split_faces(ns, s["Ks"])], [s["dn"]], shift=shift)
    zero = s["zero"].reshape(sh)
    b = S.rhs(zero, s["Q"].reshape(sh))
    h, states = zero, []
    for _ in range(T):
        h = S.grid.solve(b + shift * h, h)  # the Dirichlet heads are 0
        states.append(h)
    obs = _gpu(s["obs"])
    mu = torch.zeros_like(h)
    dK, ddh, dQ = None, torch.zeros_like(h), torch.zeros_like(h)
    for t in range(T - 1, -1, -1):
        r = shift * mu
        r.view(-1).index_add_(0, obs, 2.0 * s["w"] * states[t].reshape(-1)[obs])
        mu = S.grid.solve(r, mu)
        k, dd, q = S.tangents(states[t], mu)
        dK = k if dK is None else [u + v for u, v in zip(dK, k)]
        ddh, dQ = ddh + dd, dQ + q
    dh0 = torch.where(S.fixed, zero, shift * mu)
    return (h.reshape(-1), _join_faces(ns, [k[0] for k in dK]), ddh.reshape(-1), dQ.reshape(-1), dh0.reshape(-1))


def _exact_mesh(case, seed):
    """Conjugate gradients with the diagonal as preconditioner on the face list."""
    s = _mesh_inputs(case, seed)
    n = s["n"]
    a, b = _gpu(s["nb"][:, 0].copy()), _gpu(s["nb"][:, 1].copy())
    K = torch.exp(0.5 * (s["logK"][a] + s["logK"][b]))
    aol = _gpu(s["aol"])
    c = K * aol
    fixed = torch.zeros(n, dtype=torch.bool, device=_dev())
    fixed[_gpu(s["dn"])] = True
    both = ~fixed[a] & ~fixed[b]
    fa, fb, fc = a[both], b[both], c[both]
    g = torch.where(fixed, s["dh"], torch.zeros_like(s["dh"]))
    leak, rhs = torch.zeros(n, dtype=F64, device=_dev()), s["Q"].clone()
    for i, j in ((a, b), (b, a)):
        on = ~fixed[i] & fixed[j]
        leak.index_add_(0, i[on], c[on])
        rhs.index_add_(0, i[on], c[on] * g[j[on]])
    dg = leak.clone().index_add_(0, fa, fc).index_add_(0, fb, fc)
    inv = torch.where(fixed, torch.zeros_like(dg), 1.0 / torch.where(dg > 0, dg, torch.ones_like(dg)))

    # rows of the coupling matrix, so that a product is a gather and a segment sum in a fixed order
    order = torch.argsort(torch.cat([fa, fb]), stable=True)
    col = torch.cat([fb, fa])[order]
    row = torch.cat([fa, fb])[order]
    val = torch.cat([fc, fc])[order]
    length = torch.bincount(row, minlength=n)

    def apply(x):
        return leak * x + torch.segment_reduce(val * (x[row] - x[col]), "sum", lengths=length, initial=0.0)

    def solve(b0):
        b0 = torch.where(fixed, torch.zeros_like(b0), b0)
        x, best = torch.zeros_like(b0), None
        for _ in range(4):
            r = b0 - apply(x)
            rr = float(r @ r)
            if best is not None and rr > 0.25 * best:
                break
            best = rr
            z = inv * r
            p, rz = z, r @ z
            floor, stuck = rr, 0
            for it in range(20000):
                q = apply(p)
                al = rz / (p @ q)
                x = x + al * p
                r = r - al * q
                z = inv * r
                new = r @ z
                p, rz = z + new / rz * p, new
                if it % 100 == 99:
                    rr = float(r @ r)
                    if rr <= 1e-29 * float(b0 @ b0):
                        break
                    stuck = 0 if rr < 0.5 * floor else stuck + 1
                    floor = min(floor, rr)
                    if stuck > 10:
                        break
        return x

    h = torch.where(fixed, s["dh"], solve(rhs))
    delta = torch.zeros_like(h)
    o = _gpu(s["obs"])
    delta[o] = 2.0 * h[o]
    lam = solve(delta)
    w = -aol * (h[a] - h[b]) * (lam[a] - lam[b]) * 0.5 * K
    return h, torch.zeros_like(h).index_add_(0, a, w).index_add_(0, b, w)


def _kr(psi, al, N):
    """van Genuchten relative permeability and its derivatives by psi, alpha and N."""
    dry = psi < 0
    p = torch.where(dry, psi, torch.full_like(psi, -1.0))
    m, u = (N - 1.0) / N, al * -p
    lu = torch.log(u)
    A = 1.0 + u ** N
    lA = torch.log(A)
    w = u ** (N - 1.0) * A ** -m
    num, h = 1.0 - w, A ** (-0.5 * m)
    dA = N * u ** (N - 1.0)                     # by u
    dw = w * ((N - 1.0) / u - m * dA / A)
    du = -2.0 * num * dw * h - 0.5 * m * num * num * h / A * dA
    dm, dAN = 1.0 / (N * N), u ** N * lu        # by N
    dwN = w * (lu - dm * lA - m * dAN / A)
    dN = -2.0 * num * dwN * h + num * num * h * (-0.5 * dm * lA - 0.5 * m * dAN / A)
    one, zero = torch.ones_like(psi), torch.zeros_like(psi)
    return (torch.where(dry, num * num * h, one), torch.where(dry, -al * du, zero),
            torch.where(dry, -p * du, zero), torch.where(dry, dN, zero))


def _exact_richards(case, seed):
    """Picard steps to the root, then the transposed Jacobian by GMRES with the Picard operator's multigrid cycle."""
    s = _richards_inputs(case, seed)
    ns = s["ns"]
    sh = (1,) + tuple(ns)
    al, N, Ks = ([v[None] for v in _split_faces(ns, s[k])] for k in ("al", "N", "Ks"))
    z, Q = s["z"].reshape(sh), s["Q"].reshape(sh)
    aol = _aol(ns, s["maxs"])
    fixed = torch.zeros(sh, dtype=torch.bool, device=_dev())
    fixed.view(-1)[_gpu(s["dn"])] = True
    psi = torch.where(fixed, s["dpsi"].reshape(sh), s["psi0"].reshape(sh))

    def parts(psi):
        out = []
        for k, ((pa, pb), (za, zb)) in enumerate(zip(_pairs(psi), _pairs(z))):
            ka, kb = _kr(pa, al[k], N[k]), _kr(pb, al[k], N[k])
            t = ka[0] + kb[0]
            out.append({"H": 2.0 * ka[0] * kb[0] / t, "wa": 2.0 * (kb[0] / t) ** 2, "wb": 2.0 * (ka[0] / t) ** 2,
                        "ka": ka, "kb": kb, "D": pb + zb - pa - za})
        return out

    def residual(ps):
        R = Q.clone()
        for k, (p, (ra, rb)) in enumerate(zip(ps, _pairs(R))):
            f = p["H"] * Ks[k] * aol[k] * p["D"]
            ra += f
            rb -= f
        return torch.where(fixed, torch.zeros_like(R), R)

    ps = parts(psi)
    R = residual(ps)
    rn, r0, stuck = float(R.norm()), float(R.norm()), 0
    for _ in range(300):
        S = _Steady(ns, s["maxs"], [p["H"] * Ks[k] for k, p in enumerate(ps)], [s["dn"]])
        d = S.grid.solve(R)
        w = 1.0
        for _ in range(6):  # the step is halved while the residual does not drop, and taken after five halvings
            new = torch.where(fixed, psi, psi + w * d)
            qs = parts(new)
            Rn = residual(qs)
            got = float(Rn.norm())
            if got < rn:
                break
            w *= 0.5
        if got >= rn and rn < 1e-9 * r0:
            break  # the rounding floor
        psi, ps, R = new, qs, Rn
        stuck = stuck + 1 if got > 0.9 * rn and got < 1e-12 * r0 else 0
        rn = got
        if stuck > 3:
            break
    S = _Steady(ns, s["maxs"], [p["H"] * Ks[k] for k, p in enumerate(ps)], [s["dn"]])
    c, leak, _ = S.grid.lv[0]
    na = [Ks[k] * aol[k] * p["wa"] * p["ka"][1] * p["D"] for k, p in enumerate(ps)]
    nb = [-Ks[k] * aol[k] * p["wb"] * p["kb"][1] * p["D"] for k, p in enumerate(ps)]
    zero = torch.zeros_like(psi)

    def transposed(v):  # (A - N^T) v on the free cells
        y = _apply(c, leak, v)
        for k, ((va, vb), (ya, yb)) in enumerate(zip(_pairs(v), _pairs(y))):
            ya -= na[k] * (va - vb)
            yb -= nb[k] * (vb - va)
        return torch.where(fixed, zero, y)

    delta = s["delta"].reshape(sh)
    b = torch.where(fixed, zero, delta)
    mu = zero
    bn = float(b.norm())
    last = None
    for _ in range(12):  # GMRES(60), preconditioned from the right
        r = b - transposed(mu)
        beta = float(r.norm())
        if beta <= 1e-15 * bn or (last is not None and beta > 0.5 * last):
            break
        last = beta
        V, Z, H = [r / beta], [], np.zeros((61, 60))
        for j in range(60):
            Z.append(torch.where(fixed, zero, S.grid.precondition(V[j])))
            w = transposed(Z[j])
            for _ in range(2):
                for i in range(j + 1):
                    hij = float((w * V[i]).sum())
                    H[i, j] += hij
                    w = w - hij * V[i]
            H[j + 1, j] = float(w.norm())
            V.append(w / H[j + 1, j])
            e = np.zeros(j + 2)
            e[0] = beta
            y, res, _, _ = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)
            if float(np.linalg.norm(e - H[:j + 2, :j + 1] @ y)) <= 1e-3 * 1e-13 * bn:
                break
        for i, yi in enumerate(y):
            mu = mu + float(yi) * Z[i]
    dK, dal, dN = [], [], []
    ddp = zero.clone()
    for k, (p, (ma, mb), (da, db), (fa, fb)) in enumerate(zip(ps, _pairs(mu), _pairs(ddp), _pairs(fixed))):
        t = aol[k] * p["D"] * (ma - mb)
        dK.append((p["H"] * t)[0])
        dal.append((Ks[k] * t * (p["wa"] * p["ka"][2] + p["wb"] * p["kb"][2]))[0])
        dN.append((Ks[k] * t * (p["wa"] * p["ka"][3] + p["wb"] * p["kb"][3]))[0])
        q = Ks[k] * aol[k]
        db += q * (p["wb"] * p["kb"][1] * p["D"] + p["H"]) * ma
        da += q * (-p["wa"] * p["ka"][1] * p["D"] + p["H"]) * mb
    ddp = torch.where(fixed, ddp + delta, zero)
    return (psi.reshape(-1), _join_faces(ns, dK), ddp.reshape(-1), _join_faces(ns, dal), _join_faces(ns, dN),
            mu.reshape(-1))


def _exact_faces(case, seed):
    s = _faces_inputs(case, seed)
    ns, nb, F = s["ns"], s["batch"], _nfaces(s["ns"])
    Ks, gs = [], []
    for p in range(nb):
        n = ns[0] * ns[1] * ns[2]
        lk = s["logK"][p * n:(p + 1) * n].reshape(ns)
        K = _mean_faces(lk, case["mean"])
        Ks.append(_join_faces(ns, [k[0] for k in K]))
        g = torch.zeros_like(lk)
        for dk, (_, ka, kb), (ga, gb) in zip(_split_faces(ns, s["dKs"][p * F:(p + 1) * F]), K, _pairs(g)):
            ga += ka * dk
            gb += kb * dk
        gs.append(g.reshape(-1))
    return torch.cat(Ks), torch.cat(gs)


def exact(case, seed):
    f = {"dropin": _exact_steady, "steady": _exact_steady, "direct": _exact_steady, "grad": _exact_grad,
         "transient": _exact_transient, "mesh": _exact_mesh, "richards": _exact_richards, "faces": _exact_faces}
    return f[case["kind"]](case, seed)
