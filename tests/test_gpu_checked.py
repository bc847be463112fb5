"""The checked build (DPF_CHECK: device-side bounds and alignment checks that record a
violation instead of trapping) runs small and ragged cases of every kernel family with no
violation and the oracle's answers; the regular build reports the checks as absent."""
import ctypes
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_checked_build_runs_clean(gpu_lib):
    import __graft_entry__ as g
    b = g._load_build_module()
    lib = b.build(out_dir=os.path.join(ROOT, "dpfehm.jl_gb300", "_build_check"), defines=["DPF_CHECK"])
    env = dict(os.environ, DPFEHM_GPU_LIB=os.path.abspath(lib))
    r = subprocess.run([sys.executable, os.path.join(ROOT, "tests", "checked_cases.py")], env=env,
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out["rc"] == 0
    assert out["violations"] == 0, out["first"]
    e = out["errors"]
    assert e["steady"] < 1e-8 and e["batch"] < 1e-8 and e["csr"] < 1e-8 and e["transient"] < 1e-8, e
    assert e["adjoint"] < 1e-6, e
    assert e["richards"] < 1e-8 and e["richards_adjoint"] < 1e-6, e


def test_regular_build_has_no_checks(gpu_lib):
    lib = gpu_lib.load()
    nv = ctypes.c_int64(-1)
    assert lib.dpf_debug_check_report(ctypes.byref(nv), None) == 8   # DPF_UNSUPPORTED


SITES = """
import ctypes, json, sys
import numpy as np
sys.path[:0] = [%r, %r]
import __graft_entry__ as g
pkg = g.load_package()
lib = pkg.load()
for prec in ("fp64", "mixed"):
    for ns in ((9, 7, 5), (33, 20, 11)):
        n = int(np.prod(ns))
        _, nb, aol, _ = pkg.regulargrid3d((0.0, 0.0, 0.0), tuple(0.5 * (k - 1) + 0.5 for k in ns), ns)
        K, q = np.exp(np.random.default_rng(n).normal(-9, 1, len(nb))), np.zeros(n)
        q[3] = 1e-4
        for general in (False, True):
            P = pkg.GroundwaterProblem(nb, aol, np.array([n - 1]), N=n, reltol=1e-12, precision=prec, general=general)
            l0 = P.launch_count
            P.forward(K, np.zeros(n), q)
            assert P.launch_count - l0 < 60, "not a one-launch solve"
            P.close()
nv, first, sites = ctypes.c_int64(-1), (ctypes.c_int64 * 3)(), ctypes.c_int64(0)
rc = [lib.dpf_debug_check_report(ctypes.byref(nv), first), lib.dpf_debug_check_sites(ctypes.byref(sites))]
print(json.dumps({"rc": rc, "violations": nv.value, "first": list(first), "sites": sites.value}))
"""


def test_one_launch_solves_are_checked(gpu_lib):
    """The gathers of the one-launch solves are among the checks: columns (site 8) and aggregates (9) of face lists,
    children (10) of grids, beside the shared cell decode and neighbours (1, 2)."""
    import __graft_entry__ as g
    b = g._load_build_module()
    lib = b.build(out_dir=os.path.join(ROOT, "dpfehm.jl_gb300", "_build_check"), defines=["DPF_CHECK"])
    env = dict(os.environ, DPFEHM_GPU_LIB=os.path.abspath(lib))
    r = subprocess.run([sys.executable, "-c", SITES % (ROOT, os.path.join(ROOT, "oracle"))], env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out["rc"] == [0, 0] and out["violations"] == 0, out
    assert all(out["sites"] >> k & 1 for k in (1, 2, 8, 9, 10)), out


def test_regular_build_has_no_sites(gpu_lib):
    assert gpu_lib.load().dpf_debug_check_sites(None) == 8   # DPF_UNSUPPORTED
