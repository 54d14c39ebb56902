"""Species viscous kernels (k_spec_ev, k_spec_div and the face cells' k_scal_ev / k_scal_div) against
the CPU oracle, both library builds: jets whose sizes are odd, barely wider than the stencils (every
cell a face cell for CD8) or span several tiles, and a periodic box without face cells.

What the terms do to the state is the difference of a viscous and an inviscid step. The states' own
rounding (a few hundred operations, 1e-13 of the largest value) stands against it; 1e-9 of the
difference is allowed on top. The contracted build's side runs in a child process (this file as a
program), since the variant is chosen when the package is imported.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
pytestmark = pytest.mark.gpu

CASES = [("jet", 33, 9, 8, "CD6"), ("jet", 8, 10, 8, "CD8"), ("jet", 67, 37, 13, "CD6"), ("jet", 35, 18, 12, "CD8"),
         ("box", 9, 9, 9, "CD6"), ("box", 10, 10, 10, "CD8")]


def case(kind, nx, ny, nz, vis):
    from ocfd_b200 import abi, cases
    if kind == "jet":
        c = cases.jet(nx=nx, ny=ny, nz=nz)
    else:
        names = cases.h2air_structs()[0]
        c = cases.isotropic(n=nx, species=list(names), Y=[1.0 + 0.3 * k for k in range(len(names))], wilke=True, T0=1000.0)
    rng = np.random.default_rng(nx)
    c.prim5[4] *= 1.0 + 0.1 * rng.uniform(-1.0, 1.0, c.prim5[4].shape)
    c.di = np.ascontiguousarray((c.di + 1e-3 * c.di.sum(axis=0)) * rng.uniform(0.9, 1.1, c.di.shape))
    c.params.scheme_vis = abi.SCHEME_CD8 if vis == "CD8" else abi.SCHEME_CD6
    return c


def steps(make, args):
    out = []
    for visc in (1, 0):
        c = case(*args)
        c.params.if_viscous = visc
        g = make(c)
        g.init_state()
        g.step(c.dt)
        f, di, _ = g.download_state()
        out.append((f, di[:, 4:-4, 4:-4, 4:-4]))
        g.close()
    return out


def child(out):
    os.environ["OCFD_B200_LIB"] = "fma"
    sys.path.insert(0, os.path.join(ROOT, "opencfd-comb_b200"))
    from ocfd_b200 import solver
    assert solver.VARIANT == "fma"
    res = {}
    for n, args in enumerate(CASES):
        for v, (f, di) in enumerate(steps(solver.Solver, args)):
            res["f%d_%d" % (n, v)], res["d%d_%d" % (n, v)] = f, di
    np.savez(out, **res)


@pytest.fixture(scope="module")
def contracted(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("visc") / "gpu.npz")
    env = dict(os.environ, OCFD_B200_LIB="fma")
    subprocess.run([sys.executable, os.path.abspath(__file__), out], check=True, env=env, timeout=300)
    return np.load(out)


@pytest.mark.parametrize("build", ["exact", "fma"])
@pytest.mark.parametrize("n", range(len(CASES)))
def test_species_viscous_terms(oracle, contracted, build, n):
    ov, oi = steps(oracle.OracleSolver, CASES[n])
    if build == "fma":
        gv, gi = (tuple(contracted["%s%d_%d" % (k, n, v)] for k in "fd") for v in (0, 1))
    else:
        from ocfd_b200 import solver
        gv, gi = steps(solver.Solver, CASES[n])
    for a, b, r, s in zip(gv, gi, ov, oi):
        for m in range(len(r)):
            want = r[m] - s[m]
            assert np.abs((a[m] - b[m]) - want).max() <= 1e-13 * np.abs(r[m]).max() + 1e-9 * np.abs(want).max(), m


if __name__ == "__main__":
    child(sys.argv[1])
