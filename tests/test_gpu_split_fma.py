"""Flux splitting of the contracted build on tensor-product grids (split_sw_diag, split_llf_diag)
against the CPU oracle: both splittings, periodic lines and lines with end planes, tiles with
remainders, and a grid that runs against two of its axes (negative metric components). Relative
L-infinity <= 1e-10 after three steps, the bar of this path, plus 1e-13 of the largest momentum for a
momentum component (the rounding of the fluxes that cancel in the plate's small ones). The library
variant is chosen when the package is imported, so the GPU side runs in a child process (this file
as a program).
"""
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
pytestmark = pytest.mark.gpu
CASES = [("box", "WENO5", 1), ("box", "OMP6", 2), ("against", "WENO5", 1), ("against", "WENO7", 2), ("plate", "OMP6", 1),
         ("plate", "HYBRID", 2), ("plate", "WENO5", 2)]


def case(kind, scheme, splitting):
    from ocfd_b200 import cases
    if kind == "plate":
        c = cases.flatplate(nx=33, ny=19, nz=9, scheme=scheme, lx=0.01, ly=0.004, y1=2e-5)
        c.params.flux_splitting = splitting
        return c
    c = cases.isotropic(n=11, scheme=scheme, flux_splitting=splitting)
    if kind == "against":
        for d in (0, 1):
            c.coords[d] *= -1.0
            c.params.periodic_span[d][d] *= -1.0
    return c


def run(make, args):
    c = case(*args)
    g = make(c)
    g.init_state()
    for s in range(3):
        g.tt = s * c.dt
        g.step(c.dt, s * c.dt) if hasattr(g, "diag") else g.step(c.dt)  # the oracle takes the time
    out = g.download_state()
    g.close()
    return out


def child(out):
    os.environ["OCFD_B200_LIB"] = "fma"
    sys.path.insert(0, os.path.join(ROOT, "opencfd-comb_b200"))
    from ocfd_b200 import solver
    assert solver.VARIANT == "fma"
    np.savez(out, **{"f%d" % n: run(solver.Solver, args)[0] for n, args in enumerate(CASES)})


@pytest.fixture(scope="module")
def contracted(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("split") / "gpu.npz")
    env = dict(os.environ, OCFD_B200_LIB="fma")
    subprocess.run([sys.executable, os.path.abspath(__file__), out], check=True, env=env, timeout=300)
    return np.load(out)


@pytest.mark.parametrize("n", range(len(CASES)))
def test_split_on_tensor_grids(oracle, contracted, n):
    want = run(oracle.OracleSolver, CASES[n])[0]
    got = contracted["f%d" % n]
    assert np.isfinite(want).all()
    mom = 1e-13 * np.abs(want[1:4]).max()
    for m in range(5):
        assert np.abs(got[m] - want[m]).max() <= 1e-10 * np.abs(want[m]).max() + (mom if 1 <= m <= 3 else 0.0), m


if __name__ == "__main__":
    child(sys.argv[1])
