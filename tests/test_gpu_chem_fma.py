"""The contracted build's compiled-mechanism chemistry (ocfd_mech_fast.cuh) against the CPU oracle:
batched reactors at the sizes and states where its branches lie (batches that do not fill a warp,
temperatures below the equilibrium-product form's limit and beside the fit ranges' boundary, time
steps that need the pivoted elimination), constant volume and constant pressure. The library variant
is chosen when the package is imported, so the GPU side runs in a child process (this file as a
program).

Tolerance: 1e-10 of a reactor's largest density and of the energy, the bar of this path; besides,
every species' change over the call, which is small against its density in many of these states, to
1e-8 of the batch's largest change plus 1e-13 of its largest density (a hundred sub-steps' rounding).
A change of the inputs by one unit in the last place moves the oracle's own results by at most 3e-12.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

pytestmark = pytest.mark.gpu


def states(kind, n):
    from ocfd_b200 import cases
    names, th, kin, di, e, dt, nsub, T = cases.reactors(n=n, seed=n)
    rng = np.random.default_rng(n)
    if kind == "cold":  # either side of the 150 K limit
        T = rng.uniform(110.0, 190.0, n)
    elif kind == "boundary":  # either side of the 1000 K range boundary
        T = rng.uniform(999.0, 1001.0, n)
    elif kind == "stiff":  # radicals and steps far beyond the explicit limit
        di[:, [names.index(s) for s in ("O", "OH", "H", "HO2", "H2O2")]] += 1e-2 * di.sum(axis=1, keepdims=True)
        dt = np.full(n, 3.0e-6)
        nsub = np.full(n, 3, dtype=np.int32)
        T = rng.uniform(1200.0, 2200.0, n)
    e = np.ascontiguousarray(cases.energy_realgas(th, di.T.copy(), T))
    return th, kin, np.ascontiguousarray(di), e, np.ascontiguousarray(dt), np.ascontiguousarray(nsub)


CASES = [("usual", 1), ("usual", 33), ("usual", 4097), ("cold", 40), ("boundary", 97), ("stiff", 65)]


def child(out):
    os.environ["OCFD_B200_LIB"] = "fma"
    sys.path.insert(0, os.path.join(ROOT, "opencfd-comb_b200"))
    from ocfd_b200 import abi, solver
    res = {}
    for kind, n in CASES:
        for cp in (0, 1):
            th, kin, di, e, dt, nsub = states(kind, n)
            solver.chem_setup(th, kin, 1, abi.CHEM_IMPLICIT, const_p=bool(cp))
            assert solver.VARIANT == "fma" and solver.lib().ocfd_gpu_chem_compiled_mechanism(-1) == 1
            solver.chem_batch(di, e, dt, nsub)
            res["%s_%d_%d_di" % (kind, n, cp)] = di
            res["%s_%d_%d_e" % (kind, n, cp)] = e
    np.savez(out, **res)


@pytest.fixture(scope="module")
def gpu_results(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("chem") / "gpu.npz")
    env = dict(os.environ, OCFD_B200_LIB="fma")
    subprocess.run([sys.executable, os.path.abspath(__file__), out], check=True, env=env, timeout=300)
    return np.load(out)


@pytest.mark.parametrize("cp", [0, 1])
@pytest.mark.parametrize("kind,n", CASES)
def test_compiled_mechanism_step(oracle, gpu_results, kind, n, cp):
    th, kin, di, e, dt, nsub = states(kind, n)
    d0 = di.copy()
    oracle.chem_batch(th, kin, 1, -1, di, e, dt, nsub, const_p=bool(cp))
    gd, ge = (gpu_results["%s_%d_%d_%s" % (kind, n, cp, f)] for f in ("di", "e"))
    assert np.isfinite(di).all()
    assert (np.abs(gd - di).max(axis=1) <= 1e-10 * np.abs(di).max(axis=1)).all()
    change = np.abs(di - d0).max(axis=0)
    assert (np.abs(gd - di).max(axis=0) <= 1e-8 * change + 1e-13 * np.abs(di).max(axis=0)).all()
    assert (np.abs(ge - e) <= 1e-10 * np.abs(e).max()).all()


if __name__ == "__main__":
    child(sys.argv[1])
