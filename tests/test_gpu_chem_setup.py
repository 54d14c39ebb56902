"""ocfd_gpu_chem_setup on an open flow solver: the flow's later steps take the new thermodynamics in
every kernel, in both library builds. A solver whose tables were replaced is compared with one that was
opened with them, from the same uploaded state: with other enthalpy fits bit for bit; with other molar
masses (whose pair constants of the viscosity stay those of the opening) through the species' diffusion
in a gas at rest, to 1e-6 of its increment. The libraries run in child processes (this file as a
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


def case(change, visc=1):
    from ocfd_b200 import cases
    names, th, kin, _ = cases.h2air_structs()
    c = cases.isotropic(n=10, species=list(names), Y=[1.0 + 0.2 * k for k in range(9)], wilke=True, T0=900.0)
    c.kin = kin
    c.params.if_viscous = visc
    x = 2.0 * np.pi * np.arange(10) / 10
    c.di = np.ascontiguousarray(c.di * np.array([1.0 + 0.3 * np.sin(x + k) for k in range(9)])[:, None, None, :])
    c.prim5[4] = 900.0 * (1.0 + 0.2 * np.cos(x))
    if change:  # at rest for the masses: the viscosity then enters by the pressure waves alone
        c.prim5[1:4] *= 0.0 if change == "mass" else 1.0
        c.dt *= 1.0e-2
    return c


def altered(th, change):
    for k in range(9):
        if change == "fits":
            for j in range(th.n_tct):
                th.coef[k][j][0] *= 1.0 + 0.01 * (k + 1)
        else:
            th.mi[k] *= 1.0 + 0.02 * k
    return th


def run(change, replaced, visc):
    import copy

    from ocfd_b200 import solver
    c = case(change, visc)
    if not replaced:
        c.thermo = altered(copy.deepcopy(c.thermo), change)
    start = case(change, visc)
    g = solver.Solver(start)
    g.init_state()
    state = g.download_state()
    g.close()
    g = solver.Solver(c)
    g.init_state()
    if replaced:
        solver.chem_setup(altered(copy.deepcopy(c.thermo), change), c.kin, c.params.if_realgas, c.params.chem_timeadv)
    g.upload_state(*state)
    g.step(c.dt)
    f, di, _ = g.download_state()
    g.close()
    return f, di[:, 4:-4, 4:-4, 4:-4]


def child(out):
    sys.path.insert(0, os.path.join(ROOT, "opencfd-comb_b200"))
    res = {}
    for change in ("fits", "mass"):
        for replaced in (0, 1):
            for visc in (0, 1):
                key = "%s%d%d" % (change, replaced, visc)
                res["f" + key], res["d" + key] = run(change, replaced, visc)
    np.savez(out, **res)


@pytest.fixture(scope="module", params=["exact", "fma"])
def results(request, tmp_path_factory):
    out = str(tmp_path_factory.mktemp("setup") / "gpu.npz")
    env = dict(os.environ, OCFD_B200_LIB=request.param)
    subprocess.run([sys.executable, os.path.abspath(__file__), out], check=True, env=env, timeout=300)
    return np.load(out)


def test_new_fits_reach_every_kernel(results):
    for v in "fd":
        assert np.isfinite(results[v + "fits01"]).all()
        assert np.array_equal(results[v + "fits01"], results[v + "fits11"]), v


def test_new_masses_reach_the_diffusion(results):
    want, got = (results["dmass%d1" % r] - results["dmass%d0" % r] for r in (0, 1))
    for m in range(9):
        assert np.abs(want[m]).max() > 0.0
        assert np.abs(got[m] - want[m]).max() <= 1e-6 * np.abs(want[m]).max(), m


if __name__ == "__main__":
    child(sys.argv[1])
