"""Fitted mixture transport (k_transport_fit) against the CPU oracle for every species count's
dispatch and both library builds. The viscosity is compared as the mean that ana_box reports; conductivity and diffusion
through what they do to the state: the difference of a viscous and an inviscid step, which is the
viscous terms alone.

Tolerances: the coefficients are products of exponentials with a few ulp each, so the mean viscosity
agrees to 1e-12. In the step differences the states' own rounding (a few hundred operations, 1e-13
of the largest value) stands against the viscous increment; 1e-10 of the increment is allowed on top.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

if __name__ == "__main__":  # the child of the contracted build's test
    sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "opencfd-comb_b200"))
from ocfd_b200 import cases, solver

pytestmark = pytest.mark.gpu


def case(n, ns, seed):
    names = cases.h2air_structs()[0][:ns] if ns < 9 else cases.h2air_structs()[0]
    rng = np.random.default_rng(seed)
    c = cases.isotropic(n=n, species=list(names), Y=list(rng.uniform(0.1, 1.0, ns)), wilke=True, T0=900.0)
    x = 2.0 * np.pi * np.arange(n) / n
    s = np.sin(x)[None, None, :] + np.cos(x)[None, :, None] + np.sin(x)[:, None, None]
    c.prim5[4] *= 1.0 + 0.2 * s / 3.0  # temperatures on both sides of the 1000 K range boundary
    w = np.array([1.0 + 0.3 * np.roll(s, 2 * k + 1, axis=k % 3) / 3.0 for k in range(ns)])
    c.di = np.ascontiguousarray(c.di * w)
    c.dt *= 1.0e-2
    return c


def steps(make, c):
    out = []
    for visc in (1, 0):
        c.params.if_viscous = visc
        g = make(c)
        g.init_state()
        g.step(c.dt)
        f, di, _ = g.download_state()
        mu = g.ana_box(0.0)[15] if visc else None
        out.append((f, di[:, 4:-4, 4:-4, 4:-4], mu))
        g.close()
    return out


@pytest.mark.parametrize("ns,n", [(2, 9), (3, 8), (5, 13), (9, 11)])
def test_transport_fit_against_oracle(oracle, ns, n):
    c = case(n, ns, ns)
    gv, gi = steps(solver.Solver, c)
    ov, oi = steps(oracle.OracleSolver, c)
    assert abs(gv[2] - ov[2]) <= 1e-12 * abs(ov[2])
    for a, b, r, s in ((gv[0], gi[0], ov[0], oi[0]), (gv[1], gi[1], ov[1], oi[1])):
        for m in range(len(r)):
            want, got = r[m] - s[m], a[m] - b[m]
            assert np.abs(got - want).max() <= 1e-13 * np.abs(r[m]).max() + 1e-10 * np.abs(want).max(), m


def unmixed(ns, n=12, trace=0.0):
    """two of the species side by side, each alone in its half of a periodic box, but for traces of all"""
    c = case(n, ns, ns)
    half = np.where(np.arange(n) < n // 2, 1.0, 0.0)
    d = c.di.sum(axis=0)
    c.di = np.zeros_like(c.di) + trace * d
    c.di[0] += d * half
    c.di[1] += d * (1.0 - half)
    return c


@pytest.mark.parametrize("ns", [2, 9])
def test_cells_of_one_species(oracle, ns):
    """X = 1 exactly where a species is alone: its diffusion coefficient (1 - X) / (sum + 1e-20) is 0
    there. Last-place changes of the initial state move the oracle's own increments by less than a
    hundredth of the bound."""
    c = unmixed(ns)
    gv, gi = steps(solver.Solver, c)
    ov, oi = steps(oracle.OracleSolver, c)
    for a, b, r, s in ((gv[0], gi[0], ov[0], oi[0]), (gv[1], gi[1], ov[1], oi[1])):
        for m in range(len(r)):
            want, got = r[m] - s[m], a[m] - b[m]
            assert np.abs(got - want).max() <= 1e-13 * np.abs(r[m]).max() + 1e-10 * np.abs(want).max(), m


ALL = [(2, 9), (3, 8), (4, 10), (5, 13), (6, 9), (7, 12), (8, 8), (9, 11)]
CASES = [("t%d" % ns, (lambda ns=ns, n=n: case(n, ns, ns))) for ns, n in ALL]
CASES += [("u%d" % ns, (lambda ns=ns: unmixed(ns))) for ns in (2, 9)]
CASES += [("v%d" % ns, (lambda ns=ns: unmixed(ns, trace=1.0e-18))) for ns in (2, 9)]


def _child(out):
    res = {"variant": solver.VARIANT}
    for tag, make in CASES:
        c = make()
        for v, (f, di, mu) in enumerate(steps(solver.Solver, c)):
            res["%s_f%d" % (tag, v)], res["%s_d%d" % (tag, v)] = f, di
            if mu is not None:
                res[tag + "_mu"] = mu
    np.savez(out, **res)


@pytest.fixture(scope="module", params=["exact", "fma"])
def both_builds(request, tmp_path_factory):
    out = str(tmp_path_factory.mktemp("transport") / "gpu.npz")
    subprocess.run([sys.executable, os.path.abspath(__file__), out], check=True, timeout=300,
                   env=dict(os.environ, OCFD_B200_LIB=request.param))
    z = np.load(out)
    assert str(z["variant"]) == request.param
    return z


@pytest.mark.parametrize("tag,make", CASES, ids=[tag for tag, _ in CASES])
def test_every_species_count_in_both_builds(oracle, both_builds, tag, make):
    """the same comparison and bounds for every instance of the kernel in the exact and the contracted
    library; the contracted flow kernels' own rounding is that of the states, 1e-13 of the largest value"""
    ov, oi = steps(oracle.OracleSolver, make())
    if tag[0] == "t":
        assert abs(both_builds[tag + "_mu"] - ov[2]) <= 1e-12 * abs(ov[2])
    for k, v in (("f", 0), ("d", 1)):
        for m in range(len(ov[v])):
            want = ov[v][m] - oi[v][m]
            got = both_builds["%s_%s0" % (tag, k)][m] - both_builds["%s_%s1" % (tag, k)][m]
            assert np.abs(got - want).max() <= 1e-13 * np.abs(ov[v][m]).max() + 1e-10 * np.abs(want).max(), (k, m)


if __name__ == "__main__":
    _child(sys.argv[1])
