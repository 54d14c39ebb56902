"""Fitted mixture transport (k_transport_fit) against the CPU oracle for every species count's
dispatch. The viscosity is compared as the mean that ana_box reports; conductivity and diffusion
through what they do to the state: the difference of a viscous and an inviscid step, which is the
viscous terms alone.

Tolerances: the coefficients are products of exponentials with a few ulp each, so the mean viscosity
agrees to 1e-12. In the step differences the states' own rounding (a few hundred operations, 1e-13
of the largest value) stands against the viscous increment; 1e-10 of the increment is allowed on top.
"""
import numpy as np
import pytest

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


def unmixed(ns, n=12):
    """two of the species side by side, each alone in its half of a periodic box"""
    c = case(n, ns, ns)
    half = np.where(np.arange(n) < n // 2, 1.0, 0.0)
    d = c.di.sum(axis=0)
    c.di = np.zeros_like(c.di)
    c.di[0], c.di[1] = d * half, d * (1.0 - half)
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
