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
    elif kind == "limit":  # either side of the 90 K limit
        T = rng.uniform(80.0, 100.0, n)
    elif kind == "hot":  # products whose Newton's first guess, and some of whose temperatures, lie above the fits
        X = dict(H2O=0.5, N2=0.4, OH=0.05, H=0.03, O=0.02)
        Y = np.array([X.get(s, 1e-6) * th.mi[k] for k, s in enumerate(names)])
        di = np.outer(rng.uniform(0.05, 0.2, n), Y / Y.sum())
        T = rng.uniform(2900.0, 5600.0, n)
        dt, nsub = np.full(n, 1.0e-7), np.full(n, 10, dtype=np.int32)
    elif kind == "pivots":  # the first sub-step of "stiff": a tenth of the lanes
        di[:, [names.index(s) for s in ("O", "OH", "H", "HO2", "H2O2")]] += 1e-2 * di.sum(axis=1, keepdims=True)
        dt, nsub = np.full(n, 1.0e-6), np.ones(n, dtype=np.int32)
        T = rng.uniform(1900.0, 2500.0, n)
    elif kind == "overshoot":  # the first sub-step leaves negative densities to the second
        di[:, [names.index(s) for s in ("O", "OH", "H", "HO2", "H2O2")]] += 1e-2 * di.sum(axis=1, keepdims=True)
        dt, nsub = np.full(n, 2.0e-7), np.full(n, 2, dtype=np.int32)
        T = rng.uniform(1900.0, 2500.0, n)
    elif kind == "ranges":  # five fit ranges
        T = rng.uniform(400.0, 3000.0, n)
        for k in range(9):
            old = [list(th.coef[k][j]) for j in (0, 1)]
            for j, o in enumerate((0, 0, 1, 1, 1)):
                th.coef[k][j][:] = old[o]
                th.coef[k][j][0] = old[o][0] * (1.0 + 0.01 * j)
        th.n_tct = 5
        th.tct[:4] = [600.0, 1000.0, 1500.0, 2200.0]
    e = np.ascontiguousarray(cases.energy_realgas(th, di.T.copy(), T))
    if kind == "ideal":
        e = np.ascontiguousarray(2.5 * T * (di @ np.array([8.314 / th.mi[k] for k in range(9)])))
    return th, kin, np.ascontiguousarray(di), e, np.ascontiguousarray(dt), np.ascontiguousarray(nsub)


CASES = [("usual", 1), ("usual", 33), ("usual", 4097), ("cold", 40), ("boundary", 97), ("stiff", 65),
         ("limit", 41), ("hot", 65), ("pivots", 321), ("overshoot", 66), ("ranges", 67), ("ideal", 68)]


def multipliers(oracle, th, kin, di, e, h):
    """Largest multiplier of each reactor's unpivoted elimination of I - h J in moles, without N2. The rates
    are the oracle's explicit steps, J their differences at the same temperature."""
    from ocfd_b200 import cases
    M = np.array([th.mi[k] for k in range(9)])
    T = temperatures(oracle, th, di, e)

    def rate(d):
        d = np.ascontiguousarray(d)
        x, dt = d.copy(), np.full(len(d), 1.0e-3)
        oracle.chem_batch(th, kin, 1, 1, x, np.ascontiguousarray(cases.energy_realgas(th, d.T.copy(), T)), dt, None)
        return (x - d) / dt[:, None] / M

    A = np.tile(np.eye(9), (len(di), 1, 1))
    for j in range(9):
        step = 1.0e-6 * (di[:, j] + 1e-6 * di.sum(axis=1))
        up, down = di.copy(), di.copy()
        up[:, j] += step
        down[:, j] -= step
        A[:, :, j] -= h[:, None] * (rate(up) - rate(down)) / (2.0 * step / M[j])[:, None]
    A, most = A[:, :8, :8], np.zeros(len(di))
    for k in range(7):
        f = A[:, k + 1:, k] / A[:, k, k][:, None]
        most = np.maximum(most, np.abs(f).max(axis=1))
        A[:, k + 1:] -= f[:, :, None] * A[:, k, None, :]
    return most


def temperatures(oracle, th, di, e):
    return np.array([oracle.probe(th, 1, 1, np.ascontiguousarray(d), x) for d, x in zip(di, e)])


def first_guess(th, di, e):
    a0 = np.array([(th.coef[k][0][0] - 1.0) * 8.314 / th.mi[k] for k in range(9)])
    return e / (di @ a0)


def test_states_reach_their_branches(oracle):
    """the states of the cases are those that their names promise"""
    th, kin, di, e, dt, nsub = states("hot", 65)
    T = temperatures(oracle, th, di, e)
    assert (first_guess(th, di, e) > th.tct_max).mean() > 0.5 and 0.1 < (T > th.tct_max).mean() < 0.9
    th, kin, di, e, dt, nsub = states("limit", 41)
    assert 0.2 < (temperatures(oracle, th, di, e) < 90.0).mean() < 0.8
    th, kin, di, e, dt, nsub = states("pivots", 321)
    assert (multipliers(oracle, th, kin, di, e, dt / nsub) > 16.0).sum() >= 5
    th, kin, di, e, dt, nsub = states("usual", 33)
    assert (multipliers(oracle, th, kin, di, e, dt / nsub) < 16.0).all()
    th, kin, di, e, dt, nsub = states("overshoot", 66)
    oracle.chem_batch(th, kin, 1, -1, di, e, 0.5 * dt, None)
    assert (di.min(axis=1) < -1e-6 * di.sum(axis=1)).mean() > 0.5 and (e > 0.0).all()


def test_hot_reactors_take_the_same_path():
    """a sub-step costs the same at any temperature: reactors above the fits or with a first guess there ran
    13 times as long as others when they took the general step"""
    code = """if 1:
        import sys, time
        import numpy as np
        sys.path[:0] = [%r, %r]
        import test_gpu_chem_fma as t
        from ocfd_b200 import abi, solver
        best = {}
        for kind in ("usual", "hot"):
            th, kin, di, e, dt, nsub = t.states(kind, 40000)
            dt, nsub = np.full(40000, 1.0e-7), np.full(40000, 10, dtype=np.int32)
            solver.chem_setup(th, kin, 1, abi.CHEM_IMPLICIT)
            solver.chem_batch(di.copy(), e.copy(), dt, nsub)
            solver.Solver.profile(True)
            ms = []
            for _ in range(5):
                before = solver.Solver.profile_read()["chem"][0]
                solver.chem_batch(di.copy(), e.copy(), dt, nsub)
                ms.append(solver.Solver.profile_read()["chem"][0] - before)
            best[kind] = min(ms)
        print(best["usual"], best["hot"])
        assert 0.0 < best["hot"] < 3.0 * best["usual"]
    """ % (os.path.join(ROOT, "opencfd-comb_b200"), HERE)
    subprocess.run([sys.executable, "-c", code], check=True, env=dict(os.environ, OCFD_B200_LIB="fma"), timeout=300)


def child(out):
    os.environ["OCFD_B200_LIB"] = "fma"
    sys.path.insert(0, os.path.join(ROOT, "opencfd-comb_b200"))
    from ocfd_b200 import abi, solver
    res = {}
    for kind, n in CASES:
        for cp in (0, 1):
            th, kin, di, e, dt, nsub = states(kind, n)
            solver.chem_setup(th, kin, int(kind != "ideal"), abi.CHEM_IMPLICIT, const_p=bool(cp))
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
    oracle.chem_batch(th, kin, int(kind != "ideal"), -1, di, e, dt, nsub, const_p=bool(cp))
    gd, ge = (gpu_results["%s_%d_%d_%s" % (kind, n, cp, f)] for f in ("di", "e"))
    assert np.isfinite(di).all()
    assert (np.abs(gd - di).max(axis=1) <= 1e-10 * np.abs(di).max(axis=1)).all()
    change = np.abs(di - d0).max(axis=0)
    assert (np.abs(gd - di).max(axis=0) <= 1e-8 * change + 1e-13 * np.abs(di).max(axis=0)).all()
    assert (np.abs(ge - e) <= 1e-10 * np.abs(e).max()).all()


if __name__ == "__main__":
    child(sys.argv[1])
