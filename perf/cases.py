"""Performance cases of the framework: the work its users have it do, through its public entry points.

Three kinds of program use it, and each has cases over its own range of sizes:

  flow     a time-stepping run: state uploaded from pinned host memory, `ocfd_gpu_run` over a few
           Strang steps, state downloaded. Periodic turbulence boxes, the Mach 2.25 flat plate and
           the reacting H2 jet, from a few thousand to a few million cells (the 1024 x 160 flat
           plate and the 384 x 256 jet cross-section at reduced depth), every inviscid scheme, both
           splittings, CD6 and CD8, the characteristic form, one and nine species.
  reactors batched 0-D H2-air reactors on device or host arrays, constant volume or pressure, from
           hundreds to 2^20.
  network  the learned chemistry surrogate: gated inference on a batch, and the training of its
           network.

The cases run the build with contracted multiply-adds, the benchmark's default and the one a
production run takes (OCFD_B200_LIB=exact measures the other; a process holds one of the two). The
library keeps one global solver, so the states of one case share the open solver of their grid and
each pass uploads its own fields, as a restarted run does.
"""
import ctypes as C
import math
import os
import sys
import weakref

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "opencfd-comb_b200"))
os.environ.setdefault("OCFD_B200_LIB", "fma")

from ocfd_b200 import abi, cases, solver  # noqa: E402

R0, ATM, LAP = 8.314, 1.013e5, 4


# ---------------------------------------------------------------- the cases

def listed():
    flow = dict(kind="flow", splitting="SW", vis="CD6", char=False, tuned=False, nsub=1)
    box = dict(flow, flow="box", react=False, species=1)
    plate = dict(flow, flow="plate", react=False, species=1)
    jet = dict(flow, flow="jet", scheme="WENO5", react=True, species=9)
    reac = dict(kind="reactors", const_p=False, device=True)
    return [
        # the smallest flow call: one step of a 16^3 box (the smoke test's size); launches and
        # copies, not arithmetic
        dict(box, name="box16 one step", nx=16, ny=16, nz=16, scheme="WENO5", steps=1),
        # decaying isotropic turbulence at its configured 64^3, a chunk of steps between outputs
        dict(box, name="box64 WENO5", nx=64, ny=64, nz=64, scheme="WENO5", steps=32, tuned=True),
        # an odd size with the other options of the control file: OMP6, Lax-Friedrichs, CD8
        dict(box, name="box81 OMP6 LLF CD8", nx=81, ny=81, nz=81, scheme="OMP6", splitting="LLF",
             vis="CD8", steps=16),
        # the flat plate's production scheme at its production cross-section, a quarter of the depth
        dict(plate, name="plate 1024x160x32 HYBRID", nx=1024, ny=160, nz=32, scheme="HYBRID", steps=16,
             tuned=True),
        # a small ragged plate with the characteristic-space flux
        dict(plate, name="plate 217x67x19 char", nx=217, ny=67, nz=19, scheme="WENO7", char=True,
             steps=8),
        # the reacting jet at its production cross-section, an eighth of the depth
        dict(jet, name="jet 384x256x32", nx=384, ny=256, nz=32, steps=6, tuned=True),
        # a coarse ragged jet, as a set-up is tried out
        dict(jet, name="jet 97x61x43", nx=97, ny=61, nz=43, steps=8),
        # the whole C3 batch: 2^20 H2-air reactors with up to 100 sub-steps each
        dict(reac, name="reactors 2^20", n=1 << 20, nsub_max=100),
        # a ragged batch at constant pressure
        dict(reac, name="reactors 60001 const p", n=60001, nsub_max=100, const_p=True),
        # a handful of reactors on host arrays: latency of the whole call
        dict(reac, name="reactors 777 host", n=777, nsub_max=100, device=False),
        # gated surrogate chemistry of a batch
        dict(name="surrogate 2^19", kind="network", n=1 << 19, train=False, batch=0),
        # training of the surrogate's network: one epoch
        dict(name="surrogate training", kind="network", n=1 << 17, train=True, batch=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges; sizes over their logarithm, odd ones among them."""
    kind = rng.choice(["box", "box", "plate", "plate", "jet", "jet", "jet", "reactors", "reactors", "network"])
    if kind == "reactors":
        return dict(kind="reactors", n=_log(rng, 200, 1 << 20) | 1, nsub_max=rng.choice([1, 10, 100]),
                    const_p=rng.random() < 0.3, device=rng.random() < 0.7)
    if kind == "network":
        return dict(kind="network", n=_log(rng, 5000, 1 << 19) | 1, train=False, batch=0)
    c = dict(kind="flow", flow=kind, splitting=rng.choice(["SW", "SW", "LLF"]),
             vis=rng.choice(["CD6", "CD6", "CD8"]), char=False, tuned=rng.random() < 0.3, nsub=1)
    if kind == "box":
        n = _log(rng, 12, 120)
        nine = rng.random() < 0.3  # nine reacting species in a hot box, with chemistry sub-steps
        n = min(n, 72) if nine else n
        c.update(nx=n, ny=n, nz=n, scheme=rng.choice(["WENO5", "WENO5", "WENO7", "OMP6", "UD7L"]), react=nine,
                 species=9 if nine else 1, nsub=rng.choice([1, 2, 3]) if nine else 1)
        c["char"] = not nine and rng.random() < 0.2
    elif kind == "plate":
        c.update(nx=_log(rng, 60, 1024), ny=_log(rng, 40, 160), nz=_log(rng, 8, 32),
                 scheme=rng.choice(["HYBRID", "HYBRID", "OMP6", "WENO7"]), react=False, species=1, splitting="SW")
    else:
        c.update(nx=_log(rng, 40, 384), ny=_log(rng, 32, 256), nz=_log(rng, 16, 32), scheme="WENO5",
                 react=rng.random() < 0.8, species=9)
    cells = c["nx"] * c["ny"] * c["nz"]
    c["steps"] = max(1, min(16, int((8.0e6 if c["species"] == 9 else 3.0e7) / cells)))
    return c


# ---------------------------------------------------------------- flow runs

def _pinned(shape):
    """Page-locked host array of the library (ocfd_gpu_pinned_alloc), given back with its last view."""
    L, p, n = solver.lib(), C.c_void_p(), int(np.prod(shape))
    if L.ocfd_gpu_pinned_alloc(8 * n, C.byref(p)) != 0:
        raise MemoryError("pinned host memory")
    buf = (C.c_double * n).from_address(p.value)
    weakref.finalize(buf, L.ocfd_gpu_pinned_free, p).atexit = False
    return np.frombuffer(buf, dtype=np.float64).reshape(shape)


_open = []  # the open solver: its case as items, the Solver, the Case


def _flow_case(c):
    if c["flow"] == "box":
        names = cases.h2air_structs()[0] if c["species"] == 9 else None
        Y = None
        if names:  # a lean mixture with traces of every radical, hot enough to react
            Y = [{"O2": 0.22, "H2": 0.02, "H2O": 0.05, "N2": 0.71}.get(s, 1e-6) for s in names]
        case = cases.isotropic(n=c["nx"], scheme=c["scheme"], species=names, Y=Y, wilke=names is not None,
                               T0=1400.0 if names else 300.0)
        c0 = case.info["c0"]
        case.dt = 0.5 * case.info["h"] / (2.0 * c0)  # a control file's fixed step, below the CFL limit
    elif c["flow"] == "plate":
        case = cases.flatplate(nx=c["nx"], ny=c["ny"], nz=c["nz"], scheme=c["scheme"])
    else:
        case = cases.jet(nx=c["nx"], ny=c["ny"], nz=c["nz"])
    p = case.params
    p.flux_splitting = abi.SPLIT_LLF if c["splitting"] == "LLF" else abi.SPLIT_SW
    p.scheme_vis = abi.SCHEME_CD8 if c["vis"] == "CD8" else abi.SCHEME_CD6
    p.if_scheme_character = 1 if c["char"] else 0
    return case


def _solver(c):
    """The open solver of this case's grid and options (opened, and tuned where the case says so,
    by the first state of a case, as at the start of a run)."""
    key = tuple(sorted((k, v) for k, v in c.items() if k not in ("name", "steps")))
    if not _open or _open[0] != key:
        case = _flow_case(c)
        run = solver.Solver(case)
        run.init_state()
        if c["tuned"]:
            run.autotune(3)
        _open[:] = [key, run, case]
    return _open[1:]


def _smooth(rng, shape, modes=4):
    """Smooth random field of order 1: a sum of separable Fourier modes (low wave numbers)."""
    f = np.zeros(shape)
    for _ in range(modes):
        a = [np.cos(2.0 * math.pi * (rng.integers(1, 4) * np.arange(n) / n + rng.random())) for n in shape]
        f += a[0][:, None, None] * a[1][None, :, None] * a[2][None, None, :]
    return f / math.sqrt(modes)


def _flow_inputs(c, seed, case):
    """The case's initial primitives with a seeded, smooth disturbance: a few per cent of the
    velocity (tapered to nothing at non-periodic faces) and a per mille of the temperature."""
    rng = np.random.default_rng(seed)
    prim = case.prim5.copy()
    shape = prim.shape[1:]
    uref = 0.03 * max(float(np.abs(prim[1]).max()), 10.0)
    taper = 1.0
    for ax, per in zip((2, 1, 0), case.params.iperiodic):
        if not per:
            s = np.sin(math.pi * np.arange(shape[ax]) / (shape[ax] - 1)) ** 2
            taper = taper * s.reshape([-1 if a == ax else 1 for a in range(3)])
    for m in (1, 2, 3):
        prim[m] += uref * _smooth(rng, shape) * taper
    prim[4] *= 1.0 + 1.0e-3 * _smooth(rng, shape) * taper
    return prim


class Flow:
    def __init__(self, c, seed):
        self.c = c
        self.solver, case = _solver(c)
        prim = _flow_inputs(c, seed, case)
        chk, L, dp = solver._chk, solver.lib(), abi.dptr
        nx, ny, nz = case.shape
        shapes = [(5, nz, ny, nx), (case.params.n_spec,) + case.halo_shape(), (7,) + case.halo_shape()]
        self.start = [_pinned(s) for s in shapes]
        self.out = [_pinned(s) for s in shapes]
        chk(L.ocfd_gpu_init_state(dp(prim), dp(case.di), 0.0))
        chk(L.ocfd_gpu_download_state(*[dp(b) for b in self.start]))
        self.case = case

    def run(self):
        L, dp, chk = solver.lib(), abi.dptr, solver._chk
        s = self.solver
        if not _open or _open[1] is not s:
            raise RuntimeError("the library's solver was opened for another case")
        chk(L.ocfd_gpu_upload_state(*[dp(b) for b in self.start]))
        s.tt = 0.0
        if self.c["steps"] == 1:
            s.step(self.case.dt, int(self.c["react"]), self.c["nsub"])
        else:
            s.run(self.case.dt, self.c["steps"], int(self.c["react"]), self.c["nsub"])
        chk(L.ocfd_gpu_download_state(*[dp(b) for b in self.out]))
        return {"f": self.out[0], "di": self.out[1], "prims": self.out[2]}


# ---------------------------------------------------------------- reactors

def _reactors(n, seed, nsub_max):
    _, th, kin, di, e, dt, nsub, _ = cases.reactors(n=n, seed=seed, nsub_max=nsub_max)
    return th, kin, di, e, dt, nsub


class Reactors:
    def __init__(self, c, seed):
        self.c = c
        th, kin, di, e, dt, nsub = _reactors(c["n"], seed, c["nsub_max"])
        _open.clear()  # the set-up replaces an open solver's chemistry tables
        solver.chem_setup(th, kin, 1, abi.CHEM_IMPLICIT, const_p=c["const_p"])
        if c["device"]:
            self.d = [torch.from_numpy(a).cuda() for a in (di, e, dt, nsub)]
            self.di, self.e = torch.empty_like(self.d[0]), torch.empty_like(self.d[1])
        else:
            self.d = [di, e, dt, nsub]
            self.di, self.e = np.empty_like(di), np.empty_like(e)

    def run(self):
        if self.c["device"]:
            self.di.copy_(self.d[0])
            self.e.copy_(self.d[1])
            torch.cuda.current_stream().synchronize()  # the library works on its own stream
            solver.chem_batch_device(self.c["n"], self.di.data_ptr(), self.e.data_ptr(), self.d[2].data_ptr(),
                                self.d[3].data_ptr())
        else:
            self.di[...] = self.d[0]
            self.e[...] = self.d[1]
            solver.chem_batch(self.di, self.e, self.d[2], self.d[3])
        return {"di": self.di, "e": self.e}


# ---------------------------------------------------------------- the learned surrogate

NET = ((256, 16), (256, 256), (256, 256), (16, 256))  # layer shapes, padded input and output
ELEMENTS = (("O", 15.9994e-3), ("H", 1.00794e-3), ("N", 14.0067e-3))
ATOMS = {"O": (1, 0, 0), "O2": (2, 0, 0), "H2": (0, 2, 0), "H2O": (1, 2, 0), "OH": (1, 1, 0), "H": (0, 1, 0),
         "HO2": (2, 1, 0), "H2O2": (2, 2, 0), "N2": (0, 0, 2)}


def _network(names, mi):
    """A trained network's parts as a program loads them: weights and biases, the normalisation of
    the reactors' ranges, the element projection. The weights are seeded random ones at a trained
    network's scale; the increments they give are those of the reactors (mass fractions 1e-4,
    temperature a few kelvin)."""
    rng = np.random.default_rng(20)
    ns = len(names)
    layers = []
    for l, (r, k) in enumerate(NET):
        W, b = np.zeros((r, k), np.float32), np.zeros(r, np.float32)
        rows, cols = (ns + 1 if l == 3 else r), (ns + 3 if l == 0 else k)
        W[:rows, :cols] = rng.standard_normal((rows, cols)) * math.sqrt((0.5 if l == 3 else 2.0) / cols)
        b[:rows] = 0.05 * rng.standard_normal(rows)
        layers.append((W, b))
    norm = np.zeros((6, 16), np.float32)  # input mean, std; output mean, std; input min, max
    norm[1], norm[3], norm[4], norm[5] = 1.0, 0.0, -1e30, 1e30
    norm[0, :2], norm[1, :2] = (1550.0, 11.5), (375.0, 0.5)
    norm[0, 2:2 + ns], norm[1, 2:2 + ns] = 0.1, 0.1
    norm[0, 2 + ns], norm[1, 2 + ns] = -16.0, 1.3
    norm[3, :ns] = [1e-4 if s in ("O2", "H2", "H2O") else 1e-8 for s in names]
    norm[3, names.index("N2")] = 0.0
    norm[3, ns] = 2.0
    G = np.array([[ATOMS[s][e] * m / mi[k] for k, s in enumerate(names)] for e, (_, m) in enumerate(ELEMENTS)])
    proj = np.eye(ns) - G.T @ np.linalg.solve(G @ G.T, G)
    return layers, norm, proj


def _blob(layers, norm, proj):
    full = np.zeros(256)
    full[:proj.size] = proj.ravel()
    return np.ascontiguousarray(np.concatenate([np.concatenate([W.ravel(), b]) for W, b in layers]
                                               + [norm.ravel(), full.view(np.float32)]))


class Network:
    TOL_T = 1.0e6  # K: a gate that every reactor passes (the real one rejects about one in 2^20)

    def __init__(self, c, seed):
        self.c = c
        th, kin, di, e, dt, nsub = _reactors(c["n"], seed, 100)
        names = cases.h2air_structs()[0]
        _open.clear()
        solver.chem_setup(th, kin, 1, abi.CHEM_IMPLICIT)
        self.L = solver.lib()
        layers, norm, self.proj = _network(names, np.array([th.mi[k] for k in range(len(names))]))
        solver._chk(self.L.ocfd_gpu_surrogate_init(1))
        # every radical a thousandth of a mass fraction: the increments stay inside the gate
        for s in ("O", "OH", "H", "HO2", "H2O2"):
            di[:, names.index(s)] += 1.0e-3 * di.sum(axis=1)
        self.d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (di, e, dt, nsub)]
        self.fp = C.POINTER(C.c_float)
        if c["train"]:
            # target states: a smooth change of a per mille of the densities and the energy (an
            # integrator's states would carry its rounding into every weight)
            self.d1, self.e1 = self.d[0].clone(), self.d[1].clone()
            scale = 1.0 + 1.0e-3 * torch.tanh(self.d[0] / self.d[0].sum(1, keepdim=True) - 0.1)
            self.d1.mul_(scale)
            self.e1.mul_(1.001)
            torch.cuda.synchronize()
            self.proj = np.ascontiguousarray(self.proj)
            self.loss = np.zeros(1)
            self.blob = np.zeros(self.L.ocfd_gpu_surrogate_blob(None, 0, 0), np.float32)
        else:
            blob = _blob(layers, norm, self.proj)
            if self.L.ocfd_gpu_surrogate_blob(blob.ctypes.data_as(self.fp), blob.size, 1) != 0:
                raise RuntimeError("surrogate blob")
            self.di, self.e = torch.empty_like(self.d[0]), torch.empty_like(self.d[1])

    def run(self):
        chk, n = solver._chk, self.c["n"]
        ptr = [t.data_ptr() for t in self.d]
        if self.c["train"]:
            chk(self.L.ocfd_gpu_surrogate_train(n, ptr[0], ptr[1], ptr[2], self.d1.data_ptr(), self.e1.data_ptr(),
                                                abi.dptr(self.proj), 1, self.c["batch"], 1.0e-3, 7,
                                                abi.dptr(self.loss)))
            if self.L.ocfd_gpu_surrogate_blob(self.blob.ctypes.data_as(self.fp), self.blob.size, 0) != 0:
                raise RuntimeError("surrogate blob")
            split = sum(r * k + r for r, k in NET)
            return {"weights": self.blob[:split], "norm": self.blob[split:split + 96], "loss": self.loss}
        self.di.copy_(self.d[0])
        self.e.copy_(self.d[1])
        torch.cuda.current_stream().synchronize()
        nfb = C.c_int()
        chk(self.L.ocfd_gpu_chem_batch_surrogate(n, self.di.data_ptr(), self.e.data_ptr(), ptr[2], ptr[3], self.TOL_T,
                                                 C.byref(nfb)))
        return {"di": self.di, "e": self.e, "fallback": nfb.value}


KINDS = {"flow": Flow, "reactors": Reactors, "network": Network}


def prepare(case, seed):
    return KINDS[case["kind"]](dict(case), seed)


def run(state):
    return state.run()


# ---------------------------------------------------------------- the work of a pass

def work(c):
    """Operations: the schemes' own counts per cell and right-hand side (a division, square root or
    exponential as one). Bytes of a flow run: the conserved state in and out of every right-hand
    side (no state of interest stays on chip between them); elsewhere inputs and outputs once."""
    if c["kind"] == "flow":
        cells, ns = c["nx"] * c["ny"] * c["nz"], c["species"]
        rec = {"WENO5": 50, "WENO7": 85, "OMP6": 45, "UD7L": 15, "HYBRID": 16}[c["scheme"]]
        nv = 5 + (ns if ns > 1 else 0)
        flops = 3 * (2 * nv * rec + 120 + 5 * nv) + 305 + 115 + 60
        if ns > 1:
            flops += ns * (2 * 18 * 3 + 20) + 3 * ns * (ns + 3) + 5 * ns * (ns - 1) // 2
        rhs = 6 * c["steps"]
        chem = (2000 + ns ** 3) * c["nsub"] * c["steps"] if c["react"] else 0
        return {"bytes": cells * 16.0 * nv * rhs, "flops": cells * (float(flops) * rhs + chem)}
    n = c["n"]
    if c["kind"] == "reactors":
        mean = {1: 1.0, 10: 6.7, 100: 22.0}[c["nsub_max"]]
        return {"bytes": n * (2.0 * 80 + 12), "flops": n * mean * 3000.0}
    per = 2.0 * sum(r * k for r, k in NET)
    return {"bytes": n * (2.0 * 80 + 8), "flops": n * per * (3 if c["train"] else 1)}


# ---------------------------------------------------------------- the same in plain 64-bit torch

def exact(case, seed):
    """64-bit restatements: the periodic one-species box with WENO5 / Steger-Warming / CD6 (its
    conserved fields), the batched reactors, the surrogate's inference. None elsewhere: the other
    flows branch per interface or carry several thousand lines of physics, and the training shuffles
    its samples inside the library."""
    c = case
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if c["kind"] == "flow":
        if (c["flow"], c["species"], c["scheme"], c["splitting"], c["vis"], c["char"]) != ("box", 1, "WENO5", "SW",
                                                                                       "CD6", False):
            return None
        return {"f": _exact_box(c, seed, dev), "di": None, "prims": None}
    th, kin, di, e, dt, nsub = _reactors(c["n"], seed, c.get("nsub_max", 100))
    if c["kind"] == "reactors":
        t = [torch.from_numpy(a).to(dev) for a in (di, e, dt, nsub)]
        return _exact_reactors(Gas(th, kin, dev), *t, c["const_p"])
    if c["train"]:
        return None
    names = cases.h2air_structs()[0]
    for s in ("O", "OH", "H", "HO2", "H2O2"):
        di[:, names.index(s)] += 1.0e-3 * di.sum(axis=1)
    gas = Gas(th, kin, dev)
    di, e, dt = (torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in (di, e, dt))
    layers, norm, proj = _network(names, gas.M.cpu().numpy())
    nm = torch.from_numpy(norm.astype(np.float64)).to(dev)
    ns = len(names)
    T = gas.temperature(di, e)
    rho = di.sum(1)
    x = torch.zeros(len(e), 16, dtype=torch.float64, device=dev)
    x[:, 0], x[:, 1], x[:, 2 + ns] = T, torch.log((di * gas.R).sum(1) * T), torch.log(dt)
    x[:, 2:2 + ns] = di / rho[:, None]
    h = (x - nm[0]) / nm[1]
    h[:, ns + 3:] = 0.0
    for l, (W, b) in enumerate(layers):
        h = h @ torch.from_numpy(W.astype(np.float64)).to(dev).T + torch.from_numpy(b.astype(np.float64)).to(dev)
        if l < 3:
            h = torch.nn.functional.gelu(h, approximate="tanh")
    dY = (h[:, :ns] * nm[3, :ns] + nm[2, :ns]) @ torch.from_numpy(proj).to(dev).T
    d1 = (di / rho[:, None] + dY) * rho[:, None]
    return {"di": d1, "e": e - ((d1 - di) * gas.R * gas.c[:, 0, 5]).sum(1), "fallback": None}


class Gas:
    """The mechanism's thermodynamics and kinetics from its tables, in torch."""

    def __init__(self, th, kin, dev):
        ns, nt = th.n_spec, th.n_tct
        f = lambda a: torch.tensor(np.array(a, dtype=np.float64), device=dev)  # noqa: E731
        self.ns, self.tct, self.tmax = ns, [th.tct[j] for j in range(nt - 1)], th.tct_max
        self.M = f([th.mi[k] for k in range(ns)])
        self.R = R0 / self.M
        self.c = f([[list(th.coef[k][j]) for j in range(nt)] for k in range(ns)])  # species, range, 7
        ect = torch.zeros(ns, nt, dtype=torch.float64, device=dev)
        for j in range(nt - 1):
            d, t = self.c[:, j + 1] - self.c[:, j], self.tct[j]
            ect[:, j + 1] = ect[:, j] - sum(d[:, m] * t ** (m + 1) / (m + 1) for m in range(5))
        self.ect = ect
        nr = kin.n_reac
        self.nr, self.at, self.tb = nr, list(kin.af_type)[:nr], list(kin.tr_reac)[:nr]
        self.af, self.bf, self.ef = ([list(a[j]) for j in range(nr)] for a in (kin.af, kin.bf, kin.ef))
        self.fc = list(kin.fc_troe)[:nr]
        self.vf = f([list(kin.vf[j])[:ns] for j in range(nr)])
        self.vr = f([list(kin.vr[j])[:ns] for j in range(nr)])
        self.eff = f([list(kin.treff[j])[:ns] for j in range(nr)])

    def _range(self, T):
        jc = torch.zeros_like(T, dtype=torch.long)
        for j, t in enumerate(self.tct):
            jc = torch.where(T > t, j + 1, jc)
        return jc

    def energy(self, di, T):
        """Internal energy of the densities di at T, and its derivative."""
        jc, Tm, w = self._range(T), T.clamp(max=self.tmax)[:, None], self.R * di
        c = self.c[:, jc].transpose(0, 1)  # reactor, species, 7
        e = (c[..., 0] - 1.0) * Tm + self.ect[:, jc].T
        cv = c[..., 0] - 1.0
        for m in range(1, 5):
            e = e + c[..., m] * Tm ** (m + 1) / (m + 1)
            cv = cv + c[..., m] * Tm ** m
        e = e + cv * (T[:, None] - Tm)
        return (w * e).sum(1), (w * cv).sum(1)

    def temperature(self, di, E):
        T = torch.full_like(E, 1200.0)
        for _ in range(14):
            e, cv = self.energy(di, T)
            T = T - (e - E) / cv
        return T

    def gibbs(self, T):
        """g_k / R of every species."""
        c, t, lt = self.c[:, self._range(T)].transpose(0, 1), T[:, None], torch.log(T)[:, None]
        g = c[..., 0] * (1.0 - lt) * t + c[..., 5] - c[..., 6] * t
        for m in range(1, 5):
            g = g - c[..., m] * t ** (m + 1) / (m * (m + 1))
        return g

    def rates(self, ci, T):
        """Molar rates and their Jacobian by the concentrations."""
        lt, g = torch.log(T), self.gibbs(T)
        ri = torch.zeros_like(ci)
        J = torch.zeros(len(T), self.ns, self.ns, dtype=torch.float64, device=T.device)
        rc = 1.0 / (ci + 1.0e-20)
        lct, lcn = float(np.float32(0.67)), float(np.float32(1.27))
        for j in range(self.nr):
            k = [self.af[j][s] * torch.exp(self.bf[j][s] * lt - self.ef[j][s] / T) for s in range(2)]
            M = ci @ self.eff[j]
            w = k[0]
            if self.at[j] == 2:
                w = k[0] + k[1]
            elif self.at[j] == 1:  # Troe fall-off
                pr, lf = k[0] / k[1] * M, math.log10(self.fc[j])
                ac, an = -0.4 - lct * lf, 0.75 - lcn * lf
                lp = torch.log10(pr) + ac
                w = k[1] * pr / (1.0 + pr) * 10.0 ** (lf / (1.0 + (lp / (an - 0.14 * lp)) ** 2))
            s = self.vr[j] - self.vf[j]
            kc = torch.exp(-(g @ s) / T) * (R0 / ATM * 1.0e6 * T) ** float(-s.sum())
            r = w / kc
            if self.tb[j] == 1 and self.at[j] != 1:
                w, r = w * M, r * M
            fw, bw = w * (ci ** self.vf[j]).prod(1), r * (ci ** self.vr[j]).prod(1)
            ri = ri + (fw - bw)[:, None] * s
            d = (self.vf[j] * fw[:, None] - self.vr[j] * bw[:, None]) * rc
            J = J + s[None, :, None] * d[:, None, :]
        return ri, J


def _exact_reactors(gas, di, e, dt, nsub, const_p):
    order = torch.argsort(nsub, descending=True)
    di, e = di.clone(), e.clone()
    F = gas.R * gas.c[:, 0, 5]
    if const_p:
        T = gas.temperature(di, e)
        p0 = (di * gas.R).sum(1) * T
        h0 = (e + (di * F).sum(1) + p0) / di.sum(1)
    step = dt / nsub
    for s in range(int(nsub.max())):
        live = order[: int((nsub > s).sum())]
        for rows in live.split(1 << 17):
            d, E = di[rows], e[rows]
            ri, J = gas.rates(d / gas.M * 1.0e-6, gas.temperature(d, E))
            h = step[rows][:, None]
            A = torch.eye(gas.ns, dtype=torch.float64, device=d.device) - J * (gas.M[:, None] / gas.M) * h[:, :, None]
            dn = d + torch.linalg.solve(A, ri * gas.M * 1.0e6 * h)
            E = E - ((dn - d) * F).sum(1)
            if const_p:
                Y = dn / dn.sum(1, keepdim=True)
                Rm, cf, T = (gas.R * Y).sum(1), (F * Y).sum(1), gas.temperature(dn, E)
                for _ in range(6):
                    ey, cv = gas.energy(Y, T)
                    T = T - (ey + Rm * T + cf - h0[rows]) / (cv + Rm)
                dn = Y * (p0[rows] / (Rm * T))[:, None]
                E = gas.energy(dn, T)[0]
            di[rows], e[rows] = dn, E
    return {"di": di, "e": e}


def _exact_box(c, seed, dev):
    """The conserved fields of the periodic perfect-gas box after the pass's steps: WENO5 on
    Steger-Warming fluxes, sixth-order viscous terms, SSP-RK3, two half steps per step."""
    case = _flow_case(c)
    n, hx = c["nx"], case.info["h"]
    prim = torch.from_numpy(_flow_inputs(c, seed, case)).to(dev)
    R, A = R0 / 0.029, (hx * (n - 1)) ** 2  # the face metric in computational space
    d, vel, T = prim[0], list(prim[1:4]), prim[4]
    f = torch.stack([d] + [d * v for v in vel] + [2.5 * R * d * T + 0.5 * d * sum(v * v for v in vel)])
    sh = lambda a, m, ax: torch.roll(a, -m, ax)  # noqa: E731  the value m cells up the axis

    def diff(a, ax):
        return (45.0 * (sh(a, 1, ax) - sh(a, -1, ax)) - 9.0 * (sh(a, 2, ax) - sh(a, -2, ax))
                + (sh(a, 3, ax) - sh(a, -3, ax))) / (60.0 * hx)

    def weno(a, b, m, p, q):  # value at the face after m from the five upwind-ordered fields
        S = [13.0 / 12.0 * (m - 2 * p + q) ** 2 + 0.25 * (3 * m - 4 * p + q) ** 2,
             13.0 / 12.0 * (b - 2 * m + p) ** 2 + 0.25 * (b - p) ** 2,
             13.0 / 12.0 * (a - 2 * b + m) ** 2 + 0.25 * (a - 4 * b + 3 * m) ** 2]
        w = [k / (1.0e-6 + s) ** 2 for k, s in zip((0.3, 0.6, 0.1), S)]
        v = [m / 3 + 5 * p / 6 - q / 6, -b / 6 + 5 * m / 6 + p / 3, a / 3 - 7 * b / 6 + 11 * m / 6]
        return (w[0] * v[0] + w[1] * v[1] + w[2] * v[2]) / (w[0] + w[1] + w[2])

    def rhs(f):
        d = f[0]
        vel = [f[m] / d for m in (1, 2, 3)]
        Et = f[4] - 0.5 * d * sum(v * v for v in vel)
        T = Et / (2.5 * R * d)
        p = R * d * T
        g = p / Et + 1.0
        cc = torch.sqrt(g * p / d)
        out = torch.zeros_like(f)
        for dim, ax in enumerate((2, 1, 0)):
            u = vel[dim]
            lam = [A * u, A * (u - cc), A * (u + cc)]
            for sign in (1, -1):
                E = [0.5 * (x + sign * x.abs()) for x in lam]
                up = [[v - cc if m == dim else v for m, v in enumerate(vel)],
                      [v + cc if m == dim else v for m, v in enumerate(vel)]]
                k = [0.5 * sum(x * x for x in w) for w in up]
                t1, t0, W = 2.0 * (g - 1.0), d / (2.0 * g), (3.0 - g) / (2.0 * (g - 1.0)) * cc * cc
                F = [t0 * (t1 * E[0] + E[1] + E[2])]
                F += [t0 * (t1 * E[0] * vel[m] + E[1] * up[0][m] + E[2] * up[1][m]) for m in range(3)]
                F += [t0 * (E[0] * (g - 1.0) * sum(v * v for v in vel) + E[1] * k[0] + E[2] * k[1] + W * (E[1] + E[2]))]
                F = torch.stack(F)
                x = ax + 1
                if sign > 0:
                    h = weno(*[sh(F, m, x) for m in (-2, -1, 0, 1, 2)])
                else:
                    h = weno(*[sh(F, m, x) for m in (3, 2, 1, 0, -1)])
                out -= (h - sh(h, -1, x)) / (hx * A)
        gr = [[diff(a, ax) for ax in (2, 1, 0)] for a in vel + [T]]
        mu = 1.789e-5 * torch.sqrt((T / 288.15) ** 3) * (288.15 + 110.4) / (110.4 + T)
        kap, div = mu * 3.5 * R / 0.7, gr[0][0] + gr[1][1] + gr[2][2]
        s = [[mu * (gr[a][b] + gr[b][a] - (2.0 / 3.0 * div if a == b else 0.0)) for b in range(3)] for a in range(3)]
        for dim, ax in enumerate((2, 1, 0)):
            for m in range(3):
                out[1 + m] += diff(s[m][dim], ax)
            out[4] += diff(sum(vel[m] * s[m][dim] for m in range(3)) + kap * gr[3][dim], ax)
        return out

    dt = 0.5 * case.dt
    for _ in range(2 * c["steps"]):
        f0 = f
        f = f0 + dt * rhs(f0)
        f = 0.75 * f0 + 0.25 * (f + dt * rhs(f))
        f = f0 / 3.0 + 2.0 / 3.0 * (f + dt * rhs(f))
    return f
