"""Workloads of the time step at the sizes a program uses it at, each as one timed pass.

A pass restarts its runs from orbitals on the device, advances them ``steps`` steps (a window at the
centre of their pulses) and reads back the per-l dipole, acceleration and norm series, the final
orbitals and, where the density acts back, the potentials, all into device buffers through the C ABI.
The calls of ``ggb_observables_noalloc`` stand beside them.

Case fields: ``groups`` lists the grid groups as atom:N_r x N_l:runs; ``form`` is the precision form;
``angular`` the theta form or the reference's coupling chain; ``n_har`` the multipoles of the Hartree
potential; ``potentials`` adiabatic (they follow the density) or frozen (held at the ground state);
``calls`` the number of step() calls that share the steps.
"""
import ctypes
import dataclasses
import functools
import math

import numpy as np
import torch

from ggbtddft_b200 import engine
from ggbtddft_b200 import inputs as I
from ggbtddft_b200 import problems as P

DT = {"H": 0.05, "He": 0.03, "Ne3": 0.02, "Ar": 0.02}
LARGEST = 16 * 189 * 161 * 1000 ** 2          # steps x columns x N_l x N_r^2 of the largest listed case


def _steps(name, groups, form, angular, n_har, potentials, steps, calls=1):
    return dict(name=name, op="steps", groups=groups, form=form, angular=angular, n_har=n_har,
                potentials=potentials, steps=steps, calls=calls)


def listed():
    return [
        # observables of nine orbitals inside another framework's memory pool: one call
        dict(name="observables-ar9", op="observables", n_r=600, n_l=97, n_orb=9),
        # the hydrogen configuration, whole window in one call, and advanced one step at a time by a
        # program that looks in between: launches and latency
        _steps("h-fp64", "H:200x33:1", "fp64", "theta", 2, "frozen", 96),
        _steps("h-fp64-single-steps", "H:200x33:1", "fp64", "theta", 2, "frozen", 24, calls=24),
        # the helium configuration with every multipole L = 0 .. 2 l_max
        _steps("he-fp64-multipoles", "He:400x65:1", "fp64", "theta", 129, "adiabatic", 64),
        # all-electron argon in the parity form
        _steps("ar-fp64", "Ar:600x97:1", "fp64", "theta", 4, "adiabatic", 40),
        # the reference's own coupling chain with every coupling active, odd sizes
        _steps("ne3-fp64-chain", "Ne3:253x49:1", "fp64", "reference", 4, "adiabatic", 48),
        # the fast form: one argon run alone
        _steps("ar-int8-one", "Ar:600x97:1", "split_int8", "theta", 4, "frozen", 64),
        # the smallest grid group of the 64-run argon scan (10 runs), and the largest (21 runs)
        _steps("ar-int8-10runs", "Ar:600x97:10", "split_int8", "theta", 4, "frozen", 32),
        _steps("ar-int8-21runs", "Ar:1000x161:21", "split_int8", "theta", 4, "frozen", 16),
        # the lower rungs of the hydrogen / helium focal scan: grid groups on concurrent streams
        _steps("hhe-int8-scan", "H:200x33:20 He:200x33:21 H:400x65:46 He:400x65:47", "split_int8", "theta", 4,
               "adiabatic", 32),
        # the fast form on the reference's coupling chain, odd sizes
        _steps("ne3-int8-chain", "Ne3:331x61:4", "split_int8", "reference", 4, "adiabatic", 48),
    ]


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    if rng.random() < 0.12:
        while True:
            c = dict(op="observables", n_r=log_int(64, 1000), n_l=log_int(17, 161), n_orb=rng.randint(1, 16))
            if c["n_orb"] * c["n_l"] * ((c["n_r"] + 31) // 32) <= 65536:
                return c
    while True:
        form = rng.choice(["fp64", "split_int8"])
        angular = "reference" if rng.random() < 0.3 else "theta"
        atom = "Ne3" if angular == "reference" else rng.choice(["H", "He", "Ar"])
        n_r = log_int(200 if atom == "Ar" else 64, 1000)
        n_l = log_int(17, 161)
        runs = 1 if form == "fp64" else log_int(1, 47)
        groups = "%s:%dx%d:%d" % (atom, n_r, n_l, runs)
        cols = runs * {"H": 1, "He": 1, "Ne3": 3, "Ar": 9}[atom]
        cost = cols * n_l * n_r ** 2
        if atom in ("H", "He") and form == "split_int8" and rng.random() < 0.5:
            n_r2, n_l2, other = log_int(64, 400), log_int(17, 65), log_int(1, 47)
            groups += " %s:%dx%d:%d" % ("He" if atom == "H" else "H", n_r2, n_l2, other)
            cost += other * n_l2 * n_r2 ** 2
        potentials = "frozen" if atom == "H" else "adiabatic" if atom == "Ne3" else rng.choice(["frozen", "adiabatic"])
        n_har = 2 * n_l - 1 if atom == "He" and potentials == "adiabatic" and runs <= 4 and n_l <= 97 and " " not in groups else 4
        steps = log_int(6, 64)
        if steps * cost <= LARGEST:
            return dict(op="steps", groups=groups, form=form, angular=angular, n_har=n_har, potentials=potentials,
                        steps=steps, calls=1)


# --------------------------------------------------------------------------------------- inputs

def _groups(case):
    for text in case["groups"].split():
        atom, size, runs = text.split(":")
        n_r, n_l = size.split("x")
        yield atom, int(n_r), int(n_l), int(runs)


@functools.lru_cache(maxsize=8)
def _atom_on_grid(atom, n_r, n_l, absorber):
    """The run of one atom on one grid (r_max = N_r / 2, as on the ladders) with its ground state and
    radial propagators; the lasers and the starting orbitals are drawn per run."""
    r_max = 0.5 * n_r
    grid = I.make_grid(n_r, r_max, I.zeta_physical_to_ref(0.5, r_max))
    if atom == "Ne3":
        z, orbitals, interacting, corr = 8.0, [I.Orbital(1, 0, 0, 2), I.Orbital(2, 1, 0, 2), I.Orbital(2, 1, 1, 4)], True, False
    else:
        a = P.ATOMS[atom]
        z, orbitals, interacting, corr = a.Z, a.orbitals, a.interacting, a.correlation
    device = "cuda" if torch.cuda.is_available() else None
    gs = I.ground_state(grid, z, orbitals, interacting=interacting, correlation=corr, iterations=60, device=device)
    return P.build_run(grid, n_l, DT[atom], gs, np.zeros(1), absorber=absorber, cap_r_mask=r_max / 1.5,
                       mask_width=0.2 * r_max, xc_correlation=corr, name="%s-N%d-L%d" % (atom, n_r, n_l - 1),
                       target_id=1 if interacting else 0, device=device)


def _runs(case, seed):
    """[(the group's runs, their starting orbitals [run][l][kso][r])] from the seed alone."""
    rng = np.random.default_rng(seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    out = []
    for atom, n_r, n_l, count in _groups(case):
        base = _atom_on_grid(atom, n_r, n_l, "cap" if case["angular"] == "reference" else "mask")
        hartree = atom != "H" and case["potentials"] == "adiabatic"
        g = base.grid
        weight = torch.from_numpy(np.sqrt(g.drdx) / np.abs(g.P)).to(dev)      # DVR coefficient per function value
        r, bound = torch.from_numpy(g.r).to(dev), torch.from_numpy(base.x0).to(dev)
        l, l0, m = np.arange(n_l)[:, None], base.l_active[None, :], base.m_active[None, :]
        runs, x0 = [], torch.empty((count,) + base.x0.shape, dtype=torch.complex128, device=dev)
        for i in range(count):
            laser = P.LaserSpec(rng.uniform(0.8e14, 2.0e14), rng.uniform(800.0, 1300.0), 6.0, rng.uniform(0.0, 6.28))
            n_t = I.steps_for_sin2(base.dt, laser.omega, laser.cycles)
            first = n_t // 2 - case["steps"] // 2
            E = I.field_sin2(n_t, base.dt, laser.e0, laser.omega, laser.cycles, laser.cep)[first:first + case["steps"]]
            runs.append(dataclasses.replace(base, E=E, use_hartree=1 if hartree else 0, angular=case["angular"],
                                            n_har=case["n_har"] if hartree else min(case["n_har"], 4)))
            # the ground state and, as at the centre of a pulse, outgoing packets over the l above it
            centre, width, k = (torch.from_numpy(rng.uniform(a, b, base.n_orb)).to(dev)[:, None]
                                for a, b in ((0.02 * g.r_max, 0.3 * g.r_max), (0.05 * g.r_max, 0.15 * g.r_max), (-1.0, 1.0)))
            packet = torch.exp(torch.complex(-((r - centre) / width) ** 2, k * r)) * r * weight
            packet = packet / torch.linalg.vector_norm(packet, dim=1, keepdim=True)
            amp = 0.3 * np.exp(-0.15 * np.abs(l - l0)) * rng.standard_normal((n_l, base.n_orb)) * (l >= m)
            x = bound + torch.from_numpy(amp).to(dev)[:, :, None] * packet[None]
            x0[i] = x / torch.sqrt((x.abs() ** 2).sum(dim=(0, 2)))[None, :, None]
        out.append((runs, x0))
    return out


def _observables_inputs(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    shape = (case["n_l"], case["n_orb"], case["n_r"])
    grid = I.make_grid(case["n_r"], 0.5 * case["n_r"], I.zeta_physical_to_ref(0.5, 0.5 * case["n_r"]))
    r = torch.from_numpy(grid.r).to(dev)
    x = torch.view_as_complex(torch.randn(shape + (2,), generator=gen, dtype=torch.float64, device=dev))
    x = x * torch.exp(-0.1 * torch.arange(shape[0], device=dev))[:, None, None] * (r * torch.exp(-0.05 * r))
    m = torch.from_numpy(rng.integers(0, 2, case["n_orb"]).astype(np.int32)).to(dev)
    x = x * (torch.arange(shape[0], device=dev)[:, None, None] >= m[None, :, None])
    x = x / torch.sqrt((x.abs() ** 2).sum(dim=(0, 2)))[None, :, None]
    return x.contiguous(), r, m


# --------------------------------------------------------------------------------------- a pass

def prepare(case, seed):
    if case["op"] == "observables":
        x, r, m = _observables_inputs(case, seed)
        return dict(case=case, fn=engine.load_library().ggb_observables_noalloc, x=x, r=r, m=m,
                    dip=torch.empty(x.shape[:2], dtype=torch.complex128, device=x.device),
                    acc=torch.empty(x.shape[:2], dtype=torch.complex128, device=x.device),
                    norm=torch.empty(x.shape[1], dtype=torch.float64, device=x.device))
    drawn = _runs(case, seed)
    flat = [r for runs, _ in drawn for r in runs]
    tp = engine.TimePropagation(flat, precision=case["form"], per_l=True, n_t=case["steps"])
    groups, i = [], 0
    for runs, x0 in drawn:
        n, r0, dev, k = len(runs), runs[0], x0.device, case["steps"]
        c128, f64 = dict(dtype=torch.complex128, device=dev), dict(dtype=torch.float64, device=dev)
        groups.append(dict(first=i, runs=runs, x0=x0, hartree=r0.use_hartree == 1 and r0.target_id > 0,
                           dip=torch.empty((n, r0.n_l, r0.n_orb, k), **c128), acc=torch.empty((n, r0.n_l, r0.n_orb, k), **c128),
                           norm=torch.empty((n, r0.n_orb, k), **f64), x=torch.empty((n, r0.n_l, r0.n_orb, r0.n_r), **c128),
                           v=torch.empty((n, 4, r0.n_r), **f64), vexc=torch.empty((n, r0.n_r), **f64)))
        i += n
    return dict(case=case, tp=tp, groups=groups)


def _at(t, i=None):
    """The address of a tensor, or of its entry i, on the device or the host."""
    return ctypes.c_void_p((t if i is None else t[i]).data_ptr() if isinstance(t, torch.Tensor) else t.ctypes.data)


def _ok(code):
    if code != 0:
        raise RuntimeError("libggbtddft: status %d" % code)


def run(state):
    if state["case"]["op"] == "observables":
        s = state
        n_l, n_orb, n_r = s["x"].shape
        _ok(s["fn"](s["x"].data_ptr(), s["r"].data_ptr(), s["m"].data_ptr(), n_l, n_orb, n_r, s["dip"].data_ptr(),
                    s["acc"].data_ptr(), s["norm"].data_ptr(), torch.cuda.current_stream().cuda_stream))
        return dict(dipole=s["dip"], acceleration=s["acc"], norm=s["norm"])
    tp, lib, n = state["tp"], state["tp"].lib, state["case"]["steps"]
    for g in state["groups"]:
        for i, r in enumerate(g["runs"]):
            _ok(lib.ggb_set_orbitals(tp.ctx, g["first"] + i, _at(g["x0"], i), _at(r.l_active), _at(r.m_active),
                                     _at(r.occ), _at(r.rho_frozen)))
    calls = state["case"]["calls"]
    for c in range(calls):
        tp.step(n // calls)
    _ok(tp.status()[0])
    out = []
    for g in state["groups"]:
        for i in range(len(g["runs"])):
            k = g["first"] + i
            _ok(lib.ggb_get_observables(tp.ctx, k, _at(g["dip"], i), _at(g["acc"], i), _at(g["norm"], i), 1, n))
            _ok(lib.ggb_get_orbitals(tp.ctx, k, _at(g["x"], i)))
            if g["hartree"]:
                _ok(lib.ggb_get_potentials(tp.ctx, k, _at(g["v"], i), None, _at(g["vexc"], i), None))
        out.append({k: g[k] for k in ("dip", "acc", "norm", "x") + (("v", "vexc") if g["hartree"] else ())})
    return out


def work(case):
    """One step reads W and the orbitals once and writes the orbitals once (the steps follow one
    another), multiplies by W and by two or more rotations per half-step, and its series are written."""
    if case["op"] == "observables":
        n = case["n_l"] * case["n_orb"] * case["n_r"]
        return {"bytes": 16.0 * n + 8.0 * case["n_r"] + 32.0 * case["n_l"] * case["n_orb"], "flops": 28.0 * n}
    bytes_, flops = 0.0, 0.0
    for atom, n_r, n_l, runs in _groups(case):
        cols = runs * {"H": 1, "He": 1, "Ne3": 3, "Ar": 9}[atom]
        hartree = atom != "H" and case["potentials"] == "adiabatic"
        rotations = 2 if case["angular"] == "theta" or not hartree else 5
        elems = n_l * cols * n_r
        flop = 8.0 * n_r * elems + 2 * rotations * 4.0 * n_l * elems + 28.0 * elems
        if hartree and case["n_har"] > 4:
            flop += 4.0 * n_l * elems + 4.0 * n_l * case["n_har"] * n_r * runs
        bytes_ += case["steps"] * ((16.0 if case["form"] == "fp64" else 8.0) * n_l * n_r ** 2 + 32.0 * elems
                                   + 32.0 * n_l * cols)
        flops += case["steps"] * flop
    return {"bytes": bytes_, "flops": flops}


# --------------------------------------------------------------------------------------- in 64 bits

def _c(l, m):
    return np.sqrt(np.where(l >= m, ((l + 1.0) ** 2 - m ** 2) / ((2 * l + 1.0) * (2 * l + 3.0)), 0.0))


def _observe(x, r, m):
    """<x_l | r (c_l x_(l+1) + c_(l-1) x_(l-1))>, the same with r^-2, and the norm, of x[l][kso][r]."""
    n_l = x.shape[0]
    l, mm = np.arange(n_l, dtype=np.float64)[:, None], np.asarray(m, dtype=np.float64)[None, :]
    cu = torch.from_numpy(_c(l, mm)).to(x.device)[:, :, None]
    z = torch.zeros_like(x)
    z[:-1] += cu[:-1] * x[1:]
    z[1:] += cu[:-1] * x[:-1]
    p = x.conj() * z
    return (p * r).sum(-1), (p / r ** 2).sum(-1), (x.abs() ** 2).sum(dim=(0, 2))


def _l_sums(x, m, occ, n_den):
    """The density's multipoles L < 4 in l space of one run, with the octupole's count of l = N_l - 4 twice."""
    n_l, dev = x.shape[0], x.device
    l = np.arange(n_l, dtype=np.float64)
    out = torch.zeros((4, x.shape[2]), dtype=torch.float64, device=dev)
    for k in range(x.shape[1]):
        q, y = float(m[k]), x[:, k]
        with np.errstate(all="ignore"):
            ok = l >= q
            sq = [(l + s) ** 2 - q * q for s in (1.0, 2.0, 3.0)]
            c = _c(l, q)
            p2 = np.where(ok & (l >= 1), (l * (l + 1) - 3 * q * q) / ((2 * l - 1) * (2 * l + 3)), 0.0)
            q2 = np.where(ok, 1.5 / (2 * l + 3) * np.sqrt(sq[0] * sq[1] / ((2 * l + 1) * (2 * l + 5))), 0.0)
            p3 = np.where(ok, 1.5 * (l * (l + 2) - 5 * q * q) / (2 * l - 1) / (2 * l + 5)
                          * np.sqrt(sq[0] / (2 * l + 1) / (2 * l + 3)), 0.0)
            f3 = np.where(ok, 2.5 / (2 * l + 3) / (2 * l + 5) * np.sqrt(sq[0] * sq[1] * sq[2] / (2 * l + 1) / (2 * l + 7)), 0.0)

        def pair(d, coef):
            """coef(l) x_(l+d).x_l over l"""
            return torch.from_numpy(coef[:n_l - d]).to(dev) @ (y[d:].conj() * y[:n_l - d]).real

        d = [pair(0, ok.astype(np.float64)), 2 * pair(1, c), 2 * pair(2, q2) + pair(0, p2), 2 * pair(1, p3) + 2 * pair(3, f3)]
        t = n_l - 4
        d[3] = d[3] + (f3[t - 3] * y[t - 3] + p3[t - 1] * y[t - 1] + p3[t] * y[t + 1]).conj().mul(y[t]).real
        for L in range(n_den):
            out[L] += float(occ[k]) * d[L]
    return out


def _exchange(run, rho0, clamp):
    r, drdx, p = (torch.from_numpy(a).to(rho0.device) for a in (run.grid.r, run.grid.drdx, run.grid.P))
    n_g = run.n_r + 1
    den = n_g * (n_g + 1) / 2.0 * (rho0 / 4.0 / math.pi + torch.from_numpy(run.rho_frozen).to(rho0.device)) / drdx * p ** 2
    den = den.clamp(min=0.0) if clamp else den
    v = -(3.0 / math.pi * den) ** (1.0 / 3.0) / r ** (2.0 / 3.0)
    if run.xc_correlation:
        a, a1, b1, b2, b3, b4 = 0.031091, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294
        rs = (3.0 / (4.0 * math.pi * (den / r ** 2).clamp(min=1e-300))) ** (1.0 / 3.0)
        s = rs.sqrt()
        q0, q1 = -2 * a * (1 + a1 * rs), 2 * a * (b1 * s + b2 * rs + b3 * rs * s + b4 * rs * rs)
        q1p, lg = a * (b1 / s + 2 * b2 + 3 * b3 * s + 4 * b4 * rs), torch.log1p(1.0 / q1)
        v = v + q0 * lg - rs / 3.0 * (-2 * a * a1 * lg - q0 * q1p / (q1 * q1 + q1))
    return v


class _Exact:
    """One grid group propagated in complex128 with dense products."""

    def __init__(self, case, runs, x0):
        self.runs, self.r0, dev = runs, runs[0], x0.device
        r0 = self.r0
        self.n_l, self.n_orb, self.hartree = r0.n_l, r0.n_orb, r0.use_hartree == 1 and r0.target_id > 0
        self.x = x0.permute(1, 0, 2, 3).reshape(r0.n_l, -1, r0.n_r).clone()      # [l][run, kso][r]
        self.W = torch.from_numpy(r0.W).to(dev)
        self.r = torch.from_numpy(r0.grid.r).to(dev)
        self.E = torch.from_numpy(np.stack([q.E for q in runs])).to(dev)
        self.V = {c: torch.from_numpy(np.array(r0.V[c][:r0.n_m])).to(dev) for c in r0.V}
        self.D = {c: torch.from_numpy(np.array(r0.D[c][:r0.n_m])).to(dev) for c in r0.D}
        self.theta, self.n_har = r0.angular == "theta", r0.n_har
        n_v = self.n_har if self.theta else min(self.n_har, 4)
        self.v = torch.zeros((len(runs), max(n_v, 4), r0.n_r), dtype=torch.float64, device=dev)
        self.s = torch.zeros((len(runs), r0.n_r), dtype=torch.float64, device=dev)
        if self.hartree:
            small, big = torch.minimum(self.r[:, None], self.r[None]), torch.maximum(self.r[:, None], self.r[None])
            self.kernel = torch.stack([torch.exp(L * torch.log(small / big)) / big for L in range(n_v)])
            if self.theta:
                self.PL = {m: torch.from_numpy(self._legendre(r0.D["P"][m], n_v)).to(dev) for m in range(r0.n_m)}
            if self.theta and self.n_har > 4:
                xq, wq = np.polynomial.legendre.leggauss(2 * self.n_l)
                self.wP = torch.from_numpy(self._legendre(xq, n_v) * wq).to(dev)
                self.T = [torch.from_numpy(self._normalised(xq, m)).to(dev).to(torch.complex128) for m in range(r0.n_m)]
            self.vexc = torch.zeros_like(self.s)
            self._potentials(first=True)

    @staticmethod
    def _legendre(x, n):
        p = [np.ones_like(x), x]
        for L in range(1, n - 1):
            p.append(((2 * L + 1) * x * p[L] - L * p[L - 1]) / (L + 1))
        return np.stack(p[:n])

    def _normalised(self, x, m):
        """[q][l] normalised associated Legendre functions of order m."""
        out = np.zeros((x.size, self.n_l))
        c2 = 0.5
        for k in range(1, m + 1):
            c2 *= (2 * k + 1.0) / (2.0 * k)
        out[:, m] = math.sqrt(c2) * (1 - x * x) ** (0.5 * m)
        c = _c(np.arange(self.n_l, dtype=np.float64), float(m))
        for l in range(m, self.n_l - 1):
            out[:, l + 1] = (x * out[:, l] - (c[l - 1] * out[:, l - 1] if l > m else 0.0)) / c[l]
        return out

    def _potentials(self, first=False):
        for i, q in enumerate(self.runs):
            x = self.x[:, i * self.n_orb:(i + 1) * self.n_orb]
            rho = _l_sums(x, q.m_active, q.occ, min(self.n_har, 4))
            if self.theta and self.n_har > 4:
                dens = sum(float(q.occ[k]) * ((self.T[int(q.m_active[k])] @ x[:, k]).abs() ** 2) for k in range(self.n_orb))
                rho = torch.cat([rho[:1], (self.wP @ dens)[1:]])
            n = self.kernel.shape[0]
            self.v[i, :n] = (self.kernel @ rho[:n, :, None])[:, :, 0]
            if first:
                self.v00 = [] if i == 0 else self.v00
                self.v00.append((self.v[i, 0].clone(), _exchange(q, rho[0], False)))
            self.vexc[i] = _exchange(q, rho[0], True)
            self.s[i] = self.v[i, 0] - self.v00[i][0] + self.vexc[i] - self.v00[i][1]

    def _rotate(self, x, coupling, eta):
        """x <- V diag(exp(-i dt/2 eta)) V^T x of every column, eta(m) = [run][j][r]."""
        out = torch.zeros_like(x)
        for m in range(self.r0.n_m):
            ks = [k for k in range(self.n_orb) if int(self.r0.m_active[k]) == m]
            for i in range(len(self.runs)):
                cols = [i * self.n_orb + k for k in ks]
                V = self.V[coupling][m][m:, m:].to(torch.complex128)
                y = (V.T @ x[m:, cols].reshape(self.n_l - m, -1)).reshape(self.n_l - m, len(cols), -1)
                y = y * torch.exp(-0.5j * self.r0.dt * eta(m, i)[:, None, :])
                out[m:, cols] = (V @ y.reshape(self.n_l - m, -1)).reshape(self.n_l - m, len(cols), -1)
        return out

    def _half(self, x, t, second):
        def plain(coupling, values):
            return lambda m, i: self.D[coupling][m, m:, None] * values(i)[None, :]

        if self.theta:
            def eta(m, i):
                e = self.D["P"][m, m:, None] * (self.r * self.E[i, t])[None, :] + self.s[i][None, :]
                return e + self.PL[m][1:, m:].T @ self.v[i, 1:self.PL[m].shape[0]] if self.hartree else e
            return self._rotate(x, "P", eta)
        seq = [("P", lambda i: self.r * self.E[i, t] + self.v[i, 1])]
        if self.hartree and self.n_har >= 4:
            seq = [("FF", lambda i: self.v[i, 3]), ("FP", lambda i: self.v[i, 3]), ("D", lambda i: self.v[i, 2])] + seq
        if second:
            seq = seq[::-1]
            x = self._s_phase(x)
        for c, values in seq:
            x = self._rotate(x, c, plain(c, values))
        return x if second else self._s_phase(x)

    def _s_phase(self, x):
        if not self.hartree or self.n_har < 3:
            return x
        l, m = np.arange(self.n_l, dtype=np.float64)[:, None], self.r0.m_active.astype(np.float64)[None, :]
        p = np.where((l >= m) & (l >= 1), (l * (l + 1) - 3 * m * m) / ((2 * l - 1) * (2 * l + 3)), 0.0)
        p = torch.from_numpy(p).to(x.device).repeat(1, len(self.runs))
        s, v2 = (a.repeat_interleave(self.n_orb, dim=0)[None] for a in (self.s, self.v[:, 2]))
        return x * torch.exp(-0.5j * self.r0.dt * (s + p[:, :, None] * v2))

    def go(self, steps):
        n = len(self.runs)
        dip, acc, norm = [], [], []
        for t in range(steps):
            self.x = self._half(torch.matmul(self._half(self.x, t, False), self.W), t, True)
            if self.hartree:
                self._potentials()
            d, a, q = _observe(self.x, self.r, np.tile(self.r0.m_active, n))
            dip.append(d.reshape(self.n_l, n, -1).transpose(0, 1))
            acc.append(a.reshape(self.n_l, n, -1).transpose(0, 1))
            norm.append(q.reshape(n, -1))
        out = dict(dip=torch.stack(dip, -1), acc=torch.stack(acc, -1), norm=torch.stack(norm, -1),
                   x=self.x.reshape(self.n_l, n, self.n_orb, -1).transpose(0, 1).contiguous())
        if self.hartree:
            out.update(v=self.v[:, :4].contiguous(), vexc=self.vexc)
        return out


def exact(case, seed):
    if case["op"] == "observables":
        x, r, m = _observables_inputs(case, seed)
        d, a, n = _observe(x, r, m.cpu().numpy())
        return dict(dipole=d, acceleration=a, norm=n)
    return [_Exact(case, runs, x0).go(case["steps"]) for runs, x0 in _runs(case, seed)]
