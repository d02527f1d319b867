"""The work a program has the engine do, as timed cases: electrons from 4 to 128, one to thousands of
walkers, FP64 and mixed precision, through the Python binding of the C ABI (champ_b200.Engine).

A case is a dict: ``task`` (what one pass calls), ``system`` (which wave function) with its sizes,
``walkers`` and ``precision``.  ``prepare`` builds the wave function and the engine and puts
equilibrated walkers on the GPU; ``run`` is one pass; ``exact`` gives what an evaluation or a walk
through the single-electron calls returns, in plain FP64 torch.  A Metropolis or diffusion walk has no
such value: its accept decisions and copy counts are discrete.

FP32 precision (an E_L in FP32, outside the 1e-6 Ha bound of the other two) is not among the cases.
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from champ_b200 import system as S
from champ_b200.engine import Engine

SEED = 20261203


def listed():
    return [
        # the smallest job: a light atom, all electrons, few walkers -- a launch and its copies
        dict(name="be_vmc", task="vmc", system="be", walkers=256, nsweep=1, precision="fp64"),
        # a host program that walks electron by electron (the reference's hpsie / jassav+detsav calls)
        dict(name="dimer_steps", task="steps", system="dimer", nordc=4, walkers=500, precision="fp64"),
        # hpsi of walkers that a host program supplies: positions in, every result out
        dict(name="cluster5_eval", task="eval", system="cluster", centres=5, electrons=20, nordc=4, walkers=3001,
             precision="fp64"),
        # VMC of a pseudopotential dimer, the usual size of a benchmark molecule, in mixed precision
        dict(name="dimer_vmc", task="vmc", system="dimer", nordc=4, walkers=8192, nsweep=2, precision="mixed"),
        # the reference's C2 example with the reference's default mover (accelerated Metropolis)
        dict(name="c2_accel", task="accel", system="c2_example", walkers=8192, nsweep=1, precision="fp64"),
        # one sampling step of an optimisation of a multi-determinant wave function (515 parameters)
        dict(name="multidet_opt", task="opt", system="multidet", ndet=200, ncsf=60, walkers=16384, nsweep=1,
             precision="fp64"),
        # DMC at a production population
        dict(name="dimer_dmc", task="dmc", system="dimer", nordc=4, walkers=32768, nstep=4, tau=0.01, tmoves=0,
             precision="fp64"),
        # DMC of the C2 example with T-moves, as one runs it with a nonlocal pseudopotential
        dict(name="c2_dmc_tmoves", task="dmc", system="c2_example", walkers=4096, nstep=4, tau=0.02, tmoves=2,
             precision="fp64"),
        # a mid-sized open-shell molecule with a fifth-order Jastrow, walkers in no round number
        dict(name="cluster13_vmc", task="vmc", system="cluster", centres=13, electrons=51, nordc=5, walkers=1001,
             nsweep=2, precision="fp64"),
        # the headline workload of the benchmark: 128 electrons, mixed precision
        dict(name="cluster32_vmc", task="vmc", system="cluster", centres=32, electrons=128, nordc=4, walkers=4096,
             nsweep=1, precision="mixed"),
        # the same molecule driven by a host program that owns the walkers (host buffers in and out)
        dict(name="cluster32_host", task="host", system="cluster", centres=32, electrons=128, nordc=4, walkers=2048,
             nsweep=1, precision="fp64"),
        # one sampling step of its optimisation: 2064 parameters
        dict(name="cluster32_opt", task="opt", system="cluster", centres=32, electrons=128, nordc=4, walkers=1024,
             nsweep=0, precision="fp64"),
    ]


def draw(rng):
    """A case of the same ranges: any task over its systems, walkers over two to three decades."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    most = max(work(c)["flops"] for c in listed())
    while True:
        task = rng.choice(["vmc", "vmc", "vmc", "steps", "eval", "accel", "opt", "dmc", "host"])
        case = dict(task=task)
        kinds = {"vmc": ["be", "dimer", "multidet", "cluster", "cluster"], "steps": ["be", "dimer", "cluster"],
                 "eval": ["dimer", "cluster", "cluster"], "accel": ["c2_example", "dimer", "cluster"],
                 "opt": ["dimer", "multidet", "cluster"], "dmc": ["dimer", "c2_example"],
                 "host": ["dimer", "cluster", "cluster"]}[task]
        case["system"] = rng.choice(kinds)
        if case["system"] == "cluster":
            case["centres"] = rng.randint(3, 32)
            case["electrons"] = 4 * case["centres"] - rng.randint(0, 1)
        if case["system"] in ("cluster", "dimer"):
            case["nordc"] = rng.choice([0, 4, 4, 5]) if task in ("vmc", "host") else 4
        if case["system"] == "multidet":
            case["ndet"] = rng.randint(20, 200)
            case["ncsf"] = rng.randint(5, 20)
        case["walkers"] = log_int(50, {"dmc": 32768, "steps": 4096, "opt": 16384}.get(task, 8192))
        if task in ("vmc", "accel", "host"):
            case["nsweep"] = rng.randint(1, 3)
        if task == "opt":
            case["nsweep"] = 0
        if task == "dmc":
            case.update(nstep=rng.choice([2, 3, 4]), tau=0.01, tmoves=rng.choice([0, 0, 2]))
        case["precision"] = rng.choice(["fp64", "mixed"]) if task in ("vmc", "host") else "fp64"
        if work(case)["flops"] <= most:
            return case


# ---------------------------------------------------------------------------------------------
# wave functions
# ---------------------------------------------------------------------------------------------
def _terms(nord):
    """(k, l, m) of the e-e-n terms u^k (a^l + r^l) (a r)^m with k + l + 2m <= nord."""
    return [(k, l, (n - k - l) // 2) for n in range(2, nord + 1) for k in range(n - 1, -1, -1)
            for l in range(n - k - 2 if k == 0 else n - k, -1, -1) if (n - k - l) % 2 == 0]


def _cusp_free(c, nord):
    """The e-e-n coefficients nearest to c without a cusp at an electron or a centre."""
    t = _terms(nord)
    a = np.zeros((2 * nord + 1, len(t)))
    for i, (k, l, m) in enumerate(t):
        a[l + 2 * m, i] += k                  # slope in u where the two electrons meet
        a[nord + k + m, i] += l + m           # slope in r_i where electron i meets the centre
        a[nord + k + l + m, i] += m
    return c - np.linalg.pinv(a) @ (a @ c)


def _wave_function(case):
    kind = case["system"]
    if kind == "be":
        return S.be_atom()
    if kind == "c2_example":
        return S.c2_bfd_example()
    if kind == "multidet":
        return S.c2_multidet(ndet=case["ndet"], ncsf=case["ncsf"])
    if kind == "dimer":
        s = S.c2_dimer()
    else:
        nc, ne = case["centres"], case["electrons"]
        s = S.cluster128(ncent=nc, box=14.0 * (nc / 32) ** (1 / 3), norb=3 * nc)
        nup = (ne + 1) // 2
        s = dataclasses.replace(s, nelec=ne, nup=nup,
                                det_orb=np.array([list(range(nup)) + list(range(ne - nup))], np.int32))
    nord = case["nordc"]
    nt = len(_terms(nord))
    c = np.random.default_rng(77).uniform(-0.02, 0.02, nt)
    return dataclasses.replace(s, nordc=nord, een_cusp=1 if nt else 0,
                               c=_cusp_free(c, nord)[None] if nt else np.zeros((1, 0)))


def _walkers(sys, case, seed):
    return S.initial_walkers(sys, case["walkers"], seed=seed)


def _moves(sys, case, seed):
    """The single-electron moves a host program makes: new positions and accept masks per electron."""
    rng = np.random.default_rng([seed, 5])
    nw = case["walkers"]
    dx = sys.step * rng.standard_normal((sys.nelec, nw, 3))
    return dx, (rng.random((sys.nelec, nw)) < 0.6).astype(np.uint8)


def prepare(case, seed):
    sys = _wave_function(case)
    task, nw = case["task"], case["walkers"]
    eng = Engine(sys, int(1.6 * nw) + 64 if task == "dmc" else nw, case["precision"])
    x = _walkers(sys, case, seed)
    state = dict(case=case, eng=eng, sys=sys, seed=SEED + seed % 1000, sweep=0)
    if task == "eval":
        state["x"] = x
        return state
    eng.set_walkers(x)
    if task == "steps":
        dx, state["accept"] = _moves(sys, case, seed)
        state["xnew"] = [np.ascontiguousarray(x[:, e] + dx[e]) for e in range(sys.nelec)]
        return state
    if task == "accel":
        eng.set_mover(6)
    eng.vmc_sweeps(3, state["seed"], sweep0=0, step=sys.step, stats=False)  # equilibration
    state["sweep"] = 3
    if task == "host":
        state["x"] = eng.get_walkers()
    if task == "dmc":
        eng.set_option("tmoves", case["tmoves"])
        eng.dmc_init(nw, case["tau"])
        eng.dmc_steps(2, state["seed"])
        state["x"] = np.zeros((eng.w_max, eng.N, 3))  # where the program keeps a population of any size
    eng.synchronize()
    return state


def run(state):
    case, eng, task = state["case"], state["eng"], state["case"]["task"]
    if task in ("vmc", "accel"):
        # a block: sweeps, the block's statistics, and the walkers as a program saves them
        out = eng.vmc_sweeps(case["nsweep"], state["seed"], sweep0=state["sweep"], step=state["sys"].step)
        state["sweep"] += case["nsweep"]
        out["x"] = eng.get_walkers()
        return out
    if task == "host":
        x, el = eng.vmc_run_host(state["x"], case["nsweep"], state["seed"], sweep0=state["sweep"],
                                 step=state["sys"].step)
        return dict(x=x, energy=el)
    if task == "eval":
        eng.set_walkers(state["x"])
        return eng.eval_full()
    if task == "steps":
        ratio, grad = [], []
        for e in range(eng.N):
            r, g = eng.propose_1e(e, state["xnew"][e], grad=True)
            eng.accept_1e(e, state["accept"][e])
            ratio.append(r)
            grad.append(g)
        return dict(ratio=np.array(ratio), grad=np.array(grad))
    if task == "opt":
        if case["nsweep"]:
            eng.vmc_sweeps(case["nsweep"], state["seed"], sweep0=state["sweep"], step=state["sys"].step, stats=False)
            state["sweep"] += case["nsweep"]
        eng.param_grad(host=False)
        s, h = eng.accumulate_oh()
        return dict(S=s, H=h)
    stats = eng.dmc_steps(case["nstep"], state["seed"])
    x = state["x"]
    x[:eng.population()] = eng.get_walkers()
    x[eng.population():] = 0.0
    return dict(stats=stats, x=x)


def work(case):
    """Operations and bytes of one pass: FMAs count two, a primitive's exponential 20, a pair's
    distance and e-e polynomial 40."""
    kind = case["system"]
    # electrons, basis functions, primitives, occupied orbitals of a spin, centres, pseudopotential points
    n, nb, npr, no, nc, nq = {"be": (4, 7, 5, 2, 1, 0), "dimer": (8, 60, 72, 4, 2, 12), "multidet": (8, 60, 72, 16, 2, 12),
                              "c2_example": (8, 68, 36, 4, 2, 6)}.get(kind, (0,) * 6)
    if kind == "cluster":
        nc, n, nq = case["centres"], case["electrons"], 12
        nb, npr, no = 13 * nc, 15 * nc, (n + 1) // 2
    nord = case.get("nordc", 0 if kind == "be" else 4)
    mixed = sum((2 if l else 1) for k, l, m in _terms(nord) if m) and {0: 0, 4: 6, 5: 10}[nord]
    pairs = n * (n - 1) / 2
    row = 20 * npr + 2 * nb * no                            # one orbital row: values
    jrow = n * (40 + 2 * mixed * nc)                        # one electron's Jastrow pairs: values
    points = 0.6 * n * nq                                   # quadrature points of the tasks in range
    move = row + jrow + 2 * 4 * no * no
    move_grad = 20 * npr + 10 * nb * no + 4 * jrow + 8 * no * no
    evaluation = (n * (20 * npr + 10 * nb * no) + pairs * (80 + 2 * mixed * nc * 5) + 4 * n * no * no
                  + 2 * n * nb * no * (nq > 0) + points * (20 * npr + 2 * nb + jrow))
    if kind == "multidet":
        evaluation += case["ndet"] * 200
        move += case["ndet"] * 200
    w, task = case["walkers"], case["task"]
    xyz = 24 * n
    if task in ("vmc", "host"):
        f = case["nsweep"] * (n * move + evaluation)
        b = 2 * xyz + 32
    elif task == "accel":
        f = case["nsweep"] * (n * 2 * move_grad + evaluation)
        b = 2 * xyz + 32
    elif task == "eval":
        f = evaluation
        b = 2 * xyz + 8 * n + 64
    elif task == "steps":
        f = n * move_grad
        b = n * 57
    elif task == "dmc":
        f = case["nstep"] * (n * 2 * move_grad + evaluation + (points * (row + jrow) if case["tmoves"] else 0))
        b = 2 * xyz + 32
    else:
        p = {"dimer": 64, "multidet": 440 + 16 + case.get("ncsf", 1) - 1}.get(kind, 2 * nc * no + 16)
        f = case["nsweep"] * (n * move + evaluation) + 2 * evaluation + 4 * p * p + n * 4 * nb * 3 * nc
        b = xyz
        return {"bytes": float(w * b + 16 * (p + 1) ** 2), "flops": float(w * f)}
    return {"bytes": float(w * b), "flops": float(w * f)}


# ---------------------------------------------------------------------------------------------
# the same wave function in plain FP64 torch
# ---------------------------------------------------------------------------------------------
class _Psi:
    """ln|psi| of walkers x [W, N, 3]: Gaussian or Slater basis up to d, one determinant."""

    def __init__(self, s, dev):
        self.s, self.dev = s, dev
        t = self.t = lambda a: torch.as_tensor(np.asarray(a, float), dtype=torch.float64, device=dev)
        self.cent = t(s.cent)
        npr = s.shell_nprim
        self.ish = torch.as_tensor(np.repeat(np.arange(len(npr)), npr), device=dev)
        n, l, z = np.repeat(s.shell_n, npr), np.repeat(s.shell_l, npr), s.prim_zeta
        kind = np.repeat(s.shell_kind, npr)
        gauss = np.array([math.sqrt(math.pi) * math.prod(i - 0.5 for i in range(1, k + 1)) for k in n])
        fact = np.array([float(math.factorial(2 * k)) for k in n])
        norm = np.where(kind == 0, np.sqrt((2 * z) ** (2 * n + 1) * (2 * l + 1) / (fact * 4 * math.pi)),
                        np.sqrt(2 * (2 * z) ** (n + 0.5) * (2 * l + 1) / (gauss * 4 * math.pi)))
        self.z, self.w = t(z), t(s.prim_coef * norm)
        self.rpow = t(np.where(kind == 0, 1.0, 2.0))
        self.shc = torch.as_tensor(np.asarray(s.shell_cent, np.int64), device=dev)
        self.excess = [int(v) for v in s.shell_n - 1 - s.shell_l]   # R has r^(n-1), the harmonic r^-l
        self.basis = [(int(b), int(s.shell_l[b]), int(m)) for b, m in zip(s.basis_shell, s.basis_m)]
        self.coef = t(s.coef)
        self.sd = 1.0 / s.scalek

    def orbitals(self, x, orbs):
        d = x.unsqueeze(-2) - self.cent[self.shc]             # [..., shells, 3]
        r = d.square().sum(-1).sqrt()
        rp = torch.where(self.rpow == 1.0, r[..., self.ish], r[..., self.ish] ** 2)
        rad = torch.zeros_like(r).index_add(-1, self.ish, self.w * torch.exp(-self.z * rp))
        if any(self.excess):
            rad = rad * torch.stack([r[..., i] ** e for i, e in enumerate(self.excess)], -1)
        h3 = math.sqrt(3.0)
        col = []
        for b, l, m in self.basis:
            X, Y, Z = d[..., b, 0], d[..., b, 1], d[..., b, 2]
            y = {(0, 0): lambda: 1.0, (1, 0): lambda: Z, (1, 1): lambda: X, (1, -1): lambda: Y,
                 (2, 0): lambda: 0.5 * (2 * Z * Z - X * X - Y * Y), (2, 1): lambda: h3 * X * Z,
                 (2, -1): lambda: h3 * Y * Z, (2, 2): lambda: 0.5 * h3 * (X * X - Y * Y),
                 (2, -2): lambda: h3 * X * Y}[(l, m)]()
            col.append(rad[..., b] * y)
        return torch.stack(col, -1) @ self.coef[orbs].T

    def matrices(self, x):
        s = self.s
        det = np.asarray(s.det_orb[0], np.int64)
        return (self.orbitals(x[:, :s.nup], torch.as_tensor(det[:s.nup], device=self.dev)),
                self.orbitals(x[:, s.nup:], torch.as_tensor(det[s.nup:], device=self.dev)))

    def lndet(self, x):
        up, dn = self.matrices(x)
        a, b = torch.linalg.slogdet(up), torch.linalg.slogdet(dn)
        return a[1] + b[1], a[0] * b[0]

    def _en(self, r):
        s, a = self.s, self.s.a4[0]
        f = lambda u: a[0] * u / (1 + a[1] * u) + sum(a[k] * u ** k for k in range(2, s.norda + 1))  # noqa: E731
        return f(r / (1 + s.scalek * r)) - f(self.sd)

    def _pair(self, rij, par, ai, aj):
        """e-e and e-e-n terms; ai, aj [..., C]: 1 / (1 + scalek r) of the two electrons."""
        s, b = self.s, self.s.b[0]
        half = torch.where(par, 0.5, 1.0).to(torch.float64)
        u = rij / (1 + s.scalek * rij)
        ee = lambda v: half * b[0] * v / (1 + b[1] * v) + sum(b[k] * v ** k for k in range(2, s.nordb + 1))  # noqa: E731
        f = ee(u) - ee(torch.as_tensor(self.sd, dtype=torch.float64, device=self.dev))
        du = 1 / (1 + s.scalek * rij)
        for (k, l, m), c in zip(_terms(s.nordc), s.c[0]):
            f = f + c * du ** k * ((ai ** l + aj ** l) * (ai * aj) ** m).sum(-1)
        return f

    def jastrow(self, x):
        s = self.s
        i, j = torch.triu_indices(s.nelec, s.nelec, 1, device=self.dev)
        ren = (x[:, :, None] - self.cent).square().sum(-1).sqrt()
        a = 1 / (1 + s.scalek * ren)
        rij = (x[:, i] - x[:, j]).square().sum(-1).sqrt()
        return self._en(ren).sum((1, 2)) + self._pair(rij, (i < s.nup) == (j < s.nup), a[:, i], a[:, j]).sum(1)

    def lnpsi(self, x):
        return self.lndet(x)[0] + self.jastrow(x)

    def derivatives(self, x):
        """grad ln psi [W, N, 3] and lap_i ln psi [W, N]."""
        x = x.clone().requires_grad_(True)
        g, = torch.autograd.grad(self.lnpsi(x).sum(), x, create_graph=True)
        lap = torch.zeros(x.shape[:2], dtype=x.dtype, device=x.device)
        for e in range(x.shape[1]):
            for k in range(3):
                lap[:, e] += torch.autograd.grad(g[:, e, k].sum(), x, retain_graph=True)[0][:, e, k]
        return g.detach(), lap

    def nonlocal_energy(self, x, channel, v):
        """sum over electrons, centres and points of w v(r) psi(point)/psi (the s channel); v [W, N, C]."""
        s = self.s
        fi = 3.14159265359 / 5.0                               # the rule's own pi
        ct, st = 1 / math.sqrt(5), 2 / math.sqrt(5)
        q = [(0.0, 0.0, 1.0), (0.0, 0.0, -1.0)]
        q += [(st * math.cos(2 * i * fi), st * math.sin(2 * i * fi), ct) for i in range(5)]
        q += [(st * math.cos((2 * i + 1) * fi), st * math.sin((2 * i + 1) * fi), -ct) for i in range(5)]
        q = self.t(q)
        w, e, c = torch.nonzero(v.abs() > 1e-4, as_tuple=True)
        inv = [torch.linalg.inv(m) for m in self.matrices(x)]
        total = torch.zeros(x.shape[0], dtype=x.dtype, device=x.device)
        det = np.asarray(s.det_orb[0], np.int64)
        for lo in range(0, len(w), 4000):
            wi, ei, ci = w[lo:lo + 4000], e[lo:lo + 4000], c[lo:lo + 4000]
            xe = x[wi, ei]
            r = (xe - self.cent[ci]).square().sum(-1).sqrt()
            for p in range(12):
                pt = self.cent[ci] + r[:, None] * q[p]
                ratio = torch.zeros_like(r)
                for sp, (a, n0, n1) in enumerate(((inv[0], 0, s.nup), (inv[1], s.nup, s.nelec))):
                    at = torch.nonzero((ei >= n0) & (ei < n1)).squeeze(1)
                    phi = self.orbitals(pt[at], torch.as_tensor(det[n0:n1], device=self.dev))
                    ratio[at] = (phi * a[wi[at], :, ei[at] - n0]).sum(-1)
                aw = 1 / (1 + s.scalek * (x[wi][:, :, None] - self.cent).square().sum(-1).sqrt())
                other = torch.arange(s.nelec, device=self.dev) != ei[:, None]
                par = (torch.arange(s.nelec, device=self.dev) < s.nup) == (ei < s.nup)[:, None]
                f = []
                for y in (pt, xe):
                    ry = (y[:, None] - self.cent).square().sum(-1).sqrt()
                    ay = (1 / (1 + s.scalek * ry))[:, None].expand_as(aw)
                    ryj = (y[:, None] - x[wi]).square().sum(-1).sqrt()
                    ryj = torch.where(other, ryj, torch.ones_like(ryj))
                    f.append(self._en(ry).sum(-1) + torch.where(other, self._pair(ryj, par, ay, aw), 0.0).sum(-1))
                total.index_add_(0, wi, v[wi, ei, ci] / 12 * ratio * torch.exp(f[0] - f[1]))
        return total


def exact(case, seed):
    if case["task"] not in ("eval", "steps"):
        return None
    sys = _wave_function(case)
    if case["walkers"] * sys.nelec ** 3 * sys.ncent > 3e8:  # a pass per coordinate, each over all pairs and centres
        return None
    psi = _Psi(sys, "cuda" if torch.cuda.is_available() else "cpu")
    x = psi.t(_walkers(sys, case, seed))
    if case["task"] == "steps":
        dx, accept = _moves(sys, case, seed)
        x0, ratio, grad = x.clone(), [], []
        for e in range(sys.nelec):
            (l0, s0), j0 = psi.lndet(x), psi.jastrow(x)
            y = x.clone()
            y[:, e] = x0[:, e] + psi.t(dx[e])
            (l1, s1), j1 = psi.lndet(y), psi.jastrow(y)
            ratio.append((s0 * s1 * torch.exp(l1 - l0 + j1 - j0)).cpu().numpy())
            y.requires_grad_(True)
            grad.append(torch.autograd.grad(psi.lnpsi(y).sum(), y)[0][:, e].cpu().numpy())
            y = y.detach()
            x = torch.where(torch.as_tensor(accept[e], device=x.device).bool()[:, None, None], y, x)
        return dict(ratio=np.array(ratio), grad=np.array(grad))
    # div_v halves a pair's Laplacian between its electrons: not lap_i ln psi, no value here
    out = {k: [] for k in ("lnpsi", "sign", "psij", "velocity", "d2lnpsi", "pe", "pe_ee", "pe_nonloc", "energy")}
    chunk = max(1, int(2e8 // (sys.nelec ** 2 * sys.ncent * 40)))
    for y in torch.split(x, chunk):
        v, lap = psi.derivatives(y)
        (ld, sign), j = psi.lndet(y), psi.jastrow(y)
        i, k = torch.triu_indices(sys.nelec, sys.nelec, 1, device=y.device)
        ee = (1 / (y[:, i] - y[:, k]).square().sum(-1).sqrt()).sum(1)
        r = (y[:, :, None] - psi.cent).square().sum(-1).sqrt()
        vps = []
        for ch in range(2):
            f = sum(sys.ecp_coef[0, ch, t] * torch.exp(-sys.ecp_exponent[0, ch, t] * r * r)
                    for t in range(sys.necp_term[0, ch]))
            vps.append(f)
        a, b = np.triu_indices(sys.ncent, 1)
        nn = (sys.znuc[0] ** 2 / np.linalg.norm(sys.cent[a] - sys.cent[b], axis=1)).sum()
        nl = psi.nonlocal_energy(y, 0, vps[0])
        pe = nn + ee + (vps[1] - sys.znuc[0] / r).sum((1, 2)) + nl
        el = pe - 0.5 * (lap.sum(1) + v.square().sum((1, 2)))
        for key, val in zip(out, (ld + j, sign, j, v, lap.sum(1), pe, ee, nl, el)):
            out[key].append(val.cpu().numpy())
    return dict({k: np.concatenate(v) for k, v in out.items()}, div_v=None)
