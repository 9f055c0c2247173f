"""What this library's users have it do, as measurable cases.

A case is one call of Wstat's response operator (dng = sqvc chi0 sqvc dvg for m
perturbations, ``ResponseOperator.apply_operator``) or one PDEP Davidson solve
over it, on a Gamma-point ground state.  The ground state is what a user has on
disk before the run and is fixed by the case; the seed makes the perturbations
(or the Davidson's starting basis).  The context (``ResponseOperator``) is the
plan such a program keeps.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from west_b200.system import E2, FPI, SystemSpec, build_system, perturbations, randomized_basis
from west_b200.wstat import ResponseOperator

TR2 = 1e-10     # production PCG threshold (tr2_dfpt)
MAXITER = 250   # n_dfpt_maxiter


def _cell(L, ecut, n, natoms, nbnd, proj, system_seed):
    Ls, ns = (L if isinstance(L, tuple) else (L,) * 3), (n if isinstance(n, tuple) else (n,) * 3)
    return dict(L1=Ls[0], L2=Ls[1], L3=Ls[2], ecut=ecut, n1=ns[0], n2=ns[1], n3=ns[2], natoms=natoms, nbnd=nbnd,
                proj=proj, system_seed=system_seed)


# The cells of the repository's own workloads (west_b200/system.py, SPECS), and an orthorhombic one as QE boxes it.
SMALL = _cell(10.0, 8.0, 24, 3, 7, "sp", 12)
C1 = _cell(15.0, 20.0, 48, 4, 8, "s", 1)
C2 = _cell(20.0, 25.0, 64, 8, 32, "sp", 2)
C4C = _cell(25.0, 25.0, 80, 12, 64, "sp", 43)
C5 = _cell(30.0, 30.0, 108, 20, 128, "sp", 5)
ORTHO = _cell((16.0, 18.0, 21.0), 20.0, (45, 54, 60), 6, 20, "sp", 7)


def _apply(cell, m, form="fp64", host=False, tr2=TR2, **more):
    return dict(cell, do="apply", m=m, form=form, host=host, tr2=tr2, **more)


def listed():
    return [
        # A unit-test sized cell, one perturbation from host memory as the Fortran caller hands it over: launches
        # and waits are everything.
        _apply(SMALL, 1, host=True, name="small-m1-host"),
        # A small molecule's cell with the few perturbations that one of many images holds; odd, so that the last
        # pair is half empty.
        _apply(C1, 5, name="c1-m5"),
        # The PDEP solve of that cell as a whole: lite start, loose step, Davidson iterations over shrinking batches.
        dict(C1, do="davidson", m=16, form="fp64", host=True, tr2=TR2, name="c1-davidson-16"),
        # A medium cell, one perturbation: the reference's own order, and the last roots of a Davidson.
        _apply(C2, 1, name="c2-m1"),
        # The benchmark's call.
        _apply(C2, 64, name="c2-m64"),
        _apply(C2, 64, form="mixed", name="c2-m64-mixed"),
        # The lite solve (no PCG) that starts every Davidson.
        _apply(C2, 64, tr2=-1.0, name="c2-m64-lite"),
        # A ragged batch of the mixed form, from host memory.
        _apply(C2, 13, form="mixed", host=True, name="c2-m13-mixed-host"),
        # An orthorhombic cell, whose FFT box has three different edges.
        _apply(ORTHO, 16, name="ortho-m16"),
        # The larger cells, with as many perturbations as one image of many holds.
        _apply(C4C, 6, name="c4c-m6"),
        _apply(C5, 4, name="c5-m4"),
        _apply(C5, 8, form="mixed", name="c5-m8-mixed"),
    ]


def _edge(L, ecut):
    """QE's FFT edge for a wavefunction cutoff: the next number without factors above 5 that holds the density's sphere."""
    n = 2 * int(2.0 * math.sqrt(ecut) * L / (2.0 * math.pi)) + 1
    while True:
        k = n
        for p in (2, 3, 5):
            while k % p == 0:
                k //= p
        if k == 1 and n >= 16:
            return n
        n += 1


def _npw(case):
    return case["L1"] * case["L2"] * case["L3"] * case["ecut"] ** 1.5 / (12.0 * math.pi ** 2)


def draw(rng):
    """A cell between the smallest and the largest listed, cubic or orthorhombic, with QE's box for it, and a batch."""
    most = 0.4 * work(_apply(C5, 4))["flops"]   # every box, also those without kernels of their own
    while True:
        a = 9.0 * math.exp(rng.random() * math.log(28.0 / 9.0))
        ecut = rng.uniform(12.0, 30.0)
        if rng.random() < 0.35:
            Ls = tuple(round(a * rng.uniform(0.85, 1.2), 2) for _ in range(3))
        else:
            Ls = (round(a, 2),) * 3
        ecut = round(ecut, 2)
        n = tuple(_edge(L, ecut) for L in Ls)
        vol = Ls[0] * Ls[1] * Ls[2]
        nbnd = max(3, int(vol / rng.uniform(230.0, 400.0)))
        natoms = max(2, int(nbnd / rng.uniform(2.0, 6.0)))
        m = int(round(math.exp(rng.random() * math.log(64.0))))
        lite = rng.random() < 0.1
        c = _apply(_cell(Ls, ecut, n, natoms, nbnd, rng.choice(("s", "sp", "sp")), rng.randrange(1000)), m,
                   form=rng.choice(("fp64", "mixed")), host=rng.random() < 0.3, tr2=-1.0 if lite else TR2)
        if work(c)["flops"] <= most and _npw(c) < 38000:
            return c


@functools.lru_cache(maxsize=None)
def _system(L, ecut, n, natoms, nbnd, proj, seed):
    spec = SystemSpec(L=L, ecutwfc=ecut, nr=n, natoms=natoms, nbnd_occ=nbnd, proj=proj, seed=seed)
    return build_system(spec, "cuda")


def _system_of(case):
    """The ground state of a case: fixed data of the user's, computed once per process."""
    Ls, n = (case["L1"], case["L2"], case["L3"]), (case["n1"], case["n2"], case["n3"])
    if len(set(Ls)) == 1 and len(set(n)) == 1:
        Ls, n = Ls[0], n[0]
    return _system(Ls, case["ecut"], n, case["natoms"], case["nbnd"], case["proj"], case["system_seed"])


def prepare(case, seed):
    s = _system_of(case)
    op = ResponseOperator(s, n_dfpt_maxiter=MAXITER, verbose=False)
    op.set_precision(case["form"])
    state = dict(case=case, op=op)
    if case["do"] == "davidson":
        state["dvg"] = randomized_basis(s, case["m"], seed=seed)
        return state
    dvg = perturbations(s, case["m"], seed=seed)
    if case["host"]:
        state["dvg"], state["dng"] = dvg, np.zeros_like(dvg, order="F")
    else:
        state["dvg"] = torch.as_tensor(np.ascontiguousarray(dvg.T), device="cuda")
        state["dng"] = torch.zeros_like(state["dvg"])
        torch.cuda.synchronize()
    return state


def run(state):
    case, op = state["case"], state["op"]
    if case["do"] == "davidson":
        ev, conv, pdep, _ = op.davidson(state["dvg"], case["m"], n_pdep_times=4, n_pdep_maxiter=100,
                                        tr2_dfpt=case["tr2"], trev_pdep=1e-6, trev_pdep_rel=1e-1)
        return {"ev": ev, "conv": conv, "pdep": pdep}
    ierr = op.apply_operator(case["m"], state["dvg"], state["dng"], case["tr2"], 1)
    return {"dng": state["dng"], "ierr": ierr}


def _iterations(case):
    """PCG iterations of an average system, as counted on cells of 3 to 128 bands (14 to 52; within a quarter)."""
    return 10.0 + 4.0 * math.sqrt(case["nbnd"]) if case["tr2"] >= 0 else 0.0


def work(case):
    """Flops: per system and operator application one complex FFT each way for two bands (5 N log2 N), the kinetic,
    projector and Pv terms, the PCG's vector steps; the right-hand side and the density once.  Bytes: the ground
    state's arrays, the perturbations and the result once."""
    N = case["n1"] * case["n2"] * case["n3"]
    npw, nb, m = _npw(case), case["nbnd"], case["m"]
    nkb = case["natoms"] * (4 if case["proj"] == "sp" else 1)
    if case["do"] == "davidson":
        m = 6 * m      # columns that its operator calls get in all
    fft = 5.0 * N * math.log2(N)
    applications = _iterations(case) + 1.0 if case["tr2"] >= 0 else 0.0
    per_system = applications * (fft + 8.0 * npw * (nkb + nb) + 40.0 * npw) + fft + 8.0 * npw * nb
    return {"flops": m * (nb * per_system + fft),
            "bytes": 8.0 * N + 16.0 * npw * (nkb + nb + 2 * m)}


def tolerance(case):
    """Four times what 28 cells showed, against exact() and with the sums in another order.  Without a PCG it is
    rounding (4e-15).  With one, a system whose residual passes the threshold by a hair may stop one iteration apart:
    4e-10 in FP64; the mixed form's FP32 correction solves leave 9e-9 wherever they end below the threshold.  A
    Davidson carries that through its iterations, over its eigenvalues' gaps: 2e-7 where one system stopped apart."""
    if case["do"] == "davidson":
        return {"rel": 1e-6, "max": 1e-4}
    if case["tr2"] < 0:
        return {"rel": 2e-14, "max": 1e-12}
    return {"rel": 4e-8, "max": 1.2e-6} if case["form"] == "mixed" else {"rel": 2e-9, "max": 3e-7}


# ---- the same in plain torch, 64 bits --------------------------------------------------------------------------

class _Exact:
    """dfpt's Gamma branch on complex boxes, every system at once: columns [system, npw]."""

    def __init__(self, s, maxiter):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
        self.n, self.maxiter, self.alpha = (s.nrs[2], s.nrs[1], s.nrs[0]), maxiter, s.alpha_pv
        self.nl, self.nlm, self.g2, self.v, self.sq = t(s.nl), t(s.nlm), t(s.g2kin), t(s.vrs), t(s.sqvc)
        self.evc, self.vkb, self.D = t(s.evc.T), t(s.vkb.T), t(s.deeq)
        self.et, self.occ = t(s.et[: s.nbnd_occ]), t(s.occupation)
        self.N, self.scale = s.nnr, 2.0 * s.wk / s.omega
        eprec = 1.35 * ((self.evc.abs() ** 2) * self.g2).sum(1)
        self.iprec = 1.0 / torch.clamp(self.g2[None, :] / eprec[:, None], min=1.0)
        self.chunk = max(1, int(1.5e9 // (16 * self.N)))

    def to_r(self, a):
        """Columns -> real functions (two columns share a complex box)."""
        k = a.shape[0]
        p = torch.cat([a, torch.zeros_like(a[:1])]) if k % 2 else a
        box = torch.zeros((p.shape[0] // 2, self.N), dtype=torch.complex128, device=a.device)
        box[:, self.nl] = p[0::2] + 1j * p[1::2]
        box[:, self.nlm] = (p[0::2] - 1j * p[1::2]).conj()
        r = torch.fft.ifftn(box.view(-1, *self.n), dim=(1, 2, 3), norm="forward").reshape(-1, self.N)
        return torch.view_as_real(r).permute(0, 2, 1).reshape(-1, self.N)[:k]

    def to_g(self, r):
        """Real functions -> columns."""
        k = r.shape[0]
        p = torch.cat([r, torch.zeros_like(r[:1])]) if k % 2 else r
        box = torch.complex(p[0::2], p[1::2]).view(-1, *self.n)
        g = torch.fft.fftn(box, dim=(1, 2, 3), norm="forward").reshape(-1, self.N)
        a, b = g[:, self.nl], g[:, self.nlm].conj()
        return torch.stack([(a + b) / 2, (a - b) / 2j], 1).reshape(-1, a.shape[1])[:k]

    def braket(self, a, b):
        return 2.0 * (torch.view_as_real(a).flatten(1) @ torch.view_as_real(b).flatten(1).T) - torch.outer(
            a[:, 0].real, b[:, 0].real)

    def dots(self, a, b):
        return 2.0 * (a.real * b.real + a.imag * b.imag).sum(1) - a[:, 0].real * b[:, 0].real

    def A(self, x, e):
        h = torch.empty_like(x)
        for c in range(0, x.shape[0], self.chunk):
            h[c:c + self.chunk] = self.to_g(self.to_r(x[c:c + self.chunk]) * self.v)
        h += self.g2 * x
        h += (self.braket(x, self.vkb) @ self.D).to(h.dtype) @ self.vkb
        h[:, 0].imag.zero_()
        h -= e[:, None] * x
        return h + (self.alpha * self.braket(x, self.evc)).to(h.dtype) @ self.evc

    def solve(self, b, x, band, tr2):
        """The masked preconditioned CG; a system that has converged keeps its x."""
        et, n = self.et[band], b.shape[0]
        act = torch.arange(n, device=b.device)
        g, p, rho_old = self.A(x, et) - b, torch.zeros_like(b), torch.ones(n, dtype=torch.float64, device=b.device)
        for it in range(self.maxiter):
            h = g * self.iprec[band[act]]
            rho = self.dots(h, g)
            on = rho >= tr2
            act, g, p, h, rho, rho_old = act[on], g[on], p[on], h[on], rho[on], rho_old[on]
            if act.numel() == 0:
                break
            p = (rho / rho_old)[:, None] * p - h if it else -h
            t = self.A(p, et[act])
            r = (self.dots(p, g) / self.dots(p, t))[:, None]
            x[act] -= r * p
            g, rho_old = g - r * t, rho
        return x, act

    def __call__(self, dvg, tr2):
        m, nb = dvg.shape[0], self.evc.shape[0]
        dv = self.to_r(dvg * self.sq)
        psi = self.to_r(self.evc)
        b = torch.cat([self.to_g(psi * dv[p]) for p in range(m)])
        b = self.braket(b, self.evc).to(b.dtype) @ self.evc - b
        band = torch.arange(nb, device=b.device).repeat(m)
        x, left = b * self.iprec[band], None
        if tr2 >= 0:
            x, left = self.solve(b, x, band, tr2)
        rho = torch.stack([(self.occ[:, None] * psi * self.to_r(x[p * nb:(p + 1) * nb])).sum(0) for p in range(m)])
        dng = self.to_g(rho) * self.scale * self.sq
        dng[:, 0] = 0.0
        return dng, left


def exact(case, seed):
    """None for a Davidson: its eigenpairs carry its loose starting step and stop at its own test."""
    if case["do"] == "davidson":
        return None
    s = _system_of(case)
    dvg = torch.as_tensor(np.ascontiguousarray(perturbations(s, case["m"], seed=seed).T), device="cuda")
    dng, _ = _Exact(s, MAXITER)(dvg, case["tr2"])
    return {"dng": np.asfortranarray(dng.cpu().numpy().T) if case["host"] else dng, "ierr": None}
