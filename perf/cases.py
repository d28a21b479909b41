"""The work that a user of this library has it do, as measurable cases.

Every case goes through the package's public entry points (FastPipelineScheduler,
ReplicaBatch, DeviceNeighborList, DeviceEam / compute_morse_gpu, the
force-matching losses) on seeded synthetic FCC metals with the potentials of
tdmd_claude_b200.workloads.  `listed` holds fixed cases from the smallest call
(256 atoms) to the largest (1 M atoms); `draw` gives others of the same ranges.

kinds
  md        a running simulation: run_until advances the same system by `steps`
            steps, then the state is read back into pinned buffers (a dump
            frame); with thermo also the energies (a thermo line)
  job       upload from pinned buffers, run_until, download: a short run whose
            caller holds the state (restarts, sampling, coupling to host code)
  replicas  many uneven systems advanced together, energies logged
  nlist     one neighbor-list build on caller-owned device positions
  compute   one force evaluation on caller-owned device arrays and list, with
            energy and virial
  fit       one force-matching loss and its gradient over all snapshots

`exact` restates each computation in 64-bit torch (its own pair search,
splines and integrator); only the input generators are shared.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tdmd_claude_b200 import (Box, DeviceEam, DeviceNeighborList, EamAlloy, FastPipelineScheduler,
                              MorseParams, ReplicaBatch, compute_morse_gpu, make_config)
from tdmd_claude_b200 import fitting
from tdmd_claude_b200 import workloads as W

A_CU = 3.615         # lattice constants of the library's own workloads
A_TERNARY = 3.56
DT = 0.001
DT_MIN, DT_MAX = 0.0001, 0.002   # make_config's adaptive-dt defaults
C2 = 0.0025                      # at most c2 * rc = 0.0125 A per step
T_PERIOD, NHC_LENGTH = 0.1, 3    # make_config's thermostat defaults


def listed():
    return [
        # The reference's own 256-atom Cu Morse system: the smallest call, bound by launches.
        dict(name="md_morse_256", kind="md", pot="morse", prec="fp64", nx=4, ny=4, nz=4,
             vacancies=0, slab=False, shuffle=False, temp=300.0, nvt=False, thermo=False,
             steps=100),
        # A small ragged sample with vacancies, in the default mixed mode, with a thermo line.
        dict(name="md_eam_ragged", kind="md", pot="eam", prec="mixed", nx=11, ny=9, nz=7,
             vacancies=5, slab=False, shuffle=False, temp=600.0, nvt=False, thermo=True,
             steps=100),
        # The benchmark's system (131 072 atoms EAM) in both precisions.
        dict(name="md_eam_131k", kind="md", pot="eam", prec="mixed", nx=32, ny=32, nz=32,
             vacancies=0, slab=False, shuffle=False, temp=300.0, nvt=False, thermo=False,
             steps=50),
        dict(name="md_eam_131k_fp64", kind="md", pot="eam", prec="fp64", nx=32, ny=32, nz=32,
             vacancies=0, slab=False, shuffle=False, temp=300.0, nvt=False, thermo=False,
             steps=50),
        # A ternary alloy under the thermostat with adaptive dt, atoms in file order (random).
        dict(name="md_ternary_nvt", kind="md", pot="ternary", prec="mixed", nx=25, ny=24, nz=23,
             vacancies=13, slab=False, shuffle=True, temp=1000.0, nvt=True, thermo=True,
             steps=50),
        # The largest: 1.05 M atoms, out of L2.
        dict(name="md_eam_1m", kind="md", pot="eam", prec="mixed", nx=64, ny=64, nz=64,
             vacancies=0, slab=False, shuffle=False, temp=300.0, nvt=False, thermo=False,
             steps=20),
        # The benchmark's end-to-end step: state up, one window of 10 steps, state down.
        dict(name="job_eam_131k", kind="job", pot="eam", prec="mixed", nx=32, ny=32, nz=32,
             vacancies=0, slab=False, shuffle=False, temp=300.0, nvt=False, thermo=False,
             steps=10),
        # Uneven Morse replicas in one batch.
        dict(name="replicas_morse", kind="replicas", pot="morse", prec="mixed", nrep=64, nmin=4,
             nmax=11, steps=100),
        # A list for a caller who integrates with the free functions.
        dict(name="nlist_build", kind="nlist", pot="eam", nx=33, ny=29, nz=31, vacancies=7,
             slab=False, shuffle=False, temp=300.0),
        # One FP64 evaluation on the caller's arrays: relaxations, checks against other codes.
        dict(name="compute_eam_fp64", kind="compute", pot="eam", prec="fp64", nx=22, ny=20, nz=23,
             vacancies=3, slab=False, shuffle=False, temp=300.0),
        # Force matching: a step of a Morse fit on few atoms, of an EAM fit on many.
        dict(name="fit_morse", kind="fit", pot="morse", prec="fp64", ncell=5, nsnap=16),
        dict(name="fit_eam", kind="fit", pot="eam", prec="fp64", ncell=9, nsnap=24),
    ]


# Atoms x steps of one pass stay below the largest listed case's 21 M.
_MOST = 15e6


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(rng, natoms):
    """Ragged box of about natoms atoms, at least 4 cells per axis."""
    side = (natoms / 4) ** (1 / 3)
    c = [max(4, int(round(side * math.exp(rng.uniform(-0.35, 0.35))))) for _ in range(3)]
    return dict(nx=c[0], ny=c[1], nz=c[2])


def draw(rng):
    kind = rng.choice(["md", "md", "md", "job", "replicas", "nlist", "compute", "fit"])
    if kind in ("md", "job"):
        pot = rng.choice(["morse", "eam", "eam", "ternary"])
        # 256 to ~600 k atoms
        c = dict(kind=kind, pot=pot, prec=rng.choice(["mixed", "mixed", "fp64"]),
                 **_cells(rng, _log_int(rng, 256, 4e5)), vacancies=rng.randint(0, 9),
                 slab=rng.random() < 0.2, shuffle=rng.random() < 0.3,
                 temp=round(rng.uniform(100.0, 1000.0), 1), nvt=rng.random() < 0.25,
                 thermo=kind == "md" and rng.random() < 0.5)
        n = 4 * c["nx"] * c["ny"] * c["nz"]
        most = 10 if kind == "job" else 100
        c["steps"] = max(5, min(most, int(_MOST / n * rng.uniform(0.3, 1.0))))
        return c
    if kind == "replicas":
        nmin = rng.randint(4, 7)
        return dict(kind=kind, pot=rng.choice(["morse", "eam"]),
                    prec=rng.choice(["mixed", "fp64"]), nrep=_log_int(rng, 4, 96), nmin=nmin,
                    nmax=nmin + rng.randint(1, 5), steps=rng.randint(20, 60))
    if kind == "nlist":
        return dict(kind=kind, pot=rng.choice(["morse", "eam"]),
                    **_cells(rng, _log_int(rng, 256, 5e5)), vacancies=rng.randint(0, 9),
                    slab=rng.random() < 0.2, shuffle=rng.random() < 0.3, temp=300.0)
    if kind == "compute":
        pot = rng.choice(["morse", "eam", "ternary"])
        return dict(kind=kind, pot=pot, prec=rng.choice(["mixed", "fp64"]),
                    **_cells(rng, _log_int(rng, 256, 5e5)), vacancies=rng.randint(0, 9),
                    slab=rng.random() < 0.2, shuffle=rng.random() < 0.3, temp=300.0)
    pot = rng.choice(["morse", "eam", "ternary"])
    return dict(kind=kind, pot=pot, prec=rng.choice(["fp64", "fp64", "mixed"]),
                ncell=rng.randint(4, 10), nsnap=_log_int(rng, 2, 24))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _tables(pot):
    return W.ternary_eam_tables() if pot == "ternary" else W.cu_eam_tables()


def _cutoff(pot):
    return W.MORSE_CU[3] if pot == "morse" else 5.0


def _potential(pot):
    if pot == "morse":
        return MorseParams.make(*W.MORSE_CU)
    t = _tables(pot)
    return EamAlloy.from_tables(t.ntypes, t.nrho, t.drho, t.nr, t.dr, t.cutoff, t.F, t.rho,
                                t.rphi)


class _Sys:
    """Positions, velocities, 1-based types, masses[type], box of one system."""

    def __init__(self, pos, vel, types, masses, hi, periodic):
        self.pos, self.vel, self.types, self.masses = pos, vel, types, masses
        self.hi, self.periodic, self.n = hi, periodic, pos.shape[0]

    def box(self):
        return Box.make((0.0, 0.0, 0.0), self.hi, self.periodic)


def _system(case, seed):
    """Thermally displaced FCC crystal with random vacancies; a slab's free
    surfaces are its z faces."""
    rng = np.random.default_rng(seed)
    a = A_TERNARY if case["pot"] == "ternary" else A_CU
    cells = (case["nx"], case["ny"], case["nz"])
    pos = W.fcc_lattice(*cells, a)
    hi = np.array([c * a for c in cells])
    if case["vacancies"]:
        keep = np.ones(len(pos), bool)
        keep[rng.choice(len(pos), case["vacancies"], replace=False)] = False
        pos = pos[keep]
    # about the harmonic thermal displacement of Cu at this temperature
    pos = pos + rng.normal(0.0, 0.08 * math.sqrt(case["temp"] / 300.0), pos.shape)
    periodic = (1, 1, 0 if case["slab"] else 1)
    for k in range(3):
        if periodic[k]:
            pos[:, k] = np.mod(pos[:, k], hi[k])
            pos[pos[:, k] >= hi[k], k] = 0.0
    if case["shuffle"]:
        pos = pos[rng.permutation(len(pos))]
    n = len(pos)
    if case["pot"] == "ternary":
        types = rng.integers(1, 4, n).astype(np.int32)
        masses = np.array([1.0, *W.ternary_eam_tables().masses])
    else:
        types = np.ones(n, np.int32)
        masses = np.array([1.0, W.CU_MASS])
    vel = W.maxwell_boltzmann(masses[types], case["temp"], rng)
    return _Sys(np.ascontiguousarray(pos), vel, types, masses, tuple(hi), periodic)


def _replica_systems(case, seed):
    rng = np.random.default_rng(seed)
    size = np.random.default_rng(case["nrep"] * 1000 + case["nmin"] * 31 + case["nmax"])
    out = []
    for r in range(case["nrep"]):  # sizes belong to the case, the rest to the seed
        n = int(size.integers(case["nmin"], case["nmax"] + 1))
        c = dict(pot=case["pot"], nx=n, ny=n, nz=n, vacancies=int(size.integers(0, 4)),
                 slab=False, shuffle=False, temp=float(rng.uniform(100.0, 1500.0)))
        out.append(_system(c, int(rng.integers(1 << 31))))
    return out


def _fit_inputs(case, seed):
    """Snapshots, types, box edge, targets (forces at the true parameters) and
    the perturbed parameters at which the loss is evaluated."""
    rng = np.random.default_rng(seed)
    a = A_TERNARY if case["pot"] == "ternary" else A_CU
    lat = W.fcc_lattice(case["ncell"], case["ncell"], case["ncell"], a)
    L = case["ncell"] * a
    pos = np.mod(lat[None] + rng.normal(0.0, 0.12, (case["nsnap"], len(lat), 3)), L)
    pos[pos >= L] = 0.0
    nt = 3 if case["pot"] == "ternary" else 1
    types = rng.integers(1, nt + 1, len(lat)).astype(np.int32)
    if case["pot"] == "morse":
        true = torch.tensor(W.MORSE_CU[:3], dtype=torch.float64, device="cuda")
        prm = [true * torch.tensor(1.0 + 0.03 * rng.uniform(-1, 1, 3), device="cuda")]
    else:
        true = _spline_tables(_tables(case["pot"]))
        # smooth perturbation of the tabulated functions' coefficients
        prm = [c * (1.0 + 0.05 * rng.uniform(-1, 1)) for c in true]
    pairs = _snapshot_pairs(pos, L, _cutoff(case["pot"]))
    tt = torch.as_tensor(np.tile(types, case["nsnap"]), device="cuda").long() - 1
    with torch.no_grad():
        target = _fit_forces(case, true, pairs, tt)
    return pos, types, L, target, prm, pairs, tt


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory()


class _State:
    pass


def _skin(case):
    """A skin that ten steps at this temperature do not use up."""
    return 0.3 if case.get("temp", 1500.0) <= 400.0 else 0.5


def _config(case):
    more = {}
    if case["kind"] == "replicas":
        more = dict(energy_every=10, energy_log_capacity=4096)
    elif case["nvt"]:
        more = dict(t_target=case["temp"], adaptive_dt=True, c2=C2)
    return make_config(dt=DT, r_skin=_skin(case), rebuild_every=10, precision=case["prec"], **more)


def prepare(case, seed):
    st = _State()
    st.case = case
    kind = case["kind"]
    if kind in ("md", "job"):
        s = _system(case, seed)
        st.sched = FastPipelineScheduler(s.box(), s.n, _potential(case["pot"]), _config(case))
        f = torch.float32 if case["prec"] == "mixed" else torch.float64
        st.out = {"pos": torch.empty(s.n, 3, dtype=torch.float64).pin_memory(),
                  "vel": torch.empty(s.n, 3, dtype=torch.float64).pin_memory(),
                  "frc": torch.empty(s.n, 3, dtype=f).pin_memory()}
        st.step = 0
        # a program's start-up: the system goes up, launch shapes are tuned
        st.inp = [_pinned(x) for x in (s.pos, s.vel, s.types, np.arange(1, s.n + 1, dtype=np.int32),
                                       s.masses)]
        _upload(st)
        st.sched.run_until(0)
    elif kind == "replicas":
        ss = _replica_systems(case, seed)
        st.batch = ReplicaBatch([s.box() for s in ss], [s.n for s in ss], _potential(case["pot"]),
                                _config(case))
        st.batch.upload(np.concatenate([s.pos for s in ss]), np.concatenate([s.vel for s in ss]),
                        np.concatenate([s.types for s in ss]), ss[0].masses)
        st.step = 0
        st.batch.run_until(0)
    elif kind in ("nlist", "compute"):
        s = _system(case, seed)
        st.n, st.box, st.rc = s.n, s.box(), _cutoff(case["pot"])
        st.pos = torch.as_tensor(s.pos, device="cuda")
        torch.cuda.synchronize()
        st.nl = DeviceNeighborList()
        if kind == "nlist":
            # the caller's own rows, which outlive the next build (room for the
            # densest packing of the displaced crystal; -1 past the list)
            st.rows = torch.full((int(s.n * _shape(case)[1] * 1.3) + 64,), -1, dtype=torch.int32,
                                 device="cuda")
        if kind == "compute":
            st.nl.build(st.pos, s.n, st.box, st.rc, _skin(case))
            st.rows = (st.nl.d_neighbors(), st.nl.d_offsets(), st.nl.d_counts())
            st.pot = _potential(case["pot"])
            if case["pot"] != "morse":
                st.eam = DeviceEam()
                st.eam.upload_tables(st.pot)
            st.types = torch.as_tensor(s.types, device="cuda")
            f = torch.float32 if case["prec"] == "mixed" else torch.float64
            st.frc = torch.empty(s.n, 3, dtype=f, device="cuda")
            st.pe = torch.zeros(1, dtype=torch.float64, device="cuda")
            st.vir = torch.zeros(6, dtype=torch.float64, device="cuda")
            st.rho = torch.empty(s.n, dtype=torch.float64, device="cuda")
            st.fp = torch.empty(s.n, dtype=torch.float64, device="cuda")
    else:
        pos, types, L, target, prm, _, _ = _fit_inputs(case, seed)
        box = Box.make((0.0,) * 3, (L,) * 3)
        st.fm = fitting.ForceMatch(pos, types, box, _cutoff(case["pot"]), case["prec"])
        st.fm.set_targets(target.cpu().numpy())
        st.prm = [p.clone().requires_grad_(True) for p in prm]
        if case["pot"] != "morse":
            st.meta = fitting.eam_table_meta(_potential(case["pot"]))
    return st


def _upload(st):
    x, v, t, i, m = st.inp
    st.sched.upload_ptrs(x.data_ptr(), v.data_ptr(), 0, t.data_ptr(), i.data_ptr(), m.data_ptr(),
                         m.numel())


class _Dev:
    """A device array of the library for torch to view without a copy; the view
    keeps the array's owner alive."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<i4", data=(ptr, False),
                                             version=3)


def _view(owner, ptr, n):
    return torch.as_tensor(_Dev(owner, ptr, n), device="cuda")


def run(st):
    case = st.case
    kind = case["kind"]
    if kind in ("md", "job"):
        if kind == "job":
            _upload(st)
            st.sched.run_until(case["steps"])
        else:
            st.step += case["steps"]
            st.sched.run_until(st.step)
        o = st.out
        st.sched.download_ptrs(o["pos"].data_ptr(), o["vel"].data_ptr(), o["frc"].data_ptr())
        if case["thermo"]:
            pe, ke, w = st.sched.energies()
            return dict(o, pe=np.array([pe]), ke=np.array([ke]), virial=w)
        return o
    if kind == "replicas":
        st.step += case["steps"]
        st.batch.run_until(st.step)
        pos, vel, frc = st.batch.download()
        pe, ke = st.batch.energies()
        return {"pos": pos, "vel": vel, "frc": frc, "pe": pe, "ke": ke}
    if kind == "nlist":
        st.nl.build(st.pos, st.n, st.box, st.rc, _skin(case))
        nl = st.nl
        total = nl.total_pairs()
        st.rows[:total].copy_(_view(nl, nl.d_neighbors(), total))
        return {"counts": _view(nl, nl.d_counts(), st.n),
                "offsets": _view(nl, nl.d_offsets(), st.n), "neighbors": st.rows}
    if kind == "compute":
        st.pe.zero_()
        st.vir.zero_()
        out = {"frc": st.frc, "pe": st.pe, "virial": st.vir}
        if case["pot"] == "morse":
            compute_morse_gpu(st.pos, st.frc, *st.rows, st.n, st.box, st.pot, st.pe, st.vir,
                              case["prec"])
            return out
        st.eam.compute(st.pos, st.frc, st.types, *st.rows, st.n, st.box, st.pe, st.vir, st.rho,
                       st.fp, case["prec"])
        return dict(out, rho=st.rho, fp=st.fp)
    if case["pot"] == "morse":
        loss = fitting.morse_loss(st.prm[0], st.fm)
    else:
        loss = fitting.eam_loss(*st.prm, st.fm, st.meta)
    return {"loss": loss.detach(), "grads": list(torch.autograd.grad(loss, st.prm))}


# ---------------------------------------------------------------------------
# Work and tolerances
# ---------------------------------------------------------------------------
def _shape(case):
    """(atoms, mean neighbors inside the cutoff)"""
    if case["kind"] == "replicas":
        n = case["nrep"] * 4 * ((case["nmin"] + case["nmax"]) / 2) ** 3
    elif case["kind"] == "fit":
        n = case["nsnap"] * 4 * case["ncell"] ** 3
    else:
        n = 4 * case["nx"] * case["ny"] * case["nz"] - case["vacancies"]
    a = A_TERNARY if case["pot"] == "ternary" else A_CU
    rc = _cutoff(case["pot"]) + (_skin(case) if case["kind"] == "nlist" else 0.0)
    return n, 4 / a ** 3 * 4 / 3 * math.pi * rc ** 3


def work(case):
    n, k = _shape(case)
    kind = case["kind"]
    # arithmetic of one pair inside the cutoff: distance 8, radius 2, and
    # Morse 14 + force 6, or EAM twice (density 8; two derivatives 10, force 10)
    pair = 30 if case["pot"] == "morse" else 48
    if kind == "nlist":
        return {"bytes": n * (24 + 8) + 4 * n * k, "flops": 9 * n * k}
    if kind == "compute":
        return {"bytes": n * (24 + 24 + 8 + 4 * k), "flops": pair * n * k}
    if kind == "fit":
        # forces, then the adjoint over the same pairs
        return {"bytes": n * (24 + 24 + 4 * k), "flops": 2.5 * pair * n * k}
    # state in, state and forces out, and the arithmetic of every step
    return {"bytes": n * (48 + 72), "flops": case["steps"] * pair * n * k}


def tolerance(case):
    """About four times the difference from `exact` measured over the ranges."""
    kind, morse = case["kind"], case["pot"] == "morse"
    if kind == "nlist":
        return "exact"
    if case["prec"] == "fp64":
        # rounding, grown by up to 100 steps of dynamics, or of sums over all pairs
        return {"rel": 1e-12, "max": 1e-11}
    if kind == "fit" and not morse:
        # FP32 forces against targets a few percent away, summed with both signs
        # into thousands of coefficients
        return {"rel": 1.3e-2, "max": 0.25}
    if morse and kind in ("md", "replicas"):
        # the truncated pair force jumps at the cutoff: a pair may cross it a step
        # earlier or later
        return {"rel": 6e-5, "max": 2e-2}
    return {"rel": 2e-6, "max": 2e-5}


# ---------------------------------------------------------------------------
# The same computations in 64-bit torch
# ---------------------------------------------------------------------------
def _pairs(pos, hi, periodic, r):
    """Ordered pairs (i, j) closer than r: cell grid, 27 shifts, minimum image."""
    n, dev = pos.shape[0], pos.device
    nc = [max(1, int(hi[k] / r)) for k in range(3)]
    nc = [c if c >= 3 else 1 for c in nc]
    L = torch.tensor(hi, dtype=torch.float64, device=dev)
    per = torch.tensor(periodic, dtype=torch.float64, device=dev)
    c = torch.stack([(pos[:, k] / hi[k] * nc[k]).floor().long().clamp(0, nc[k] - 1)
                     for k in range(3)], 1)
    cid = (c[:, 2] * nc[1] + c[:, 1]) * nc[0] + c[:, 0]
    ncell = nc[0] * nc[1] * nc[2]
    order = torch.argsort(cid, stable=True)
    count = torch.bincount(cid, minlength=ncell)
    start = torch.cumsum(count, 0) - count
    m = int(count.max())
    table = torch.full((ncell, m), -1, dtype=torch.long, device=dev)
    cs = cid[order]
    table[cs, torch.arange(n, device=dev) - start[cs]] = order
    shifts = [[-1, 0, 1] if nc[k] > 1 else [0] for k in range(3)]
    rows = max(1, (1 << 25) // m)
    ii, jj = [], []
    for dz in shifts[2]:
        for dy in shifts[1]:
            for dx in shifts[0]:
                q = c + torch.tensor([dx, dy, dz], device=dev)
                ok = torch.ones(n, dtype=torch.bool, device=dev)
                for k in range(3):
                    if not periodic[k]:
                        ok &= (q[:, k] >= 0) & (q[:, k] < nc[k])
                    q[:, k] %= nc[k]
                nb = (q[:, 2] * nc[1] + q[:, 1]) * nc[0] + q[:, 0]
                for a in range(0, n, rows):
                    cand = table[nb[a:a + rows]]
                    i = torch.arange(a, min(n, a + rows), device=dev)[:, None].expand_as(cand)
                    keep = (cand >= 0) & (cand != i) & ok[a:a + rows, None]
                    i, j = i[keep], cand[keep]
                    d = pos[i] - pos[j]
                    d -= per * L * torch.round(d / L)
                    near = (d * d).sum(1) < r * r
                    ii.append(i[near])
                    jj.append(j[near])
    return torch.cat(ii), torch.cat(jj)


def _spline_coeffs(v, h):
    """Cubic Hermite coefficients a|b|c|d with averaged finite-difference slopes."""
    d = (v[..., 1:] - v[..., :-1]) / h
    s = torch.cat([d[..., :1], 0.5 * (d[..., 1:] + d[..., :-1]), d[..., -1:]], -1)
    m0, m1 = s[..., :-1], s[..., 1:]
    return torch.cat([v[..., :-1], m0, (3 * d - 2 * m0 - m1) / h, (m0 + m1 - 2 * d) / h ** 2], -1)


def _spline_tables(t):
    """(F, rho, phi) coefficient arrays [nfunctions, 4 * intervals] on the GPU."""
    dev = "cuda"
    F = torch.as_tensor(t.F, device=dev)
    rho = torch.as_tensor(t.rho, device=dev)
    r = torch.arange(t.nr, dtype=torch.float64, device=dev) * t.dr
    phi = torch.as_tensor(t.rphi, device=dev) / torch.where(r > 0, r, torch.ones_like(r))
    phi[:, 0] = 0.0
    return [_spline_coeffs(F, t.drho), _spline_coeffs(rho, t.dr), _spline_coeffs(phi, t.dr)]


def _spl(c, f, x, h):
    """(value, derivative) of function f of the coefficient array c at x."""
    ns = c.shape[1] // 4
    k = (x.detach() / h).long().clamp(0, ns - 1)
    dx = x - k.double() * h
    flat = c.reshape(-1)
    a, b, cc, d = (flat[f * 4 * ns + m * ns + k] for m in range(4))
    return a + dx * (b + dx * (cc + dx * d)), b + dx * (2 * cc + 3 * d * dx)


def _pair_slot(ti, tj, nt):
    lo, hi = torch.minimum(ti, tj), torch.maximum(ti, tj)
    return lo * nt - lo * (lo + 1) // 2 + hi


def _eam(i, j, d, r, types, n, coeffs, t):
    """Forces, potential energy per atom, fpair, rho, F' of listed pairs (r < cutoff)."""
    F, rho_c, phi_c = coeffs
    ti, tj = types[i], types[j]
    frj, drj = _spl(rho_c, tj, r, t.dr)
    rho = torch.zeros(n, dtype=torch.float64, device=r.device).index_add(0, i, frj)
    Fv, Fp = _spl(F, types, rho, t.drho)
    dri = drj if t.ntypes == 1 else _spl(rho_c, ti, r, t.dr)[1]
    pv, pd = _spl(phi_c, _pair_slot(ti, tj, t.ntypes), r, t.dr)
    fpair = -(pd + Fp[i] * drj + Fp[j] * dri) / r
    f = torch.zeros(n, 3, dtype=torch.float64, device=r.device).index_add(0, i, fpair[:, None] * d)
    pe = (Fv + torch.zeros_like(rho).index_add(0, i, 0.5 * pv)).detach()
    return f, pe, fpair, rho, Fp


def _morse(i, d, r, n, prm):
    D, alpha, r0 = prm[0], prm[1], prm[2]
    ex = torch.exp(-alpha * (r - r0))
    fpair = -2 * D * alpha * (1 - ex) * ex / r
    f = torch.zeros(n, 3, dtype=torch.float64, device=r.device).index_add(0, i, fpair[:, None] * d)
    pe = torch.zeros(n, dtype=torch.float64, device=r.device).index_add(
        0, i, 0.5 * D * ((1 - ex) ** 2 - 1))
    return f, pe, fpair


class _Md:
    """Atoms of one or several boxes advanced together."""

    def __init__(self, systems, pot):
        dev = "cuda"
        self.systems, self.pot = systems, pot
        self.pos = torch.as_tensor(np.concatenate([s.pos for s in systems]), device=dev)
        self.vel = torch.as_tensor(np.concatenate([s.vel for s in systems]), device=dev)
        self.types = torch.as_tensor(np.concatenate([s.types for s in systems]),
                                     device=dev).long() - 1
        self.mass = torch.as_tensor(systems[0].masses, device=dev)[self.types + 1][:, None]
        rep = lambda f: torch.as_tensor(np.concatenate(  # noqa: E731
            [np.broadcast_to(np.array(f(s), float), (s.n, 3)) for s in systems]), device=dev)
        self.L, self.per = rep(lambda s: s.hi), rep(lambda s: s.periodic)
        self.n = self.pos.shape[0]
        self.rc = _cutoff(pot)
        if pot != "morse":
            self.tab = _tables(pot)
            self.coeffs = _spline_tables(self.tab)
        else:
            self.prm = torch.tensor(W.MORSE_CU[:3], dtype=torch.float64, device=dev)
        self.build()
        self.forces()

    def build(self):
        ii, jj, off = [], [], 0
        for s in self.systems:
            i, j = _pairs(self.pos[off:off + s.n], s.hi, s.periodic, self.rc + 0.6)
            ii.append(i + off)
            jj.append(j + off)
            off += s.n
        self.i, self.j = torch.cat(ii), torch.cat(jj)

    def delta(self, i, j):
        d = self.pos[i] - self.pos[j]
        L = self.L[i]
        return d - self.per[i] * L * torch.round(d / L)

    def forces(self):
        d = self.delta(self.i, self.j)
        r2 = (d * d).sum(1)
        keep = r2 < self.rc ** 2
        i, j, d = self.i[keep], self.j[keep], d[keep]
        r = torch.sqrt(r2[keep])
        if self.pot == "morse":
            self.f, self.pe, fpair = _morse(i, d, r, self.n, self.prm)
        else:
            self.f, self.pe, fpair, self.rho, self.fp = _eam(i, j, d, r, self.types, self.n,
                                                             self.coeffs, self.tab)
        self.vir = torch.stack([(0.5 * fpair * d[:, a] * d[:, b]).sum()
                                for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))])

    def kick(self, dt):
        self.vel = self.vel + dt / (self.mass * W.MVV2E) * self.f

    def drift(self, dt):
        p = self.pos + dt * self.vel
        p = p + self.per * self.L * (p < 0).double()
        self.pos = p - self.per * self.L * (p >= self.L).double()

    def ke(self):
        return (0.5 * W.MVV2E * self.mass * self.vel ** 2).sum(1)

    def advance(self, steps, chain=None):
        """Velocity Verlet; with chain, thermostat half steps around each step
        and the time step from the largest speed."""
        for s in range(steps):
            dt = DT
            if chain is not None:
                vmax = float(torch.sqrt((self.vel ** 2).sum(1).max()))
                dt = max(DT_MIN, min(DT_MAX, C2 * self.rc / vmax))
                self.vel = self.vel * chain.half_step(float(self.ke().sum()))
            self.kick(0.5 * dt)
            self.drift(dt)
            if s and s % 10 == 0:
                self.build()
            self.forces()
            self.kick(0.5 * dt)
            if chain is not None:
                self.vel = self.vel * chain.half_step(float(self.ke().sum()))


class _Chain:
    """Nose-Hoover chain half step: outermost thermostat first, exp(-v dt/8)
    around each inner update, velocities scaled by exp(-v_0 dt/2)."""

    def __init__(self, temp, n_dof):
        self.kt, self.n_dof, self.v = W.KB * temp, n_dof, [0.0] * NHC_LENGTH
        self.m = [n_dof * self.kt * T_PERIOD ** 2] + [self.kt * T_PERIOD ** 2] * (NHC_LENGTH - 1)

    def half_step(self, ke):
        h, v, m, last = 0.5 * DT, self.v, self.m, NHC_LENGTH - 1
        g = lambda k: (m[k - 1] * v[k - 1] ** 2 - self.kt) / m[k]  # noqa: E731
        v[last] += g(last) * h
        for k in range(last - 1, 0, -1):
            e = math.exp(-v[k + 1] * h / 4)
            v[k] = (v[k] * e + g(k) * h) * e
        e = math.exp(-v[1] * h / 4)
        v[0] = (v[0] * e + (2 * ke - self.n_dof * self.kt) / m[0] * h) * e
        return math.exp(-v[0] * h)


def _snapshot_pairs(pos, L, rc):
    """Pairs of all snapshots: (i, j, d, r) over the concatenated atoms."""
    ii, jj = [], []
    p = torch.as_tensor(pos, device="cuda")
    for s in range(p.shape[0]):
        i, j = _pairs(p[s], (L,) * 3, (1, 1, 1), rc)
        ii.append(i + s * p.shape[1])
        jj.append(j + s * p.shape[1])
    i, j = torch.cat(ii), torch.cat(jj)
    flat = p.reshape(-1, 3)
    d = flat[i] - flat[j]
    d = d - L * torch.round(d / L)
    return i, j, d, torch.sqrt((d * d).sum(1))


def _fit_forces(case, prm, pairs, types):
    i, j, d, r = pairs
    if case["pot"] == "morse":
        return _morse(i, d, r, types.numel(), prm)[0]
    return _eam(i, j, d, r, types, types.numel(), prm, _tables(case["pot"]))[0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "nlist":
        return None
    if kind == "fit":
        _, _, _, target, prm, pairs, tt = _fit_inputs(case, seed)
        prm = [p.clone().requires_grad_(True) for p in prm]
        f = _fit_forces(case, prm[0] if case["pot"] == "morse" else prm, pairs, tt)
        loss = ((f - target) ** 2).mean()
        return {"loss": loss.detach(), "grads": list(torch.autograd.grad(loss, prm))}
    if kind == "replicas":
        ss = _replica_systems(case, seed)
        md = _Md(ss, case["pot"])
        md.advance(case["steps"])
        rep = torch.as_tensor(np.repeat(np.arange(len(ss)), [s.n for s in ss]), device="cuda")
        per = lambda x: torch.zeros(len(ss), dtype=torch.float64,  # noqa: E731
                                    device="cuda").index_add(0, rep, x)
        return {"pos": md.pos, "vel": md.vel, "frc": md.f, "pe": per(md.pe), "ke": per(md.ke())}
    md = _Md([_system(case, seed)], case["pot"])
    if kind == "compute":
        out = {"frc": md.f, "pe": md.pe.sum().reshape(1), "virial": md.vir}
        return out if case["pot"] == "morse" else dict(out, rho=md.rho, fp=md.fp)
    md.advance(case["steps"], _Chain(case["temp"], 3 * md.n - 3) if case["nvt"] else None)
    out = {"pos": md.pos, "vel": md.vel, "frc": md.f}
    if case["thermo"]:
        out.update(pe=md.pe.sum().reshape(1), ke=md.ke().sum().reshape(1), virial=md.vir)
    return out
