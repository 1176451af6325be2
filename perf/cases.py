"""Performance cases: the work a user of this library has it do, through the Python mirror (mdgpu) and the C-ABI
under it, from the smallest calls to the largest runs.

Kinds of case:
  step     a user's own loop over VelocityVerletIntegrator.step, then one trajectory frame (writeXyzFrame's data)
  run      md_run: a device-resident run with its thermostat, g(r) samples and per-step records, then one frame
  frames   analysis of a stored frame: upload, list build, forces and energies, download
  brute    the O(N^2) step (md_sim --brute)
  batch    many replicas advanced together (md_batch_run), their records and final states
  adjoint  trajectory gradients: forward and backward

Every start is an FCC lattice with a few sites left empty (so that sizes are odd) and Maxwell-Boltzmann velocities,
as md_sim starts; `equil` steps of velocity rescaling melt it in `prepare` where a case stands for production in the
liquid. A state keeps its system, list, force field and pinned host buffers from pass to pass, as a program does.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "molecular-dynamics_b200"))
import mdgpu as md  # noqa: E402

PRECISION = {"fp64": md.PREC_FP64, "fp32fx": md.PREC_FP32FX, "fp32": md.PREC_FP32, "fx64": md.PREC_FX64,
             "fx32": md.PREC_FX32}
DT = 0.005
BINS = 100


def listed():
    return [
        # the smallest call: one 500-atom NIST replica stepped from the user's own loop
        dict(name="step_500_fp64", kind="step", cells=5, empty=0, rho=0.776, temp=0.85, rc=3.0, skin=0.2,
             precision="fp64", steps=10),
        # md_sim's default system in the default precision: Bussi NVT with g(r) every 10 steps
        dict(name="run_2048_fp64_bussi_rdf", kind="run", cells=8, empty=0, rho=0.8442, temp=0.71, rc=2.5, skin=0.3,
             precision="fp64", steps=256, thermostat="bussi", rdf_every=10, equil=0),
        # equilibration of a mid-sized system from its lattice (rescale every 10 steps), one atom short of 32,000
        dict(name="run_31999_fx32_rescale", kind="run", cells=20, empty=1, rho=0.8442, temp=1.5, rc=2.5, skin=0.3,
             precision="fx32", steps=128, thermostat="rescale", rdf_every=0, equil=0),
        # the precision sweep's system: NVE production in the mixed precision the reference calls --mixed
        dict(name="run_256000_fp32fx", kind="run", cells=40, empty=0, rho=0.8442, temp=0.71, rc=2.5, skin=0.3,
             precision="fp32fx", steps=128, thermostat="none", rdf_every=0, equil=100),
        # a large production run in the reference's own precision, energies of every step
        dict(name="run_864000_fp64", kind="run", cells=60, empty=0, rho=0.8442, temp=0.71, rc=2.5, skin=0.3,
             precision="fp64", steps=128, thermostat="none", rdf_every=0, equil=60),
        # the headline workload: 4M atoms in the headline precision
        dict(name="run_4000000_fx32", kind="run", cells=100, empty=0, rho=0.8442, temp=0.71, rc=2.5, skin=0.3,
             precision="fx32", steps=128, thermostat="none", rdf_every=0, equil=100),
        # re-evaluating a stored frame of odd size: upload, list, forces, download
        dict(name="frames_97333_fx64", kind="frames", cells=29, empty=223, rho=0.8442, temp=0.0, rc=2.5, skin=0.3,
             precision="fx64"),
        # the all-pairs step, the reference's check of its list path
        dict(name="brute_4000_fp64", kind="brute", cells=10, empty=0, rho=0.8442, temp=0.71, rc=2.5, skin=0.0,
             precision="fp64", steps=1),
        # NIST validation's production phase: 16 state points x 8 replicas of 500 atoms, every step recorded
        dict(name="batch_nist_128x500_fp64", kind="batch", replicas=128, cells_lo=5, cells_hi=5, rho_lo=0.776,
             rho_hi=0.9, temp_lo=0.85, temp_hi=0.9, rc=3.0, skin=0.2, precision="fp64", steps=100,
             thermostat="bussi", tau=0.5, energy_every=1),
        # uneven replicas of many state points under Bussi
        dict(name="batch_96_uneven_fp32fx", kind="batch", replicas=96, cells_lo=4, cells_hi=20, rho_lo=0.7,
             rho_hi=0.95, temp_lo=0.7, temp_hi=2.0, rc=2.5, skin=0.3, precision="fp32fx", steps=100,
             thermostat="bussi", tau=0.1, energy_every=10),
        # trajectory gradients with respect to epsilon, sigma and the initial state
        dict(name="adjoint_32000", kind="adjoint", cells=20, empty=0, rho=0.8442, temp=1.0, rc=2.5, skin=0.3,
             precision="fp64", steps=50, every=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "run", "run", "run", "frames", "brute", "batch", "adjoint"])
    rho, temp = round(rng.uniform(0.7, 0.95), 4), round(rng.uniform(0.7, 2.0), 3)
    rc, skin = rng.choice([(2.5, 0.3), (2.5, 0.3), (3.0, 0.2), (2.5, 0.4)])

    def lattice(lo, hi):  # cells per side over the logarithm of the size, and up to 1 % of the sites empty
        cells = _log_int(rng, lo, hi)
        return dict(cells=cells, empty=rng.randint(0, max(1, 4 * cells ** 3 // 100)))

    base = dict(kind=kind, rho=rho, temp=temp, rc=rc, skin=skin)
    if kind == "step":
        return {**base, **lattice(5, 20), "precision": rng.choice(list(PRECISION)), "steps": 10}
    if kind == "run":
        precision = rng.choice(list(PRECISION))
        lat = lattice(5, 60 if precision == "fp64" else 90)
        return {**base, **lat, "precision": precision, "steps": rng.randint(128, 200 if lat["cells"] < 60 else 140),
                "thermostat": rng.choice(["none", "rescale", "bussi"]), "rdf_every": rng.choice([0, 0, 10]),
                "equil": 0 if lat["cells"] <= 20 else 60}
    if kind == "frames":
        return {**base, **lattice(5, 60), "precision": rng.choice(list(PRECISION))}
    if kind == "brute":
        return {**base, **lattice(5, 9), "precision": "fp64", "skin": 0.0, "steps": 1}
    if kind == "batch":
        lo = rng.randint(5, 8)
        hi = rng.randint(lo, 12)
        return {**base, "replicas": _log_int(rng, 4, 128), "cells_lo": lo, "cells_hi": hi, "rho_lo": 0.7, "rho_hi": rho,
                "temp_lo": 0.7, "temp_hi": temp, "precision": rng.choice(["fp64", "fp32fx", "fp32"]),
                "steps": rng.randint(50, 100), "thermostat": rng.choice(["none", "rescale", "bussi"]), "tau": 0.1,
                "energy_every": rng.choice([0, 1, 10])}
    return {**base, **lattice(5, 18), "precision": "fp64", "steps": rng.randint(10, 50), "every": rng.choice([10, 20])}


# ---- inputs --------------------------------------------------------------------------------------------------


def _start(cells, empty, rho, temp, seed, jitter=0.0):
    """(positions (n, 4), box, velocities (3, n)) in host arrays: lattice sites (md_sim's basis), `empty` of them
    left out, at number density rho; velocities of temperature temp without net momentum."""
    g = torch.Generator(device="cuda").manual_seed(1 + seed)
    sites = 4 * cells ** 3
    n = sites - empty
    box = (n / rho) ** (1.0 / 3.0)
    k = torch.arange(cells, device="cuda", dtype=torch.float64)
    grid = torch.stack(torch.meshgrid(k, k, k, indexing="ij"), dim=-1).reshape(-1, 1, 3)
    basis = torch.tensor([[0.0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]], device="cuda", dtype=torch.float64)
    pos = ((grid + basis + 0.25) * (box / cells)).reshape(-1, 3)
    if empty:
        keep = torch.randperm(sites, generator=g, device="cuda")[:n].sort().values
        pos = pos[keep]
    if jitter:
        pos = pos + jitter * torch.randn(pos.shape, generator=g, device="cuda", dtype=torch.float64)
        pos = pos - box * torch.floor(pos / box)
    pos4 = torch.zeros((n, 4), dtype=torch.float64, device="cuda")
    pos4[:, :3] = pos
    vel = torch.randn((3, n), generator=g, device="cuda", dtype=torch.float64) * math.sqrt(max(temp, 0.0))
    vel -= vel.mean(dim=1, keepdim=True)
    return pos4.cpu().numpy(), box, vel.cpu().numpy()


def _draws(n, steps, seed):
    """Bussi draws of `steps` steps, given to md_run by the caller."""
    r = np.random.default_rng(7 + seed)
    return r.standard_normal(steps), r.gamma(0.5 * (3 * n - 4), 2.0, steps)


def _systems(case, seed):
    """The replicas of a batch: sizes, densities and temperatures spread over the case's ranges (the same for every
    seed, which makes the velocities)."""
    r = np.random.default_rng(11)
    out, temps = [], []
    for k in range(case["replicas"]):
        cells = int(r.integers(case["cells_lo"], case["cells_hi"] + 1))
        rho, temp = r.uniform(case["rho_lo"], case["rho_hi"]), r.uniform(case["temp_lo"], case["temp_hi"])
        least = math.ceil(2.0 * (case["rc"] + case["skin"]) * (rho / 4.0) ** (1.0 / 3.0) + 0.01)  # the box holds the list
        pos, box, vel = _start(max(cells, least), 0, rho, temp, 1000 * seed + k)
        out.append((pos, box, vel, np.ones(len(pos))))
        temps.append(temp)
    return out, np.array(temps)


def _pinned(shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def _at(t, kind=C.c_double):
    return C.cast(t.data_ptr(), C.POINTER(kind))


def _frame(st):
    """(n, 6) positions and velocities in id order into the state's pinned buffer"""
    md._check(md.LIB.md_system_frame_by_id(st["s"].h, _at(st["frame"]), 1))
    return st["frame"]


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "batch":
        systems, temps = _systems(case, seed)
        st["b"] = md.Batch(systems, cutoff=case["rc"], skin=case["skin"], dt=DT, precision=PRECISION[case["precision"]],
                           thermostat=case["thermostat"], temperatures=temps, seeds=1000 + seed + np.arange(len(systems)),
                           rescale_every=10, bussi_tau=case["tau"], energy_every=case["energy_every"])
        atoms = int(st["b"].n.sum())
        st["pos"], st["vel"], st["ids"] = _pinned((atoms, 4)), _pinned((3 * atoms,)), _pinned((atoms,), torch.int64)
        return st
    if kind == "frames":
        pos, box, _ = _start(case["cells"], case["empty"], case["rho"], 0.0, seed, jitter=0.06)
        st["pos"], st["ids"] = pos, np.arange(len(pos), dtype=np.uint64)
        st["s"] = md.System(len(pos), box)
        st["nl"] = md.NeighbourList(case["rc"], case["skin"], reverse_index=True)
        st["ff"] = md.LennardJonesForceField(1.0, 1.0, case["rc"], PRECISION[case["precision"]])
        st["force"], st["order"] = _pinned((3, len(pos))), _pinned((len(pos),), torch.int64)
        return st
    pos, box, vel = _start(case["cells"], case["empty"], case["rho"], case["temp"], seed)
    if kind == "adjoint":
        st["a"] = md.Adjoint(pos, box, vel, cutoff=case["rc"], skin=case["skin"], dt=DT, steps=case["steps"],
                             checkpoint_every=case["every"])
        return st
    st["s"] = md.System.from_arrays(pos, box, vel=vel)
    st["ff"] = md.LennardJonesForceField(1.0, 1.0, case["rc"], PRECISION[case["precision"]])
    st["vv"] = md.VelocityVerletIntegrator(DT)
    st["frame"] = _pinned((len(pos), 6))
    if kind == "brute":
        st["ff"].compute_forces(st["s"])
        return st
    st["nl"] = md.NeighbourList(case["rc"], case["skin"], reverse_index=True)
    st["nl"].build(st["s"])
    st["ff"].compute_forces(st["s"], st["nl"])
    if kind == "run":
        st["options"] = dict(thermostat=case["thermostat"], rescale_temperature=case["temp"])
        if case["thermostat"] == "bussi":
            r1, chi2 = _draws(len(pos), case["steps"], seed)
            st["options"].update(bussi_temperature=case["temp"], bussi_r1=r1, bussi_chi2=chi2)
        if case["rdf_every"]:
            st["rdf"] = md.RadialDistribution(case["rc"], BINS)
            st["options"].update(rdf=st["rdf"], rdf_every=case["rdf_every"])
        if case["equil"]:
            st["vv"].run(st["s"], st["ff"], st["nl"], case["equil"], thermostat="rescale",
                         rescale_temperature=case["temp"], record=False)
    return st


# ---- one pass ------------------------------------------------------------------------------------------------


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "step":
        pe = [st["vv"].step(st["s"], st["ff"], st["nl"]) for _ in range(case["steps"])]
        return {"pe": pe, "virial": st["ff"].virial, "inside": st["ff"].inside_pairs, "frame": _frame(st)}
    if kind == "run":
        pe, ke, w = st["vv"].run(st["s"], st["ff"], st["nl"], case["steps"], **st["options"])
        out = {"pe": pe, "ke": ke, "virial": w, "frame": _frame(st)}
        if "rdf" in st:
            out["histogram"] = st["rdf"].histogram()
        return out
    if kind == "frames":
        st["s"].upload(pos=st["pos"], ids=st["ids"])
        st["nl"].build(st["s"])
        pe = st["ff"].compute_forces(st["s"], st["nl"])
        md._check(md.LIB.md_system_download(st["s"].h, None, None, _at(st["force"]), None, _at(st["order"], C.c_uint64)))
        return {"pe": pe, "virial": st["ff"].virial, "inside": st["ff"].inside_pairs, "force": st["force"],
                "order": st["order"]}
    if kind == "brute":
        pe = [st["vv"].step(st["s"], st["ff"]) for _ in range(case["steps"])]
        return {"pe": pe, "virial": st["ff"].virial, "inside": st["ff"].inside_pairs, "frame": _frame(st)}
    if kind == "batch":
        b = st["b"]
        rec = b.run(case["steps"], inside=True)
        at = 0
        for r, n in enumerate(b.n.tolist()):
            md._check(md.LIB.md_batch_download(b.h, r, _at(st["pos"][at:]), _at(st["vel"][3 * at:]), None, None,
                                               _at(st["ids"][at:], C.c_uint64)))
            at += n
        out = {"pos": st["pos"], "vel": st["vel"], "ids": st["ids"]}
        return {**out, "records": rec} if rec is not None else out
    u, p, us, ws, ks = st["a"].forward(record=True)
    return {"mean_pe": u, "mean_pressure": p, "pe": us, "virial": ws, "ke": ks, "grad": st["a"].backward(1.0, 1.0)}


# ---- what a pass cannot do without ------------------------------------------------------------------------------


def _atoms(case):
    if case["kind"] == "batch":
        c = 0.5 * (case["cells_lo"] + case["cells_hi"])
        return case["replicas"] * 4.0 * c ** 3
    return 4.0 * case["cells"] ** 3 - case["empty"]


def work(case):
    """Every particle's position (32 B), velocity (24 B) and mass (8 B) read and position and velocity written: at
    every step where that outgrows the 126 MB L2, once for the pass where it does not; about 30 operations per pair
    inside the cutoff and 60 per particle for the step itself."""
    n, kind = _atoms(case), case["kind"]
    pairs = n * 0.5 * 4.18879 * case["rc"] ** 3 * case["rho"] if kind != "batch" else \
        n * 0.5 * 4.18879 * case["rc"] ** 3 * 0.5 * (case["rho_lo"] + case["rho_hi"])
    sweeps = case.get("steps", 1) if n * 120 > 126e6 else 1
    if kind == "frames":  # positions and ids up, forces and ids down
        return {"bytes": n * (32 + 8 + 24 + 8), "flops": 30.0 * pairs}
    if kind == "brute":  # every pair's separation is tested
        return {"bytes": sweeps * n * 120.0, "flops": case["steps"] * (0.5 * n * n * 14.0 + 30.0 * pairs)}
    if kind == "adjoint":  # forward, recomputation and two Hessian-vector passes a step
        return {"bytes": 4 * sweeps * n * 120.0, "flops": case["steps"] * pairs * (2 * 30.0 + 2 * 80.0)}
    return {"bytes": sweeps * n * 120.0, "flops": case["steps"] * (30.0 * pairs + 60.0 * n)}


# ---- the same in 64 bits, in plain torch ------------------------------------------------------------------------


class _World:
    """Systems side by side in one array: pairs inside each box by a chunked all-pairs search, redone every `every`
    steps with a margin that no particle crosses in between."""

    def __init__(self, systems, rc, eps=1.0, sigma=1.0, margin=0.8, every=8):
        dev = "cuda"
        self.n = [len(p) for p, *_ in systems]
        self.pos = torch.cat([torch.as_tensor(np.asarray(p)[:, :3], device=dev) for p, *_ in systems])
        self.vel = torch.cat([torch.as_tensor(np.asarray(v).T.copy(), device=dev) for _, _, v in systems])
        self.box = torch.tensor([b for _, b, _ in systems], dtype=torch.float64, device=dev)
        self.rep = torch.repeat_interleave(torch.arange(len(systems), device=dev), torch.tensor(self.n, device=dev))
        self.L = self.box[self.rep].unsqueeze(1)
        self.rc, self.eps, self.sigma, self.margin, self.every = rc, eps, sigma, margin, every
        self.dof = 3.0 * torch.tensor(self.n, dtype=torch.float64, device=dev) - 3.0
        self.search()

    def search(self):
        at, I, J = 0, [], []
        with torch.no_grad():
            for r, n in enumerate(self.n):
                x, L = self.pos[at:at + n].detach(), float(self.box[r])
                step = max(1, min(n, 40_000_000 // max(n, 1)))
                for a in range(0, n, step):
                    y = x[a:a + step]
                    r2 = torch.zeros((len(y), n), dtype=torch.float64, device=x.device)
                    for k in range(3):
                        d = y[:, k:k + 1] - x[:, k].unsqueeze(0)
                        d = d - L * torch.round(d / L)
                        r2 += d * d
                    hit = r2 < (self.rc + self.margin) ** 2
                    i, j = torch.nonzero(hit, as_tuple=True)
                    i = i + a
                    keep = i < j
                    I.append(i[keep] + at)
                    J.append(j[keep] + at)
                at += n
        self.i, self.j = torch.cat(I), torch.cat(J)

    def forces(self):
        """Forces, and per system energy, virial and pairs inside the cutoff"""
        i, j = self.i, self.j
        d = self.pos[i] - self.pos[j]
        L = self.L[i]
        d = d - L * torch.round(d.detach() / L)
        r2 = (d * d).sum(dim=1)
        inside = r2.detach() < self.rc ** 2
        i, j, d, r2 = i[inside], j[inside], d[inside], r2[inside]
        s6 = (self.sigma ** 2 / r2) ** 3
        c6 = (self.sigma / self.rc) ** 6
        e = 4 * self.eps * (s6 * s6 - s6) - 4 * self.eps * (c6 * c6 - c6)
        f = 24 * self.eps * (2 * s6 * s6 - s6) / r2
        fd = f.unsqueeze(1) * d
        force = torch.zeros_like(self.pos).index_add(0, i, fd).index_add(0, j, -fd)
        zero = torch.zeros(len(self.n), dtype=torch.float64, device=d.device)
        self.r2 = r2.detach()
        return (force, zero.index_add(0, self.rep[i], e), zero.index_add(0, self.rep[i], f * r2),
                zero.index_add(0, self.rep[i], torch.ones_like(r2.detach())))

    def kinetic(self):
        zero = torch.zeros(len(self.n), dtype=torch.float64, device=self.pos.device)
        return zero.index_add(0, self.rep, 0.5 * (self.vel * self.vel).sum(dim=1))

    def step(self, k, force):
        """Step k (1-based) of velocity Verlet; returns the new (force, energy, virial, inside)"""
        self.vel = self.vel + 0.5 * DT * force
        p = self.pos + DT * self.vel
        self.pos = p - self.L * torch.floor(p.detach() / self.L)
        if k % self.every == 0:
            self.search()
        out = self.forces()
        self.vel = self.vel + 0.5 * DT * out[0]
        return out

    def scale(self, factor):
        self.vel = self.vel * factor[self.rep].unsqueeze(1)


def _heavy(case):
    """Would the 64-bit values take long? (pair tests of the searches, 1e10 a second or so)"""
    if case["kind"] == "batch":
        n2 = case["replicas"] * (4.0 * case["cells_hi"] ** 3) ** 2
    else:
        n2 = _atoms(case) ** 2
    return n2 * (1 + case.get("steps", 0) // 8) > 4e10


def exact(case, seed):
    kind = case["kind"]
    if _heavy(case) or case.get("equil", 0) or (kind == "batch" and case["thermostat"] == "bussi"):
        return None  # too many pairs, a start that the library melted, or draws of its own generator
    num = lambda t: float(t[0].detach())  # noqa: E731
    if kind == "frames":
        pos, box, vel = _start(case["cells"], case["empty"], case["rho"], 0.0, seed, jitter=0.06)
        w = _World([(pos, box, vel)], case["rc"], margin=0.0)
        f, pe, vir, inside = w.forces()
        per_side = int(box / (case["rc"] + case["skin"]))  # the particles come back sorted by cell
        c = torch.clamp((w.pos * (per_side / box)).to(torch.int64), max=per_side - 1)
        order = torch.argsort((c[:, 0] * per_side + c[:, 1]) * per_side + c[:, 2], stable=True)
        return {"pe": num(pe), "virial": num(vir), "inside": num(inside), "force": f[order].T.contiguous(), "order": None}
    if kind == "batch":
        systems, temps = _systems(case, seed)
        w = _World([(p, b, v) for p, b, v, _ in systems], case["rc"])
    else:
        w = _World([_start(case["cells"], case["empty"], case["rho"], case["temp"], seed)], case["rc"])
        temps = np.array([case["temp"]])
    if kind == "adjoint":
        return _exact_adjoint(case, w)
    target = torch.as_tensor(temps, device="cuda")
    r1, chi2 = _draws(sum(w.n), case["steps"], seed) if case.get("thermostat") == "bussi" else (None, None)
    hist = np.zeros(BINS)
    force = w.forces()[0]
    rec = []
    for k in range(1, case["steps"] + 1):
        force, pe, vir, inside = w.step(k, force)
        if case.get("thermostat") == "rescale" and k % 10 == 0:
            w.scale(torch.sqrt(target * w.dof / (2 * w.kinetic())))
        elif case.get("thermostat") == "bussi":
            c, ke, half = math.exp(-DT / 0.5), w.kinetic(), 0.5 * w.dof * target
            new = ke + (1 - c) * (half * (chi2[k - 1] + r1[k - 1] ** 2) / w.dof - ke) + \
                2 * r1[k - 1] * torch.sqrt(half / w.dof * ke * (1 - c) * c)
            w.scale(torch.sqrt(new / ke))
        if case.get("rdf_every") and k % case["rdf_every"] == 0:
            b = (torch.sqrt(w.r2) / (case["rc"] / BINS)).to(torch.int64)
            hist += torch.bincount(b[b < BINS], minlength=BINS).cpu().numpy()
        rec.append((pe, vir, w.kinetic(), inside))
    frame = torch.cat([w.pos, w.vel], dim=1)
    if kind == "batch":
        out = {"pos": None, "vel": None, "ids": None}  # in the list's order
        every = case["energy_every"]
        if not every or case["steps"] < every:
            return out
        rows = [rec[k - 1] for k in range(every, case["steps"] + 1, every)]
        return {**out, "records": tuple(torch.stack([r[q] for r in rows]) for q in range(4))}
    if kind == "run":
        out = {"pe": torch.cat([r[0] for r in rec]), "ke": torch.cat([r[2] for r in rec]),
               "virial": torch.cat([r[1] for r in rec]), "frame": frame}
        return {**out, "histogram": hist} if case["rdf_every"] else out
    return {"pe": [num(r[0]) for r in rec], "virial": num(rec[-1][1]), "inside": num(rec[-1][3]), "frame": frame}


def _exact_adjoint(case, w):
    eps = torch.tensor(1.0, dtype=torch.float64, device="cuda", requires_grad=True)
    sigma = torch.tensor(1.0, dtype=torch.float64, device="cuda", requires_grad=True)
    pos = w.pos.clone().requires_grad_(True)
    vel = w.vel.clone().requires_grad_(True)
    w.pos, w.vel, w.eps, w.sigma = pos, vel, eps, sigma
    force = w.forces()[0]
    U, W, K = [], [], []
    for k in range(1, case["steps"] + 1):
        force, pe, vir, _ = w.step(k, force)
        U.append(pe[0])
        W.append(vir[0])
        K.append(w.kinetic()[0])
    U, W, K = torch.stack(U), torch.stack(W), torch.stack(K)
    mean_u, mean_p = U.mean(), ((2 * K + W) / (3 * w.box[0] ** 3)).mean()
    g = torch.autograd.grad(mean_u + mean_p, (eps, sigma, pos, vel))
    return {"mean_pe": float(mean_u.detach()), "mean_pressure": float(mean_p.detach()), "pe": U.detach(),
            "virial": W.detach(), "ke": K.detach(),
            "grad": {"d_epsilon": float(g[0]), "d_sigma": float(g[1]), "d_pos": g[2].T.contiguous(),
                     "d_vel": g[3].T.contiguous()}}
