"""The workloads whose speed is followed: force evaluations, energies, dynamics,
replica exchange and parameter gradients, through the package's public entry
points, over the sizes and settings its users run.

Three families share the ranges:

* liquids and solvated solutes in a periodic box (LJ + Coulomb with PD's energy
  or force switch): 300 to 8,000 generated waters, the solvated 120-residue
  peptide (22,489 atoms) and its periodic copies (up to 179,912 atoms);
* peptides in implicit solvent (GB, with or without the LCPO surface term and
  the bonded terms), all pairs or PD's default 15 / 12 A cutoffs: 525 to 7,741
  atoms one at a time, and batches of up to 64;
* parameter fitting over frames of one system.

Pair arithmetic and force accumulation inputs are 32-bit (forces agree with PD's
FP64 to ~2e-6), so the programs here keep forces, trajectories, gradients and GB
energies in 32 bits; FF_NonBonded energies are FP64 and stay so.
"""
import functools
import math

import numpy as np
import torch

from pd_gb300 import (FF_Bonded_GPU, FF_GeneralizedBorn_Still_GPU, FF_NonBonded_GPU, FF_SASA_LCPO_GPU, Forcefield,
                      SystemImage, WorkSpace, ffi, load_workload)
from pd_gb300.adjoint import FrameSet
from pd_gb300.engine import DeviceContext
from pd_gb300.md import maxwell_boltzmann

NA, KCAL = 6.0221418e23, 4184.0
TO_J = KCAL / NA                         # kcal/mol -> J per molecule
ECONV = (NA / KCAL) * 1.60217645e-19 ** 2 / (4.0 * math.pi * 8.854187817e-12 * 1e-10)


def listed():
    return [
        # one call of the whole force field on the smallest peptide: a minimiser's
        # or a Monte Carlo program's inner call, bound by latency
        {"name": "peptide-33-forces", "kind": "gb_forces", "system": "c4_remd64", "first": 51, "count": 1,
         "cutoff": 0.0, "whole": True, "rebuild": False},
        # GB forces of a 256-residue peptide with no cutoff, successive calls
        {"name": "peptide-256-forces", "kind": "gb_forces", "system": "c3_gb256", "first": 0, "count": 1,
         "cutoff": 0.0, "whole": False, "rebuild": False},
        # the same with PD's default cutoffs (15 / 12 A, Still cutoff 10 A) on
        # unrelated conformations, a new list each (rescoring a decoy set)
        {"name": "peptide-256-cutoff", "kind": "gb_forces", "system": "c3_gb256", "first": 0, "count": 1,
         "cutoff": 15.0, "whole": False, "rebuild": True},
        # Forcefield.calcEnergies of the GB component (a Monte Carlo step)
        {"name": "peptide-256-energies", "kind": "gb_energies", "system": "c3_gb256", "first": 0, "count": 1,
         "cutoff": 0.0},
        # LJ + Coulomb of a small water box, successive calls
        {"name": "water-667-forces", "kind": "nb_forces", "system": "water", "waters": 667, "copies": 1,
         "mode": "energy", "cutoff": 12.0, "inner": 10.0, "padding": 2.0, "rebuild": False},
        # PD's default FF_NonBonded (force switch, 15 / 12 A) on new coordinates
        # of the solvated peptide, a new list each
        {"name": "solvated-22k-forces", "kind": "nb_forces", "system": "c2_solvated", "waters": 0, "copies": 1,
         "mode": "force", "cutoff": 15.0, "inner": 12.0, "padding": 0.5, "rebuild": True},
        # dynamics: the small water box (velocity Verlet), the solvated peptide
        # and eight copies of it (Langevin)
        {"name": "water-667-md", "kind": "nb_md", "system": "water", "waters": 667, "copies": 1, "steps": 20,
         "cadence": 5, "langevin": False},
        {"name": "solvated-22k-md", "kind": "nb_md", "system": "c2_solvated", "waters": 0, "copies": 1, "steps": 20,
         "cadence": 5, "langevin": True},
        {"name": "solvated-180k-md", "kind": "nb_md", "system": "c2_solvated", "waters": 0, "copies": 8, "steps": 10,
         "cadence": 5, "langevin": True},
        # implicit-solvent dynamics of one peptide, and a replica-exchange round
        # of 64 uneven peptides (steps, energies, exchange sweep)
        {"name": "peptide-256-md", "kind": "gb_md", "system": "c3_gb256", "first": 0, "count": 1, "steps": 20,
         "cadence": 20, "exchange": False},
        {"name": "remd-64", "kind": "gb_md", "system": "c4_remd64", "first": 0, "count": 64, "steps": 20,
         "cadence": 20, "exchange": True},
        # a fitting step: energies of 16 frames and their parameter gradients
        {"name": "fit-16-frames", "kind": "fit", "system": "c3_gb256", "waters": 0, "first": 0, "frames": 16,
         "cutoff": 0.0},
    ]


def draw(rng):
    kind = rng.choice(["gb_forces", "gb_energies", "nb_forces", "nb_forces", "nb_md", "gb_md", "fit", "fit"])
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    liquid = rng.random() < 0.7
    box = {"system": "water" if liquid else "c2_solvated", "waters": log(300, 8000) if liquid else 0,
           "copies": 1 if liquid else rng.choice([1, 1, 2, 4])}
    pep = {"system": "c4_remd64", "first": rng.randrange(64), "count": min(64, log(1, 24))}
    gbcut = rng.choice([0.0, 0.0, 12.0, 13.5, 15.0])
    if kind == "gb_forces":
        return dict(pep, kind=kind, cutoff=gbcut, whole=rng.random() < 0.3, rebuild=rng.random() < 0.5)
    if kind == "gb_energies":
        return dict(pep, kind=kind, cutoff=gbcut)
    if kind == "nb_forces":
        cut = round(rng.uniform(9.0, 15.0), 2)
        return dict(box, kind=kind, mode=rng.choice(["energy", "force", "plain"]), cutoff=cut,
                    inner=round(cut - rng.uniform(1.0, 3.0), 2), padding=rng.choice([0.5, 1.0, 2.0]),
                    rebuild=rng.random() < 0.5)
    if kind == "nb_md":
        return dict(box, kind=kind, steps=rng.choice([5, 10, 15, 20]), cadence=5, langevin=rng.random() < 0.5)
    if kind == "gb_md":
        return dict(pep, kind=kind, steps=rng.choice([5, 10, 20]), cadence=rng.choice([5, 10, 20]),
                    exchange=pep["count"] > 1 and rng.random() < 0.5)
    if rng.random() < 0.5:
        return {"kind": "fit", "system": "water", "waters": log(300, 1500), "first": 0, "frames": log(1, 16),
                "cutoff": 10.0}
    return {"kind": "fit", "system": "c4_remd64", "waters": 0, "first": rng.randrange(64), "frames": log(1, 8),
            "cutoff": gbcut}


# ---------------------------------------------------------------------------
# systems
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def image_file(name):
    return load_workload(name)


@functools.lru_cache(maxsize=4)
def water_image(n):
    """n TIP3P-style waters at 31.2 A^3 each: molecules on random sites of a cubic
    lattice in random orientations (positions are drawn per seed)."""
    w = image_file("c1_water")
    rep = lambda a: np.tile(a[:3], n)
    off = 3 * np.arange(n)
    idx = lambda t, k: (np.concatenate([t[0][:k] + o for o in off]), np.tile(t[1][:k], (n, 1)))
    excl = np.concatenate([w.excl[:3] + np.array([o, o, 0]) for o in off])
    L = (31.2 * n) ** (1.0 / 3.0)
    return SystemImage([3 * n], [L, L, L], rep(w.charge), rep(w.radius), rep(w.epsilon), rep(w.mass), excl,
                       bonds=idx(w.bonds, 2), angles=idx(w.angles, 1), scaling14=w.scaling14)


def water_positions(n, rng):
    m = int(math.ceil(n ** (1.0 / 3.0) - 1e-9))
    L = (31.2 * n) ** (1.0 / 3.0)
    site = rng.permutation(m ** 3)[:n]
    o = (np.stack([site // (m * m), site // m % m, site % m], 1) + 0.5) * (L / m) - 0.5 * L
    o = o + rng.uniform(-0.1, 0.1, (n, 3))
    q = rng.standard_normal((n, 4))
    a, b, c, d = (q / np.linalg.norm(q, axis=1)[:, None]).T
    R = np.stack([a*a+b*b-c*c-d*d, 2*(b*c-a*d), 2*(b*d+a*c), 2*(b*c+a*d), a*a-b*b+c*c-d*d, 2*(c*d-a*b),
                  2*(b*d-a*c), 2*(c*d+a*b), a*a-b*b-c*c+d*d], 1).reshape(n, 3, 3)
    h = 0.5 * 1.82421813
    mol = 0.9572 * np.array([[0, 0, 0], [math.sin(h), math.cos(h), 0], [-math.sin(h), math.cos(h), 0]])
    return (o[:, None, :] + np.einsum("nij,kj->nki", R, mol)).reshape(-1, 3)


@functools.lru_cache(maxsize=6)
def image_of(system, waters, copies, first, count):
    if system == "water":
        return water_image(waters)
    im = image_file(system)
    if system == "c4_remd64" and count < im.nsystems:
        parts = [im.subset((first + k) % im.nsystems) for k in range(count)]
        return parts[0] if count == 1 else SystemImage.concat(parts)
    if copies > 1:
        return im.replicate({2: (2, 1, 1), 4: (2, 2, 1), 8: (2, 2, 2)}[copies])
    return im


def image(case):
    return image_of(case["system"], case.get("waters", 0), case.get("copies", 1), case.get("first", 0),
                    case.get("count", 1))


def positions(case, seed):
    """This seed's coordinates: new waters, or the built structure with every
    atom displaced by a thermal amplitude."""
    rng = np.random.default_rng(seed)
    if case["system"] == "water":
        return water_positions(case["waters"], rng)
    im = image(case)
    return im.pos + 0.02 * rng.standard_normal(im.pos.shape)


def nb_settings(case, im):
    mode = case.get("mode", "energy")
    cut, inner = case.get("cutoff", 12.0), case.get("inner", 10.0)
    if case["system"] == "water":   # a box holds twice its cutoff
        f = min(1.0, 0.49 * float(im.box.min()) / cut)
        cut, inner = cut * f, inner * f
    return dict(Cutoff=cut, InnerCutoff=inner, VdwCutoff=cut, VdwInnerCutoff=inner,
                Vdw14Scaling=float(im.scaling14[0]), Elec14Scaling=float(im.scaling14[1]), Dielectric=1.0,
                EnergySwitch=int(mode == "energy"), ForceSwitch=int(mode == "force"), DoVdw=1, DoElec=1)


def gb_settings(case, im):
    cut = case.get("cutoff", 0.0)
    c, i, still = (cut, cut - 3.0, 10.0) if cut else (999.0, 998.0, 999.0)
    return dict(Cutoff=c, InnerCutoff=i, VdwCutoff=c, VdwInnerCutoff=i, Vdw14Scaling=float(im.scaling14[0]),
                Elec14Scaling=float(im.scaling14[1]), DielectricSolute=1.0, DielectricSolvent=80.0,
                GbsaStillCutoff=still, ExpApproxThreshold=-4.0, BornRadiusOffset=0.0, P4=float(im.gb_P[3]),
                P5=float(im.gb_P[4]))


def set_attributes(component, settings):
    for k, v in settings.items():
        if hasattr(component, k):
            setattr(component, k, v)
    component.AutoScaling14 = True


# ---------------------------------------------------------------------------
# programs
# ---------------------------------------------------------------------------
def prepare(case, seed):
    im = image(case)
    pos = positions(case, seed)
    s = {"case": case, "image": im, "pos": pos}
    kind = case["kind"]
    if kind in ("nb_forces", "gb_forces", "gb_energies"):
        ws = WorkSpace(im, positions=pos)
        ff = Forcefield(ws)
        if kind == "nb_forces":
            ws.Padding = case["padding"]
            nb = FF_NonBonded_GPU(ws)
            set_attributes(nb, nb_settings(case, im))
            ff.add(nb)
        else:
            ws.Padding = 2.0
            gb = FF_GeneralizedBorn_Still_GPU(ws)
            set_attributes(gb, gb_settings(case, im))
            ff.add(gb)
            if case.get("whole"):
                sa = FF_SASA_LCPO_GPU(ws)
                sa.GlobalASP = 0.005
                ff.add(sa)
                ff.add(FF_Bonded_GPU(ws))
        s.update(ws=ws, ff=ff)
    elif kind in ("nb_md", "gb_md"):
        ctx = DeviceContext(im)
        what = ffi.BONDED
        if kind == "nb_md":
            ctx.set_nb(**nb_settings(case, im))
            what |= ffi.NB
        else:
            ctx.set_gb(**gb_settings(case, im))
            what |= ffi.GB | ffi.SA
        ctx.set_list(2.0)
        ctx.set_positions(pos)
        n = im.nsystems
        temps = 300.0 * (500.0 / 300.0) ** (np.arange(n) / max(n - 1, 1))
        # (the built structures are not equilibrated: the first, short time steps of a run)
        ctx.md_setup(temps, integrator=int(case.get("langevin", True)),
                     timestep=0.5e-15 if kind == "nb_md" else 0.25e-15, update_nlist=case["cadence"], update_sasa=5,
                     what=what, seed=seed)
        s.update(ctx=ctx, vel=maxwell_boltzmann(im.mass, temps, seed, im.natoms), p_out=ffi.host_array(pos.shape),
                 p_in=ffi.host_array(pos.shape))
        s["p_in"][:] = pos
    else:
        rng = np.random.default_rng(seed + 1)
        frames = np.stack([positions(case, seed + 1000 * (k + 1)) for k in range(case["frames"])])
        if case["system"] == "water":
            fs = FrameSet(im, frames, ffi.NB, nb_settings({**case, "inner": case["cutoff"] - 2.0}, im))
        else:
            fs = FrameSet(im, frames, ffi.GB, gb_settings(case, im))
        t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")
        s.update(fs=fs, frames=frames, weights=t(rng.uniform(-1.0, 1.0, case["frames"])),
                 params=[t(a) for a in fit_params(case, im, rng)])
    return s


def fit_params(case, im, rng):
    """Perturbed per-atom parameters: charges, LJ radii and well depths, GB radii and terms."""
    n = im.natom
    p = [im.charge + 0.02 * rng.standard_normal(n), im.radius * rng.uniform(0.95, 1.05, n),
         im.epsilon * rng.uniform(0.95, 1.05, n)]
    if case["system"] != "water":
        p += [im.gb_radius * rng.uniform(0.98, 1.02, n), im.gb_vj * rng.uniform(0.98, 1.02, n),
              im.gb_terms123 * rng.uniform(0.99, 1.01, n)]
    return p


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind in ("nb_forces", "gb_forces"):
        ws, ff = state["ws"], state["ff"]
        if case["rebuild"]:
            ctx = ff._prepare()
            ctx.set_positions(ws.cur.p)
            ctx.rebuild_list()
        ff.calcForces()
        e = ws.ene
        f = torch.from_numpy(ws.cur.f).to(torch.float32)
        if kind == "nb_forces":
            return {"ene": np.array([e.epot_vdw, e.epot_elec, e.InternalVirial]), "forces": f}
        out = {"ene": np.array([e.epot_vdw, e.epot_elec, e.epot_pol_cross, e.epot_pol_self], np.float32), "forces": f}
        if case["whole"]:
            out["more"] = np.array([e.epot_surf, e.epot_bond, e.epot_angle, e.epot_torsion], np.float32)
        return out
    if kind == "gb_energies":
        state["ff"].calcEnergies()
        e = state["ws"].ene
        return {"ene": np.array([e.epot_vdw, e.epot_elec, e.epot_pol_cross, e.epot_pol_self], np.float32)}
    if kind in ("nb_md", "gb_md"):
        ctx = state["ctx"]
        ctx.set_positions(state["p_in"])
        ctx.set_velocities(state["vel"])
        exchange = case.get("exchange", False)
        ctx.md_run(case["steps"], energy_on_last=exchange)
        out = {}
        if exchange:
            out["epot"] = np.array([e["epot"] for e in ctx.energies()], np.float32)
            out["accepted"], out["temps"] = ctx.remd_exchange(0)
        out["positions"] = torch.from_numpy(ctx.get_positions(state["p_out"])).to(torch.float32)
        out["velocities"] = torch.from_numpy(ctx.get_velocities()).to(torch.float32)
        out["kinetic"] = ctx.kinetic().astype(np.float32)
        return out
    leaves = [p.detach().requires_grad_(True) for p in state["params"]]
    E = state["fs"].energies(*leaves)
    (E * state["weights"]).sum().backward()
    return {"energies": E.detach().float(), "grads": [p.grad.float() for p in leaves]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Flops: the pair terms inside the cutoffs (58 per LJ + Coulomb pair; Born
    sums 19, GB + LJ + Coulomb 44, chain rule 31 per GB pair; gradients about as
    many again).  Bytes: positions in and results out, per atom and evaluation."""
    im = image(case)
    kind = case["kind"]
    if kind == "nb_md" or kind == "nb_forces" or case["system"] == "water":
        c = nb_settings(case, im)["Cutoff"]
        n = im.natom
        pairs = 0.5 * n * min(n - 1, n * 4.0 / 3.0 * math.pi * c ** 3 / float(np.prod(im.box[0])))
        per = 58.0
    else:
        cut = case.get("cutoff", 0.0)
        k = im.natoms.astype(np.float64)
        # (a compact peptide's density is near 0.06 atoms per A^3 in its own volume)
        pairs = float((0.5 * k * (np.minimum(k, 0.06 * 4.0 / 3.0 * math.pi * cut ** 3) if cut else k)).sum())
        per = 94.0 if kind != "gb_energies" else 63.0
    n = im.natom
    if kind in ("nb_md", "gb_md"):
        # per step: positions and velocities read and written, mass; ends: in, in, out
        return {"bytes": n * (case["steps"] * 104.0 + 72.0), "flops": case["steps"] * pairs * per}
    if kind == "fit":
        F, npar = case["frames"], 6 if case["system"] != "water" else 3
        return {"bytes": F * n * 24.0 + n * 16.0 * npar, "flops": F * pairs * 2.0 * per}
    return {"bytes": n * (48.0 if kind != "gb_energies" else 24.0), "flops": pairs * per}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind, im = case["kind"], image(case)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda a: torch.tensor(np.asarray(a, np.float64), device=dev)
    if kind in ("nb_md", "gb_md"):
        return None
    if kind == "nb_forces":
        if im.natom > 100000:
            return None
        pos = positions(case, seed)
        E, F = nb_exact(t(pos), [t(im.charge), t(im.radius), t(im.epsilon)], im.excl, im.box[0],
                        nb_settings(case, im), True)
        return {"ene": (E * TO_J).cpu().numpy(), "forces": (F * (TO_J / 1e-10)).cpu().numpy()}
    if kind in ("gb_forces", "gb_energies"):
        pos, p = positions(case, seed), gb_settings(case, im)
        tot, forces = torch.zeros(4, dtype=torch.float64, device=dev), []
        o = im.offsets
        for k in range(im.nsystems):
            a, b = int(o[k]), int(o[k + 1])
            m = (im.excl[:, 0] >= a) & (im.excl[:, 0] < b)
            ex = im.excl[m] - np.array([a, a, 0])
            par = [t(x[a:b]) for x in (im.charge, im.radius, im.epsilon, im.gb_radius, im.gb_vj, im.gb_terms123)]
            x = t(pos[a:b])
            if kind == "gb_energies":
                E, _ = gb_exact(x, par, ex, p, False, threshold=False)
                V, _ = nb_exact(x, par[:3], ex, np.zeros(3), dict(p, Dielectric=1.0, EnergySwitch=1, ForceSwitch=0),
                                False)
                tot += torch.stack([V[0], V[1], E[2], E[3]])
            else:
                E, F = gb_exact(x, par, ex, p, True)
                tot += E
                forces.append(F)
        out = {"ene": (tot * TO_J).cpu().numpy()}
        if kind == "gb_forces":
            whole = case["whole"]   # (surface and bonded forces are in the sum then)
            out["forces"] = None if whole else (torch.cat(forces) * (TO_J / 1e-10)).cpu().numpy()
            if whole:
                out["more"] = None
        return out
    rng = np.random.default_rng(seed + 1)
    w = rng.uniform(-1.0, 1.0, case["frames"])
    leaves = [t(a).requires_grad_(True) for a in fit_params(case, im, rng)]
    E = []
    for k in range(case["frames"]):
        x = t(positions(case, seed + 1000 * (k + 1)))
        if case["system"] == "water":
            e, _ = nb_exact(x, leaves, im.excl, im.box[0], nb_settings({**case, "inner": case["cutoff"] - 2.0}, im),
                            False)
            e = e[0] + e[1]
        else:
            e = gb_exact(x, leaves, im.excl, gb_settings(case, im), False)[0].sum()
        (e * (w[k] * TO_J)).backward()
        E.append(float(e.detach()) * TO_J)
    return {"energies": np.array(E), "grads": [p.grad.cpu().numpy() for p in leaves]}


def pair_chunks(x, excl, box, most=24_000_000):
    """Row chunks of all ordered pairs: rows, displacement to j (minimum image),
    r^2 (1 on the diagonal), and masks: other atom, not bonded closer than 1-4, 1-4."""
    n = len(x)
    L = torch.tensor(np.asarray(box, np.float64), device=x.device)
    e = np.asarray(excl, np.int64)
    e = torch.tensor(np.concatenate([e, e[:, [1, 0, 2]]]), device=x.device)
    rows = max(1, most // n)
    for a in range(0, n, rows):
        b = min(n, a + rows)
        d = x[None, :, :] - x[a:b, None, :]
        if float(L.min()) > 0:
            d = d - L * torch.round(d / L)
        r2 = (d * d).sum(-1)
        me = torch.arange(a, b, device=x.device)
        other = torch.ones((b - a, n), dtype=torch.bool, device=x.device)
        other[me - a, me] = False
        far, one4 = other.clone(), torch.zeros_like(other)
        s = e[(e[:, 0] >= a) & (e[:, 0] < b)]
        s3, s2 = s[s[:, 2] == 3], s[s[:, 2] <= 2]
        one4[s3[:, 0] - a, s3[:, 1]] = True
        far[s2[:, 0] - a, s2[:, 1]] = False
        yield a, b, d, torch.where(other, r2, torch.ones_like(r2)), other, far, one4


def scale14(one4, s, dtype):
    """s on the 1-4 pairs, 1 elsewhere."""
    return 1.0 + (s - 1.0) * one4.to(dtype)


def switch(r, inner, cut):
    """Energy switch (1 - u^2/w^2)^2 beyond `inner`, and its derivative."""
    u = torch.clamp(r - inner, min=0.0)
    w2 = 1.0 / (cut - inner) ** 2
    s = 1.0 - u * u * w2
    return s * s, -4.0 * w2 * u * s


def lj(r2, r, R, eps, inner, cut):
    B = (R * R / r2) ** 3
    E, dE = eps * (B * B - 2.0 * B), -12.0 * eps / r * (B * B - B)
    S, dS = switch(r, inner, cut)
    keep = (r < cut).to(r.dtype)
    return E * S * keep, (S * dE + E * dS) * keep


def nb_exact(x, par, excl, box, p, forces):
    """FF_NonBonded: (vdw, elec, virial) in kcal/mol and forces in kcal/mol/A."""
    q, R, se = par[0], par[1], par[2] * math.sqrt(NA / KCAL)
    C, I = p["Cutoff"], p["InnerCutoff"]
    ec = ECONV / p["Dielectric"]
    E, F = 0.0, []
    for a, b, d, r2, other, far, one4 in pair_chunks(x, excl, box):
        f = (far & (r2 <= C * C)).to(x.dtype)
        r = torch.sqrt(r2)
        sv = scale14(one4, p["Vdw14Scaling"], x.dtype) * f
        qq = q[a:b, None] * q[None, :] * ec * scale14(one4, p["Elec14Scaling"], x.dtype) * f
        ev, dv = lj(r2, r, R[a:b, None] + R[None, :], se[a:b, None] * se[None, :] * sv, p["VdwInnerCutoff"],
                    p["VdwCutoff"])
        if p["ForceSwitch"]:
            A = 1.0 / (C * C - I * I) ** 3
            sB, sC, sD, sE = -(C ** 6 - 3.0 * C ** 4 * I ** 2), 6.0 * C * C * I * I, -(C * C + I * I), 0.4
            V = lambda y: A * (sB / y + sC * y + sD * y ** 3 + sE * y ** 5)
            out = r > I
            ee = torch.where(out, -qq * (V(r) - V(C)), qq * (1.0 / r - (1.0 / I + V(I) - V(C))))
            de = torch.where(out, -qq * A / r2 * (C * C - r2) ** 2 * (C * C - 3.0 * I * I + 2.0 * r2), -qq / r2)
        else:
            ee, de = qq / r, -qq / r2
            if p["EnergySwitch"]:
                S, dS = switch(r, I, C)
                ee, de = ee * S, S * de + ee * dS
        E = E + 0.5 * torch.stack([ev.sum(), ee.sum(), (r * (dv + de)).sum()])
        if forces:
            F.append((((dv + de) / r)[..., None] * d).sum(1))
    return E, torch.cat(F) if forces else None


def contact(r2, rs, P5):
    """CCF of the Still pairwise Born radii, and -d ln-type factor dCCF used by the force."""
    y = r2 / (rs * rs) * P5
    on = y <= 1.0
    y = torch.where(on, y, torch.ones_like(y))
    h = 0.5 - 0.5 * torch.cos(math.pi * y)
    return h * h, 2.0 * h * torch.sin(math.pi * y) * math.pi * y * on.to(y.dtype)


def gb_exact(x, par, excl, p, forces, threshold=True):
    """Still GB with its vacuum LJ + Coulomb: (vdw, elec, pol cross, pol self) in
    kcal/mol and forces in kcal/mol/A.  threshold False: the GB term of every pair."""
    q, R, se, gR, gV, gT = par[0], par[1], par[2] * math.sqrt(NA / KCAL), par[3], par[4], par[5]
    box = np.zeros(3)
    still2 = min(p["GbsaStillCutoff"], p["Cutoff"] + 2.0) ** 2
    cut2 = p["Cutoff"] ** 2
    sums = []
    for a, b, d, r2, other, far, one4 in pair_chunks(x, excl, box):
        on = (far & (r2 <= still2)).to(x.dtype)
        ccf, _ = contact(r2, gR[a:b, None] + gR[None, :], p["P5"])
        sums.append((on * p["P4"] * gV[None, :] * ccf / (r2 * r2)).sum(1))
    born = -0.5 * ECONV / (gT + torch.cat(sums)) + p["BornRadiusOffset"]
    pre = -0.5 * ECONV * (1.0 / p["DielectricSolute"] - 1.0 / p["DielectricSolvent"])
    E, F, da = 0.0, [], []
    for a, b, d, r2, other, far, one4 in pair_chunks(x, excl, box):
        ins = other & (r2 <= cut2)
        f = ins.to(x.dtype)
        r = torch.sqrt(r2)
        aa = born[a:b, None] * born[None, :]
        u = -0.25 * r2 / aa
        on = (u > p["ExpApproxThreshold"]) if threshold else torch.ones_like(ins)
        qq = q[a:b, None] * q[None, :]
        tg = torch.exp(u)
        fgb = 1.0 / torch.sqrt(r2 + tg * aa)
        S, dS = switch(r, p["InnerCutoff"], p["Cutoff"])
        ep = pre * qq * fgb * f * on.to(x.dtype)
        vac = (far & ins).to(x.dtype)
        near = on.to(x.dtype)
        ec = near * (ECONV / p["DielectricSolute"]) + (1.0 - near) * (ECONV / p["DielectricSolvent"])
        el = ec * qq / r * scale14(one4, p["Elec14Scaling"], x.dtype) * vac
        ev, dv = lj(r2, r, R[a:b, None] + R[None, :],
                    se[a:b, None] * se[None, :] * scale14(one4, p["Vdw14Scaling"], x.dtype) * vac,
                    p["VdwInnerCutoff"], p["VdwCutoff"])
        E = E + torch.stack([0.5 * ev.sum(), 0.5 * (el * S).sum(), (ep * S).sum()])
        if forces:
            l = fgb * fgb
            g = 2.0 * (S * -ep * (r - 0.25 * r * tg) * l + dS * ep) + S * -el / r + el * dS + dv
            F.append(((g / r)[..., None] * d).sum(1))
            da.append((-ep * tg * (1.0 - u) * l * S * born[None, :]).sum(1))
    own = pre * q * q / born
    E = torch.cat([E, own.sum()[None]])
    if not forces:
        return E, None
    F = torch.cat(F)
    c = born * born / 166.0 * (torch.cat(da) - own / born) * p["P4"]
    for a, b, d, r2, other, far, one4 in pair_chunks(x, excl, box):
        on = (far & (r2 <= still2)).to(x.dtype)
        ccf, dccf = contact(r2, gR[a:b, None] + gR[None, :], p["P5"])
        w = on * (c[a:b, None] * gV[None, :] + c[None, :] * gV[a:b, None]) * (4.0 * ccf - dccf) / r2 ** 3
        F[a:b] -= (w[..., None] * d).sum(1)
    return E, F
