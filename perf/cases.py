"""Performance cases of the batched implicit-solvent path, through the calls a program makes.

Every case keeps a Synthesis (the batch's topologies, resident on the GPU) and page-locked host
buffers, as a scoring or minimization loop does, and one pass hands it new coordinates and takes
the results back.  Molecules come from the seeded generator of the repository's workloads; a
batch holds several replicas of each topology with their own coordinates (conformers of a
compound), placed by Gaussian noise about the built geometry.

The cases and what they stand for:

  single_64        one drug-sized molecule, force + energy: a client that evaluates one geometry
                   at a time, where launches and copies are the cost
  batch_384_salt   a middling batch under the pairwise-descreening (HCT) model with salt: the
                   model and screening options, and fewer work units than fill the GPU twice
  batch_1024       the batched single point of 16-256 atoms, the benchmark's workload
  rescore_poses    MM-GBSA rescoring, energies only: a receptor, poses of a ligand and their
                   complexes (molecules above 256 atoms beside small ones)
  surface_poses    the surface-area term of the same systems
  minimize_one     one small molecule through the default minimizer, a 60-cycle relaxation
  minimize_4096    the minimization workload: 24-96 atoms, perturbed by 0.3 A
  minimize_served  a served batch: lognormal sizes, the on-chip minimizer with an RMS target
  chain_1          one protein-sized chain, force + energy
  chains_32        the large-system workload: chains of 2,000-5,000 atoms
  fp64_batch       the double-precision mode on a batch of small molecules
  fp64_chains      the double-precision mode on chains
"""
from __future__ import annotations

import math

import numpy as np
import torch

import stormm_b200 as sb
from stormm_b200 import mmgbsa, synthetic

SPHERE_POINTS = 272          # STORMM's MM-GBSA default
PROBE = 1.4
SD_CYCLES = 30               # steepest descent before conjugate gradient
SCEE, SCNB = 1.2, 2.0        # 1-4 scaling of the generated molecules


def _evaluate(name, **kw):
    case = {"name": name, "kind": "evaluate", "chain": False, "igb": 5, "salt": 0.0,
            "precision": 0}
    case.update(kw)
    return case


def listed():
    return [
        _evaluate("single_64", systems=1, topologies=1, min_atoms=64, max_atoms=64),
        _evaluate("batch_384_salt", systems=384, topologies=48, min_atoms=20, max_atoms=200,
                  igb=1, salt=0.1),
        _evaluate("batch_1024", systems=1024, topologies=128, min_atoms=16, max_atoms=256),
        {"name": "rescore_poses", "kind": "rescore", "receptor": 500, "ligand": 40, "poses": 63},
        {"name": "surface_poses", "kind": "surface", "receptor": 500, "ligand": 40, "poses": 31},
        {"name": "minimize_one", "kind": "minimize", "systems": 1, "topologies": 1,
         "min_atoms": 48, "max_atoms": 48, "served": False, "cycles": 60},
        {"name": "minimize_4096", "kind": "minimize", "systems": 4096, "topologies": 256,
         "min_atoms": 24, "max_atoms": 96, "served": False, "cycles": 60},
        {"name": "minimize_served", "kind": "minimize", "systems": 128, "topologies": 128,
         "min_atoms": 12, "max_atoms": 512, "served": True, "cycles": 60},
        _evaluate("chain_1", systems=1, topologies=1, min_atoms=2500, max_atoms=2500, chain=True),
        _evaluate("chains_32", systems=32, topologies=8, min_atoms=2000, max_atoms=5000,
                  chain=True),
        _evaluate("fp64_batch", systems=128, topologies=32, min_atoms=16, max_atoms=256,
                  precision=1),
        _evaluate("fp64_chains", systems=8, topologies=4, min_atoms=2000, max_atoms=5000,
                  chain=True, precision=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["small", "small", "small", "chain", "fp64", "rescore", "surface",
                       "minimize", "minimize", "served"])
    igb, salt = rng.choice([5, 5, 5, 2, 1]), rng.choice([0.0, 0.0, round(rng.uniform(0.02, 0.3), 3)])
    if kind in ("small", "fp64"):
        systems = _log_int(rng, 1, 1024 if kind == "small" else 128)
        lo = rng.randint(12, 80)
        case = _evaluate("", systems=systems, topologies=min(systems, rng.randint(24, 96)),
                         min_atoms=lo, max_atoms=rng.randint(lo, 256), igb=igb, salt=salt,
                         precision=1 if kind == "fp64" else 0)
    elif kind == "chain":
        systems = _log_int(rng, 1, 24)
        lo = rng.randint(2049, 3500)
        precision = rng.choice([0, 0, 1])
        case = _evaluate("", systems=systems if precision == 0 else min(systems, 8),
                         topologies=min(systems, 4), min_atoms=lo,
                         max_atoms=rng.randint(lo, 5000), chain=True, igb=igb, salt=salt,
                         precision=precision)
    elif kind in ("rescore", "surface"):
        case = {"kind": kind, "receptor": rng.randint(150, 900), "ligand": rng.randint(12, 90),
                "poses": _log_int(rng, 1, 63 if kind == "rescore" else 31)}
    elif kind == "minimize":
        systems = _log_int(rng, 1, 2048)
        lo = rng.randint(12, 60)
        case = {"kind": "minimize", "systems": systems,
                "topologies": min(systems, rng.randint(32, 128)), "min_atoms": lo,
                "max_atoms": rng.randint(lo, 128), "served": False,
                "cycles": rng.randint(56, 72)}
    else:
        systems = _log_int(rng, 1, 128)
        case = {"kind": "minimize", "systems": systems, "topologies": systems, "min_atoms": 12,
                "max_atoms": rng.randint(64, 384), "served": True, "cycles": 60}
    case.pop("name", None)
    return case


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _sphere(n):
    """n nearly even unit vectors (golden-angle spiral)."""
    k = np.arange(n) + 0.5
    z = 1.0 - 2.0 * k / n
    phi = k * math.pi * (3.0 - math.sqrt(5.0))
    r = np.sqrt(1.0 - z * z)
    return np.stack([r * np.cos(phi), r * np.sin(phi), z], axis=1)


def _poses(receptor, ligand, count, rng):
    """Ligand placements at the receptor's surface, no atom of the two closer than 2.8 A."""
    rec = receptor.coords - receptor.coords.mean(axis=0)
    lig = ligand.coords - ligand.coords.mean(axis=0)
    reach = np.linalg.norm(rec, axis=1).max() + np.linalg.norm(lig, axis=1).max() + 3.0
    out = []
    for _ in range(count):
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        body = lig @ q
        u = rng.normal(size=3)
        u /= np.linalg.norm(u)
        dist = reach
        while dist > 0.0:
            d2 = ((rec[:, None, :] - (body + (dist - 0.7) * u)[None, :, :]) ** 2).sum(axis=2)
            if d2.min() < 2.8 ** 2:
                break
            dist -= 0.7
        out.append(receptor.coords.mean(axis=0) + body + dist * u)
    return out


def _systems(case, seed):
    """(topologies, topology index of every system, coordinates of every system)."""
    rng = np.random.default_rng([int(seed), 20261204])
    if case["kind"] in ("rescore", "surface"):
        rec = synthetic.make_molecule(int(rng.integers(1 << 40)), case["receptor"], noise=0.1)
        lig = synthetic.make_molecule(int(rng.integers(1 << 40)), case["ligand"], noise=0.1)
        poses = _poses(rec, lig, case["poses"], rng)
        index = [0] + [1] * len(poses) + [2] * len(poses)
        xyz = [rec.coords] + poses + [np.concatenate([rec.coords, p]) for p in poses]
        return [rec, lig, mmgbsa.combine(rec, lig)], np.array(index, dtype=np.int32), xyz
    count = case["topologies"]
    # the sizes belong to the case, everything else to the seed
    size_rng = np.random.default_rng([case["systems"], count, case["min_atoms"],
                                      case["max_atoms"]])
    if case.get("served"):
        # request sizes of the served workload: lognormal about 48 atoms
        sizes = np.clip(np.rint(48.0 * np.exp(size_rng.normal(0.0, 0.6, size=count))),
                        case["min_atoms"], case["max_atoms"]).astype(int)
    else:
        sizes = size_rng.integers(case["min_atoms"], case["max_atoms"] + 1, size=count)
    make = synthetic.make_chain if case.get("chain") else synthetic.make_molecule
    mols = [make(int(rng.integers(1 << 40)), int(n), noise=0.0) for n in sizes]
    index = np.arange(case["systems"], dtype=np.int32) % count
    noise = 0.3 if case["kind"] == "minimize" else (0.05 if case.get("chain") else 0.1)
    xyz = [mols[t].coords + rng.normal(0.0, noise, size=mols[t].coords.shape) for t in index]
    return mols, index, xyz


def _pinned(values):
    a = torch.empty(int(values), dtype=torch.float64, pin_memory=True).numpy()
    a[:] = 0.0
    return a


def prepare(case, seed):
    mols, index, xyz = _systems(case, seed)
    options = sb.default_options(igb=case.get("igb", 5), saltcon=case.get("salt", 0.0),
                                 precision=case.get("precision", 0))
    syn = sb.Synthesis(mols, topology_index=index, options=options)
    coords = _pinned(3 * syn.total_atoms)
    coords[:] = np.concatenate([x.reshape(-1) for x in xyz])
    state = {"case": case, "syn": syn, "xyz": coords,
             "energies": _pinned(syn.nsys * sb.NRG_STRIDE)}
    if case["kind"] == "evaluate":
        state["forces"] = _pinned(3 * syn.total_atoms)
    elif case["kind"] == "minimize":
        state["final"] = _pinned(3 * syn.total_atoms)
    elif case["kind"] == "surface":
        state["points"] = _sphere(SPHERE_POINTS)
    return state


def run(state):
    case, syn = state["case"], state["syn"]
    syn.set_coordinates(state["xyz"])
    if case["kind"] == "evaluate":
        syn.initialize(sb.INIT_FORCES | sb.INIT_ENERGIES)
        syn.evaluate()
        return {"forces": syn.forces(out=state["forces"]),
                "energies": syn.energies(out=state["energies"])}
    if case["kind"] == "rescore":
        syn.initialize(sb.INIT_ENERGIES)
        syn.evaluate(force=False, energy=True)
        return {"energies": syn.energies(out=state["energies"])}
    if case["kind"] == "surface":
        return {"area": syn.surface_area(state["points"], probe_radius=PROBE)}
    if case["served"]:
        syn.minimize(total_cycles=case["cycles"], sd_cycles=SD_CYCLES, kernel=sb.MIN_PERSISTENT,
                     convergence_rms=0.01)
    else:
        syn.minimize(total_cycles=case["cycles"], sd_cycles=SD_CYCLES)
    return {"coordinates": syn.coordinates(out=state["final"]),
            "energy": syn.energies(out=state["energies"]).sum(axis=1)}


# ------------------------------------------------------------------------------------------------
# work and tolerances
# ------------------------------------------------------------------------------------------------
def _mean_pairs(case):
    """Atoms and pairs of the case's systems (expected values of the size distribution)."""
    if case["kind"] in ("rescore", "surface"):
        r, l, p = case["receptor"], case["ligand"], case["poses"]
        sizes = [(r, 1), (l, p), (r + l, p)]
        return (sum(n * c for n, c in sizes), sum(n * (n - 1) / 2 * c for n, c in sizes),
                1 + 2 * p)
    lo, hi, n = case["min_atoms"], case["max_atoms"], case["systems"]
    if case.get("served"):
        mean, sq = 48.0 * math.exp(0.18), 48.0 ** 2 * math.exp(0.72)
    else:
        mean = 0.5 * (lo + hi)
        sq = mean * mean + ((hi - lo + 1) ** 2 - 1) / 12.0
    return n * mean, n * 0.5 * (sq - mean), n


def work(case):
    """Coordinates in and results out once, per-atom and valence parameters once; 190 flops a
    pair for forces and energies (descreening 48, pair terms 79, radius chain rule 63), 93 for
    energies alone."""
    atoms, pairs, systems = _mean_pairs(case)
    parameters = 32 * atoms + 16 * atoms + 48 * 1.8 * atoms + 112 * 2.8 * atoms
    moved = 24 * atoms + 128 * systems + parameters
    if case["kind"] == "surface":
        # every sphere point placed and tested once (12 flops and a distance test of 9)
        return {"bytes": 24 * atoms + 8 * atoms + 8 * systems,
                "flops": 21.0 * atoms * SPHERE_POINTS}
    if case["kind"] == "rescore":
        return {"bytes": moved, "flops": 93.0 * pairs}
    if case["kind"] == "minimize":
        # per cycle a force and energy evaluation and three energies
        return {"bytes": moved + 24 * atoms,
                "flops": case["cycles"] * (190.0 + 3 * 93.0) * pairs}
    return {"bytes": moved + 24 * atoms, "flops": 190.0 * pairs}


def tolerance(case):
    if case["kind"] == "surface":
        # each point survives or not by the same test; only the order of the sum is free
        return {"rel": 1e-12, "max": 1e-11}
    if case["kind"] == "minimize":
        # line searches amplify the rounding of an FP32 evaluation: a cycle whose trial energies
        # differ in their last bits may take another step.  Measured over 60 cycles against the
        # FP64 mode: coordinates 2.3e-3 (largest 0.19), energies 3.8e-3 (0.06)
        return {"rel": 1e-2, "max": 0.6}
    if case.get("precision") == 1:
        # forces on the 2^-23 grid, energies on the 2^-26 grid
        return {"rel": 4e-8, "max": 2e-6}
    return {"rel": 2e-6, "max": 8e-5}


# ------------------------------------------------------------------------------------------------
# the same results in plain FP64 torch
# ------------------------------------------------------------------------------------------------
GB_MODELS = {2: (0.8, 0.0, 2.909125), 5: (1.0, 0.8, 4.85)}
TAYLOR = (1.0 / 3.0, 2.0 / 5.0, 3.0 / 7.0, 4.0 / 9.0, 5.0 / 11.0)


def _descreening(r, rho, sj):
    """Pairwise descreening of radii rho by neighbours of screened radius sj at distance r."""
    far = r > 4.0 * sj
    apart = ~far & (r > rho + sj)
    part = ~far & ~apart & (r > (rho - sj).abs())
    inside = ~far & ~apart & ~part & (rho < sj)
    one = torch.ones_like(r)
    rf = torch.where(far, r, 8.0 * sj + one)
    t = (sj / rf) ** 2
    series = TAYLOR[4]
    for c in TAYLOR[3::-1]:
        series = c + t * series
    out = torch.where(far, sj * t / rf ** 2 * series, torch.zeros_like(r))
    ra = torch.where(apart, r, 2.0 * sj + one)
    va = 0.5 * (sj / (ra ** 2 - sj ** 2) + 0.5 / ra * torch.log((ra - sj) / (ra + sj)))
    out = torch.where(apart, va, out)
    rp = torch.where(part, r, one)
    theta = 0.5 / rho / rp * (rp ** 2 + rho ** 2 - sj ** 2)
    u = 1.0 / (rp + sj)
    vp = 0.25 * ((2.0 - theta) / rho - u + torch.log(rho * u) / rp)
    out = torch.where(part, vp, out)
    if bool(inside.any()):
        ri = torch.where(inside, r, 0.5 * sj)
        vi = 0.5 * (sj / (ri ** 2 - sj ** 2) + 2.0 / rho +
                    0.5 / ri * torch.log((sj - ri) / (sj + ri)))
        out = torch.where(inside, vi, out)
    return out


def _exact_topology(mol, xyz, igb, salt, dev):
    """Energies (replicas, 16) and forces (replicas, atoms, 3) of replicas of one topology."""
    def d(a):
        return torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev)

    def ix(a):
        return torch.as_tensor(np.asarray(a, dtype=np.int64), device=dev)

    n = mol.natom
    x = torch.tensor(xyz, dtype=torch.float64, device=dev, requires_grad=True)
    q = d(mol.charge) * math.sqrt(332.05221729)
    e = {}
    b = ix(mol.bonds)
    if len(b):
        r = (x[:, b[:, 1]] - x[:, b[:, 0]]).norm(dim=2)
        e[0] = (d(mol.bond_k) * (r - d(mol.bond_r0)) ** 2).sum(dim=1)
    a = ix(mol.angles)
    if len(a):
        ba, bc = x[:, a[:, 0]] - x[:, a[:, 1]], x[:, a[:, 2]] - x[:, a[:, 1]]
        th = torch.atan2(torch.cross(ba, bc, dim=2).norm(dim=2), (ba * bc).sum(dim=2))
        e[1] = (d(mol.angl_k) * (th - d(mol.angl_theta0)) ** 2).sum(dim=1)
    w = ix(mol.dihedrals)
    if len(w):
        ab, bc, cd = (x[:, w[:, k + 1]] - x[:, w[:, k]] for k in range(3))
        n1, n2 = torch.cross(ab, bc, dim=2), torch.cross(bc, cd, dim=2)
        ph = torch.atan2(bc.norm(dim=2) * (ab * n2).sum(dim=2), (n1 * n2).sum(dim=2))
        e[2] = (d(mol.dihe_amp) * (1.0 + torch.cos(d(mol.dihe_freq) * ph - d(mol.dihe_phase)))
                ).sum(dim=1)
        s = w[ix(np.flatnonzero(mol.dihe_has14))]
        ty = ix(mol.lj_idx)
        lja, ljb = d(mol.lja), d(mol.ljb)
        r2 = ((x[:, s[:, 3]] - x[:, s[:, 0]]) ** 2).sum(dim=2)
        e[10] = (q[s[:, 0]] * q[s[:, 3]] / SCEE / r2.sqrt()).sum(dim=1)
        ta, tb = ty[s[:, 0]], ty[s[:, 3]]
        e[8] = ((lja[ta, tb] / r2 ** 6 - ljb[ta, tb] / r2 ** 3) / SCNB).sum(dim=1)
    # all pairs as a full matrix (each pair twice), the diagonal set aside
    eye = torch.eye(n, dtype=torch.bool, device=dev)
    dx = x[:, :, None, :] - x[:, None, :, :]
    r2 = (dx ** 2).sum(dim=3)
    del dx
    r2 = torch.where(eye, torch.full_like(r2, 25.0), r2)
    r = r2.sqrt()
    excl = eye.clone()
    rows = [i for i in range(n) for _ in set(mol.excl12[i]) | set(mol.excl13[i]) | set(mol.excl14[i])]
    cols = [j for i in range(n) for j in set(mol.excl12[i]) | set(mol.excl13[i]) | set(mol.excl14[i])]
    if rows:
        excl[ix(rows), ix(cols)] = True
    ty = ix(mol.lj_idx)
    keep = torch.where(excl, 0.0, 0.5).to(torch.float64)
    qq = q[:, None] * q[None, :]
    e[9] = (keep * qq / r).sum(dim=(1, 2))
    i6 = 1.0 / r2 ** 3
    e[7] = (keep * (d(mol.lja)[ty][:, ty] * i6 * i6 - d(mol.ljb)[ty][:, ty] * i6)).sum(dim=(1, 2))
    rho = d(mol.pb_radii) - 0.09
    sj = d(mol.gb_screen) * rho
    h = _descreening(r, rho[:, None].expand(n, n), sj[None, :].expand(n, n))
    psi = -torch.where(eye, torch.zeros_like(h), h).sum(dim=2)
    del h
    if igb == 1:
        born = 1.0 / (1.0 / rho + psi)
        born = torch.where(born < 0.0, torch.full_like(born, 30.0), born)
    else:
        al, be, ga = GB_MODELS[igb]
        f = -psi * rho
        born = 1.0 / (1.0 / rho - torch.tanh((al - be * f + ga * f * f) * f) / d(mol.pb_radii))
    kappa = math.sqrt(0.10806 * salt) * 0.73 if salt > 1e-8 else 0.0
    bb = born[:, :, None] * born[:, None, :]
    fgb = (r2 + bb * torch.exp(-r2 / (4.0 * bb))).sqrt()
    pair = -qq * (1.0 - torch.exp(-kappa * fgb) / 80.0) / fgb
    e[11] = 0.5 * torch.where(eye, torch.zeros_like(pair), pair).sum(dim=(1, 2))
    e[11] = e[11] - (0.5 * q * q * (1.0 - torch.exp(-kappa * born) / 80.0) / born).sum(dim=1)
    total = sum(v.sum() for v in e.values())
    forces = -torch.autograd.grad(total, x)[0]
    out = torch.zeros((len(xyz), 16), dtype=torch.float64)
    for k, v in e.items():
        out[:, k] = v.detach().cpu()
    return out.numpy(), forces.cpu().numpy()


def _exact_surface(mol, xyz, points, dev):
    """Surface area of one system: the points of each atom's probe sphere that lie inside no
    other atom's, an atom tested against those of its own and the lower neighbour cells."""
    ty = np.asarray(mol.lj_idx)
    a, b = np.asarray(mol.lja)[0, ty], np.asarray(mol.ljb)[0, ty]
    rad = torch.as_tensor(np.where(b > 1e-6, 0.5 * np.sqrt(np.cbrt(a / np.where(b > 0, b, 1.0))),
                                   0.0), device=dev)
    # coordinates as the fixed-point grid holds them
    x = torch.as_tensor(np.rint(xyz * 2.0 ** 32) * 2.0 ** -32, device=dev)
    n = len(x)
    lo, hi = x.min(dim=0).values, x.max(dim=0).values
    count = torch.ceil((hi - lo) / (2.0 * (rad.max() + PROBE)))
    if bool((count == 0).any()):
        return 0.0
    cell = torch.floor((x - lo) / ((hi - lo) / count)).clamp(min=0)
    cell = torch.minimum(cell, count - 1)
    pts = torch.as_tensor(points, device=dev)
    reach = rad + PROBE
    alive = 0.0
    for m0 in range(0, n, 32):
        m1 = min(n, m0 + 32)
        p = x[m0:m1, None, :] + pts[None, :, :] * reach[m0:m1, None, None]
        d = cell[m0:m1, None, :] - cell[None, :, :]
        near = ((d >= 0) & (d <= 1)).all(dim=2)
        near[torch.arange(m1 - m0, device=dev), torch.arange(m0, m1, device=dev)] = False
        d = p[:, :, None, :] - x[None, None, :, :]
        d2 = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]
        hit = ((d2 < (reach * reach)[None, None, :]) & near[:, None, :]).any(dim=2)
        alive += float(((~hit).sum(dim=1) * reach[m0:m1] ** 2).sum())
    return alive * 4.0 * math.pi / len(points)


def exact(case, seed):
    if case["kind"] == "minimize":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if dev == "cpu" and _mean_pairs(case)[1] > 3e7:
        return None
    mols, index, xyz = _systems(case, seed)
    if case["kind"] == "surface":
        pts = _sphere(SPHERE_POINTS)
        return {"area": np.array([_exact_surface(mols[t], x, pts, dev)
                                  for t, x in zip(index, xyz)])}
    energies = np.zeros((len(index), 16))
    forces = [None] * len(index)
    for t, mol in enumerate(mols):
        mine = np.flatnonzero(index == t)
        # replicas of a topology at once, up to about 20 million matrix elements
        step = max(1, int(2e7 / mol.natom ** 2))
        for k in range(0, len(mine), step):
            part = mine[k:k + step]
            e, f = _exact_topology(mol, np.stack([xyz[s] for s in part]), case.get("igb", 5),
                                   case.get("salt", 0.0), dev)
            energies[part] = e
            for s, one in zip(part, f):
                forces[s] = one
    if case["kind"] == "rescore":
        return {"energies": energies}
    return {"forces": np.concatenate(forces), "energies": energies}
