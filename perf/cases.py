"""The work a user of this package has it do, as cases to be timed and checked.

Every case goes through the public Python classes: the fused Lennard-Jones
stepper, the drop-in actions (one by one, as the reference's drivers call
them), the AdResS stepper, a batch of AdResS replicas and the trajectory
gradient.  Sizes come from the benchmark's and the tests' configurations; the
ranges in draw() span what those configurations reach.  exact() is an
independent FP64 restatement in plain torch.
"""
import ctypes
import math

import numpy as np
import torch

import mrmd_gb300 as M

RC, SKIN, DT = 2.5, 0.3, 0.005
LIST = RC + SKIN
T_LJ = 0.728
CAP_ADRESS = 0.7842  # force cap 1000
HYBRID = {"adress": 10.0, "actions": 10.0, "batch": 8.0, "diff": 10.0}
TF_BIN = 1.2
NOISE_SEED = 1234


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # the smallest ordinary run: 10^3 fcc cells in plain FP64, where launches and rebuilds count
        _nve("nve_4k_fp64", 10, 10, 10, 0, "fp64", 50, False),
        # an energy-conservation run with every step's observables recorded
        _nve("nve_32k_mixed_observed", 20, 20, 20, 0, "mixed", 50, True),
        # a production FP64 fluid whose size is no multiple of anything
        _nve("nve_256k_fp64", 40, 40, 40, 1003, "fp64", 20, False),
        # the headline 4,000,000-atom fluid in the mixed form
        _nve("nve_4m_mixed", 100, 100, 100, 0, "mixed", 20, False),
        # the reference's examples/02 time loop, written with the drop-in actions
        {"name": "loop_32k_fp64", "kind": "loop", "cx": 20, "cy": 20, "cz": 20, "drop": 0, "rho": 0.8442,
         "precision": "fp64", "steps": 10},
        # forces of one configuration through the drop-in actions: ghosts, list, mixed pair force, fold-back
        {"name": "forces_256k_mixed", "kind": "loop", "cx": 40, "cy": 40, "cz": 40, "drop": 501, "rho": 0.8442,
         "precision": "mixed", "steps": 0},
        # the 34,560-molecule AdResS box in both forms
        _adress("adress_34k_fp64", 60, 12, 12, 30.0, "fp64", 50),
        _adress("adress_34k_mixed", 60, 12, 12, 30.0, "mixed", 50),
        # a million molecules of the same physics
        _adress("adress_1m_mixed", 182, 38, 38, 91.0, "mixed", 50),
        # one AdResS force evaluation with the drop-in actions (examples/04's sequence)
        {"name": "actions_34k_fp64", "kind": "actions", "cx": 60, "cy": 12, "cz": 12, "at": 30.0, "sites": 1,
         "precision": "fp64"},
        # 64 independent replicas of 1,000 to 50,000 molecules
        {"name": "batch_64_mixed", "kind": "batch", "replicas": 64, "nmin": 1000, "nmax": 50000, "set_seed": 4,
         "precision": "mixed", "layout": 1, "lanes": 1, "steps": 50},
        # one gradient of a trajectory loss with respect to the thermodynamic force and the LJ parameters
        {"name": "gradient_65k_mixed", "kind": "diff", "cx": 128, "cy": 8, "cz": 16, "at": 40.0, "steps": 50,
         "window": 20, "checkpoint": 25, "precision": "mixed"},
    ]


def _nve(name, cx, cy, cz, drop, precision, steps, observe):
    return {"name": name, "kind": "nve", "cx": cx, "cy": cy, "cz": cz, "drop": drop, "rho": 0.8442,
            "precision": precision, "steps": steps, "observe": observe}


def _adress(name, cx, cy, cz, at, precision, steps):
    return {"name": name, "kind": "adress", "cx": cx, "cy": cy, "cz": cz, "at": at, "precision": precision,
            "steps": steps}


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["nve", "nve", "nve", "loop", "loop", "adress", "adress", "actions", "batch", "diff"])
    precision = rng.choice(["fp64", "mixed"])
    if kind in ("nve", "loop"):
        # 4,000 to about 1,400,000 atoms (FP64: 400,000) in boxes of unequal sides
        top = 100000 if precision == "fp64" or kind == "loop" else 350000
        edge = _log(rng, 1000, top) ** (1.0 / 3.0)
        c = [max(8, int(round(edge * rng.uniform(0.8, 1.25)))) for _ in range(3)]
        steps = rng.choice([10, 20, 30, 50]) if kind == "nve" else rng.choice([0, 0, 10, 20])
        d = {"kind": kind, "cx": c[0], "cy": c[1], "cz": c[2], "drop": rng.randint(0, 4 * c[0] * c[1] * c[2] // 50),
             "rho": round(rng.uniform(0.7, 0.9), 4), "precision": precision, "steps": steps}
        if kind == "nve":
            d["observe"] = rng.random() < 0.3
        return d
    if kind in ("adress", "actions"):
        # 5,000 to about 400,000 molecules; the slab and its hybrid edges inside the box
        cross = rng.randint(6, 20 if kind == "adress" else 14)
        cx = int(_log(rng, 36, 250))
        d = {"kind": kind, "cx": cx, "cy": cross, "cz": rng.randint(6, cross + 2),
             "at": round(rng.uniform(4.0, 2.0 * cx - 30.0), 2), "precision": precision}
        d.update({"steps": rng.choice([10, 50, 100])} if kind == "adress" else {"sites": rng.randint(1, 3)})
        return d
    if kind == "batch":
        d = {"kind": "batch", "replicas": rng.randint(2, 60), "nmin": 1000, "nmax": rng.choice([5000, 20000, 50000]),
             "set_seed": rng.randint(1, 10 ** 6), "precision": precision, "layout": 0, "lanes": rng.choice([1, 2]),
             "steps": 50}
        if precision == "mixed":
            d["layout"] = rng.choice([0, 1, 1])
        return d
    cx = rng.randint(40, 128)
    return {"kind": "diff", "cx": cx, "cy": rng.randint(5, 10), "cz": rng.randint(5, 14),
            "at": round(rng.uniform(8.0, 2.0 * cx - 40.0), 2), "steps": rng.choice([20, 40]), "window": 10,
            "checkpoint": rng.choice([10, 20]), "precision": precision}


# ----------------------------------------------------------------- inputs --
def _fcc(cx, cy, cz, edge):
    base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    g = np.stack(np.meshgrid(np.arange(cx), np.arange(cy), np.arange(cz), indexing="ij"), -1).reshape(-1, 3)
    return ((g[:, None, :] + base[None, :, :]).reshape(-1, 3) + 0.25) * edge, np.array([cx, cy, cz]) * edge


def _velocities(rng, n, T):
    v = rng.standard_normal((n, 3)) * math.sqrt(T)
    return v - v.mean(0)


def _lj_inputs(case, seed):
    """A dense fluid: lattice sites with thermal displacements, some of them
    vacant, in lattice order."""
    rng = np.random.default_rng([seed, 11])
    pos, L = _fcc(case["cx"], case["cy"], case["cz"], (4.0 / case["rho"]) ** (1.0 / 3.0))
    if case["drop"]:
        pos = np.delete(pos, rng.choice(len(pos), case["drop"], replace=False), axis=0)
    pos += rng.standard_normal(pos.shape) * 0.05
    return np.mod(pos, L), _velocities(rng, len(pos), T_LJ), L


def _gas_inputs(case, seed):
    """Single-site molecules at density 0.5 (fcc edge 2 with displacements)."""
    rng = np.random.default_rng([seed, 12])
    pos, L = _fcc(case["cx"], case["cy"], case["cz"], 2.0)
    pos = np.mod(pos + rng.standard_normal(pos.shape) * 0.1, L)
    if case["kind"] == "adress":  # a seeded placement has no order in space
        pos = pos[rng.permutation(len(pos))]
    return pos, _velocities(rng, len(pos), 1.0), L


def _table(seed, bins):
    """A thermodynamic force as a fit leaves it: smooth, below 1 epsilon/sigma."""
    ph = np.random.default_rng([seed, 13]).uniform(0, 2 * math.pi, 3)
    x = (np.arange(bins) + 0.5) / bins
    return 0.3 * sum(np.sin(2 * math.pi * (k + 1) * x + ph[k]) for k in range(3))


def _replicas(case, seed):
    geo = np.random.default_rng([case["set_seed"], 14])  # the set of boxes, the same for every seed
    rng = np.random.default_rng([seed, 15])
    out = []
    for r in range(case["replicas"]):
        n = int(_log_uniform(geo, case["nmin"], case["nmax"]))
        rho, at = geo.uniform(0.4, 0.6), geo.uniform(10.0, 30.0)
        L = np.array([n / (400.0 * rho), 20.0, 20.0])
        if L[0] < 10.0:
            L[0] = 10.0
        # sites of the sparsest cubic grid that holds the molecules, some vacant
        m = np.maximum(1, np.floor(L / (np.prod(L) / n) ** (1.0 / 3.0))).astype(int)
        while np.prod(m) < n:
            m[np.argmax(L / m)] += 1
        sites = geo.permutation(int(np.prod(m)))[:n]
        g = np.stack(np.unravel_index(np.sort(sites), tuple(m)), -1)
        pos = (g + 0.5) * (L / m) + rng.standard_normal((n, 3)) * 0.06
        out.append((np.mod(pos, L), _velocities(rng, n, 1.0), L, float(at)))
    return out


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _precision(case):
    return M.PREC_FP64 if case["precision"] == "fp64" else M.PREC_MIXED


def _molecule_sites(pos, sites, seed):
    """Atoms of molecules of `sites` sites around their centres; relative masses."""
    rng = np.random.default_rng([seed, 16])
    n = len(pos)
    if sites == 1:
        return pos.copy(), np.ones(n)
    w = rng.uniform(0.5, 1.5, (n, sites))
    w /= w.sum(1, keepdims=True)
    d = rng.standard_normal((n, sites, 3)) * 0.1
    d -= (w[:, :, None] * d).sum(1, keepdims=True)
    return (pos[:, None, :] + d).reshape(-1, 3), w.reshape(-1)


class _Array:
    """A [rows][4] device buffer of an Atoms object as a CUDA array.  A tensor
    made from it holds it, and it holds the atoms: the buffer outlives the
    tensor.  (The atoms are made with room for every ghost, so that their
    buffers are never replaced.)"""

    def __init__(self, atoms, pointer, rows):
        addr = ctypes.cast(pointer, ctypes.c_void_p).value
        self.atoms = atoms
        self.__cuda_array_interface__ = {"shape": (rows, 4), "typestr": "<f8", "data": (addr, False), "version": 3}


def _device(atoms, field, rows):
    return torch.as_tensor(_Array(atoms, getattr(atoms.s, field), rows), device="cuda")[:, :3]


def _pinned(n):
    return [torch.empty((n, 3), dtype=torch.float64, pin_memory=True).numpy() for _ in range(3)]


# ---------------------------------------------------------------- prepare --
def prepare(case, seed):
    s = {"case": case}
    kind = case["kind"]
    if kind == "nve":
        pos, vel, L = _lj_inputs(case, seed)
        s["system"] = M.LJSystem(pos, vel, [0, 0, 0], list(L), rc=RC, skin=SKIN, precision=_precision(case), dt=DT,
                                 observe=case["observe"])
        s["out"] = _pinned(len(pos))
    elif kind == "loop":
        pos, vel, L = _lj_inputs(case, seed)
        n = len(pos)
        a = M.Atoms.from_arrays(pos, vel=vel, capacity=int(n * (1 + 3 * LIST / min(L)) ** 3) + 1024)
        s.update(atoms=a, n=n, box=M.Subdomain([0, 0, 0], list(L), LIST), ghosts=M.GhostLayer(a.ctx),
                 list=M.HalfVerletList(a.ctx), lj=M.LennardJones(RC, 1.0, 1.0, 0.7, is_shifted=True, ctx=a.ctx),
                 pos=_device(a, "pos", n), vel=_device(a, "vel", n), force=_device(a, "force", n))
        _forces(s)
    elif kind == "adress":
        pos, vel, L = _gas_inputs(case, seed)
        s["system"] = M.AdResSSystem(pos, vel, [0, 0, 0], list(L), list(L / 2), case["at"], HYBRID["adress"], rc=RC,
                                     skin=SKIN, capping_distance=CAP_ADRESS, precision=_precision(case), dt=DT,
                                     seed=NOISE_SEED, tf_bin_width=TF_BIN)
        s["system"].set_thermodynamic_force(_table(seed, _bins(L)))
    elif kind == "actions":
        pos, vel, L = _gas_inputs(case, seed)
        n, k = len(pos), case["sites"]
        apos, w = _molecule_sites(pos, k, seed)
        cap = int(2.2 * (1 + 2 * LIST / min(L)) ** 2 * n) + 1024
        atoms = M.Atoms.from_arrays(apos, relative_mass=w, capacity=cap * k)
        mol = M.Molecules(cap, atoms.ctx)
        mol.upload(n, pos=pos, atoms_offset=np.arange(n) * k, num_atoms=np.full(n, k))
        box = M.Subdomain([0, 0, 0], list(L), LIST)
        tf = M.ThermodynamicForce(0.5, box, TF_BIN, 1.0, use_periodicity=True, ctx=atoms.ctx)
        tf.setForce(_table(seed, tf.num_bins).reshape(-1, 1))
        s.update(atoms=atoms, mol=mol, box=box, tf=tf, ghosts=M.MultiResGhostLayer(atoms.ctx),
                 list=M.HalfVerletList(atoms.ctx), slab=M.Slab(L / 2, case["at"], HYBRID["actions"], 1),
                 pair=M.LJ_IdealGas(CAP_ADRESS, RC, 1.0, 1.0, True, ctx=atoms.ctx),
                 force=_device(atoms, "force", n * k))
    elif kind == "batch":
        reps = _replicas(case, seed)
        s["system"] = M.BatchSystem(
            [M.Replica(len(p), [0, 0, 0], list(L), list(L / 2), at, 10000 + r) for r, (p, _, L, at) in enumerate(reps)],
            np.concatenate([r[0] for r in reps]), np.concatenate([r[1] for r in reps]), hybrid_diameter=HYBRID["batch"],
            rc=RC, skin=SKIN, capping_distance=CAP_ADRESS, precision=_precision(case), dt=DT, tf_bin_width=TF_BIN,
            list_layout=case["layout"], threads_per_row=case["lanes"])
    else:
        pos, vel, L = _gas_inputs(case, seed)
        rep = M.Replica(len(pos), [0, 0, 0], list(L), list(L / 2), case["at"], NOISE_SEED)
        s["system"] = M.DiffSystem(rep, pos, vel, HYBRID["diff"], steps=case["steps"], window=case["window"],
                                   checkpoint_interval=case["checkpoint"], rc=RC, skin=SKIN,
                                   capping_distance=CAP_ADRESS, precision=_precision(case), dt=DT,
                                   tf_bin_width=L[0] / 100)
        s["table"] = _table(seed, s["system"].num_bins)
    return s


def _bins(L):
    return int(math.ceil(L[0] / TF_BIN))


# -------------------------------------------------------------------- run --
def _rebuild(s):
    a, box = s["atoms"], s["box"]
    s["ghosts"].exchangeRealAtoms(a, box)
    s["ghosts"].createGhostAtoms(a, box)
    s["list"].build(a, 0, a.numLocalAtoms, LIST, 1.0, box.minGhostCorner, box.maxGhostCorner, 64)


def _forces(s, rebuild=True):
    a = s["atoms"]
    if rebuild:
        _rebuild(s)
    a.setForce(0.0)
    s["lj"].apply(a, s["list"], _precision(s["case"]))
    s["ghosts"].contributeBackGhostToReal(a)
    return s["lj"].getEnergy(), s["lj"].getVirial()


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "nve":
        sys_ = state["system"]
        rec = sys_.run_observed(case["steps"]) if case["observe"] else sys_.run(case["steps"])
        pos, vel, force = sys_.state(out=state["out"])
        return {"records": rec, "pos": pos, "vel": vel, "force": force}
    if kind == "loop":
        a = state["atoms"]
        ev = []
        if case["steps"] == 0:
            ev.append(_forces(state))
        for k in range(case["steps"]):
            M.VelocityVerlet.preForceIntegrate(a, DT)
            if k % 10 == 0:
                _rebuild(state)
            else:
                state["ghosts"].updateGhostAtoms(a, state["box"])
            ev.append(_forces(state, rebuild=False))
            M.VelocityVerlet.postForceIntegrate(a, DT)
        return {"records": np.array(ev), "pos": state["pos"], "vel": state["vel"], "force": state["force"]}
    if kind == "adress":
        sys_ = state["system"]
        e = sys_.run(case["steps"])
        pos, vel, force = sys_.state()
        table, density = sys_.thermodynamic_force()
        return {"energy": e, "pos": pos, "vel": vel, "force": force, "table": table, "density": density}
    if kind == "actions":
        atoms, mol, box = state["atoms"], state["mol"], state["box"]
        M.UpdateMolecules.update(mol, atoms, state["slab"])
        state["ghosts"].exchangeRealAtoms(mol, atoms, box)
        state["ghosts"].createGhostAtoms(mol, atoms, box)
        state["list"].build(mol, 0, mol.numLocalMolecules, LIST, 1.0, box.minGhostCorner, box.maxGhostCorner, 64)
        M.UpdateMolecules.update(mol, atoms, state["slab"])
        atoms.setForce(0.0)
        mol.setForce(0.0)
        e = state["pair"].run(mol, state["list"], atoms, _precision(case))
        M.ContributeMoleculeForceToAtoms.update(mol, atoms)
        state["tf"].apply(atoms)
        state["ghosts"].contributeBackGhostToReal(atoms)
        state["tf"].sample(atoms)
        return {"energy": e, "force": state["force"]}
    if kind == "batch":
        sys_ = state["system"]
        e = sys_.run(case["steps"])
        pos, vel, force = sys_.state()
        return {"energy": e, "pos": pos, "vel": vel, "force": force}
    sys_ = state["system"]
    loss = sys_.forward(state["table"], 1.0, 1.0)
    table, eps, sigma = sys_.backward()
    return {"loss": loss, "table": table, "epsilon": eps, "sigma": sigma}


# ------------------------------------------------------------------- work --
def work(case):
    """A pass reads each atom's position and velocity (48 B), writes them and
    the force (72 B) and evaluates every interacting pair once a step.
    Operations of a pair in range: the distance (8), the LJ force factor (9),
    the force on both partners (9), energy and virial (5), 31; with AdResS
    weights and the drift term 45.  A force evaluation alone reads positions
    and writes forces."""
    kind = case["kind"]
    half = 0.5 * 4.0 / 3.0 * math.pi * RC ** 3  # pairs per atom and unit density
    if kind in ("nve", "loop"):
        n = 4 * case["cx"] * case["cy"] * case["cz"] - case["drop"]
        pairs = half * case["rho"]
        if case["steps"] == 0:
            return {"bytes": n * 48.0, "flops": n * pairs * 31}
        return {"bytes": n * 120.0, "flops": n * case["steps"] * (pairs * 31 + 18)}
    if kind == "batch":
        reps = _replicas(case, 0)
        n = sum(len(r[0]) for r in reps)
        inside = sum(min(1.0, (r[3] + 2 * HYBRID["batch"]) / r[2][0]) * len(r[0]) for r in reps)
    else:
        n = 4 * case["cx"] * case["cy"] * case["cz"]
        inside = n * min(1.0, (case["at"] + 2 * HYBRID[kind]) / (2.0 * case["cx"]))
    pairs = inside * half * 0.5
    if kind == "actions":
        k = case["sites"]
        return {"bytes": n * k * 48.0, "flops": pairs * k * k * 45}
    if kind == "diff":
        # the forward and, per step of the sweep, the adjoint of the same pairs
        return {"bytes": n * 48.0, "flops": case["steps"] * (pairs * (45 + 90) + n * 80)}
    return {"bytes": n * 120.0, "flops": case["steps"] * (pairs * 45 + n * 60)}


# ------------------------------------------------------------------ exact --
def _pairs(x, L, r):
    """Unordered pairs within r under periodic boundaries, from sorted cells."""
    dev = x.device
    Lt = torch.as_tensor(L, dtype=torch.float64, device=dev)
    n = [max(1, int(v // r)) for v in L]
    if min(n) < 3:
        idx = torch.arange(len(x), device=dev)
        out = []
        for c in torch.split(idx, 2048):
            d = x[c, None, :] - x[None, :, :]
            d = d - Lt * torch.round(d / Lt)
            k = ((d * d).sum(-1) <= r * r) & (c[:, None] < idx[None, :])
            a, b = torch.nonzero(k, as_tuple=True)
            out.append((c[a], b))
        return torch.cat([o[0] for o in out]), torch.cat([o[1] for o in out])
    nt = torch.tensor(n, device=dev)
    w = torch.remainder(x, Lt)
    c3 = torch.minimum((w / Lt * nt).long(), nt - 1)
    cell = (c3[:, 0] * n[1] + c3[:, 1]) * n[2] + c3[:, 2]
    order = torch.argsort(cell, stable=True)
    count = torch.bincount(cell, minlength=n[0] * n[1] * n[2])
    start = torch.cumsum(count, 0) - count
    m = int(count.max())
    slots = torch.arange(m, device=dev)
    ids = torch.arange(len(count), device=dev)
    g = torch.stack([ids // (n[1] * n[2]), ids // n[2] % n[1], ids % n[2]], -1)
    have = slots[None, :] < count[:, None]
    tab = torch.where(have, order[torch.clamp(start[:, None] + slots, max=len(x) - 1)], -1)
    out = []
    for o in range(14):
        off = torch.tensor([o // 9, o // 3 % 3, o % 3], device=dev) if o < 13 else None
        if off is not None:
            # 13 of the 26 neighbours: one of each opposite couple
            off = torch.tensor([(1, a, b) for a in (-1, 0, 1) for b in (-1, 0, 1)]
                               + [(0, 1, b) for b in (-1, 0, 1)] + [(0, 0, 1)], device=dev)[o]
            h = torch.remainder(g + off, nt)
            other = tab[(h[:, 0] * n[1] + h[:, 1]) * n[2] + h[:, 2]]
        else:
            other = tab
        for part in torch.split(ids, max(1, 60_000_000 // (m * m))):
            a, b = tab[part][:, :, None], other[part][:, None, :]
            keep = (a >= 0) & (b >= 0)
            if off is None:
                keep = keep & (slots[:, None] < slots[None, :])
            p, q, t = torch.nonzero(keep, as_tuple=True)
            i, j = a[p, q, 0], b[p, 0, t]
            d = x[i] - x[j]
            d = d - Lt * torch.round(d / Lt)
            near = (d * d).sum(-1) <= r * r
            out.append((i[near], j[near]))
    return torch.cat([o[0] for o in out]), torch.cat([o[1] for o in out])


def _lj(r2, cap, eps=1.0, sig=1.0):
    """Force factor and shifted energy of the capped potential."""
    s6 = sig ** 6

    def raw(q):
        u3 = 1.0 / (q * q * q)
        return (48 * eps * s6 * s6 * u3 - 24 * eps * s6) * u3 / q, (4 * eps * s6 * s6 * u3 - 4 * eps * s6) * u3

    shift = raw(torch.tensor(RC * RC, dtype=torch.float64, device=r2.device))[1]
    f, e = raw(torch.clamp(r2, min=cap * cap))
    if cap > 0:
        inside = r2 < cap * cap
        if bool(inside.any()):
            fc, ec = raw(torch.tensor(cap * cap, dtype=torch.float64, device=r2.device))
            r = torch.sqrt(r2)
            f = torch.where(inside, fc * cap / r, f)
            e = torch.where(inside, ec - (r - cap) * fc * cap, e)
    return f, e - shift


def _exact_lj(case, seed):
    pos, vel, L = _lj_inputs(case, seed)
    x, v = torch.from_numpy(pos).cuda(), torch.from_numpy(vel).cuda()
    Lt = torch.from_numpy(L).cuda()
    cap = 0.0 if case["kind"] == "nve" else 0.7

    def wrap(x):
        x = torch.where(x >= Lt, x - Lt, x)
        return torch.where(x < 0, x + Lt, x)

    def forces(x, ij):
        F = torch.zeros_like(x)
        E = W = 0.0
        for i, j in zip(torch.split(ij[0], 20_000_000), torch.split(ij[1], 20_000_000)):
            d = x[i] - x[j]
            d -= Lt * torch.round(d / Lt)
            r2 = (d * d).sum(-1)
            near = torch.nonzero(r2 <= RC * RC)[:, 0]
            i, j, d, r2 = i[near], j[near], d[near], r2[near]
            f, e = _lj(r2, cap)
            E, W = E + float(e.sum()), W - 0.5 * float((f * r2).sum())
            d *= f[:, None]
            F.index_add_(0, i, d)
            F.index_add_(0, j, d, alpha=-1.0)
        return F, E, W

    x = wrap(x)
    ij = _pairs(x, L, LIST)
    F, E, W = forces(x, ij)
    rec = []
    if case["kind"] == "loop" and case["steps"] == 0:
        rec.append((E, W))
    for k in range(case["steps"]):
        v = v + 0.5 * DT * F
        x = x + DT * v
        if k % 10 == 0:
            x = wrap(x)
            ij = _pairs(x, L, LIST)
        F, E, W = forces(x, ij)
        v = v + 0.5 * DT * F
        rec.append((E, W) + ((0.5 * float((v * v).sum()),) + tuple(v.sum(0).tolist()) if case.get("observe") else ()))
    return {"records": np.array(rec), "pos": x, "vel": v, "force": F}


def _slab(x, center, at, hy):
    """lambda and its x derivative (cos^2 weighting, nu = 1)."""
    dx = x - center
    ad = dx.abs()
    arg = math.pi / (2 * hy) * (ad - 0.5 * at)
    hybrid = (ad >= 0.5 * at) & (ad <= 0.5 * at + hy)
    c, s = torch.cos(arg), torch.sin(arg)
    lam = torch.where(hybrid, c * c, (ad < 0.5 * at).double())
    grad = torch.where(hybrid, -math.pi / hy * s * c * torch.sign(dx), torch.zeros_like(x))
    return lam, grad


def _noise(seed, step, atom):
    """Three normals per molecule: Philox4x32-10 and Box-Muller on 23-bit
    uniforms, in FP32 as the thermostat defines them."""
    mask = 0xFFFFFFFF
    c = [atom & mask, atom >> 32, torch.full_like(atom, step), torch.zeros_like(atom)]
    k0, k1 = seed & mask, seed >> 32
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & mask) ^ c[1] ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ c[3] ^ k1, p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    u = [((q >> 9).float() + 0.5) * 2.0 ** -23 for q in c]
    ra, rb = torch.sqrt(_log_f32(u[0]) * -2.0), torch.sqrt(_log_f32(u[2]) * -2.0)
    (ca, sa), (cb, _) = _cos_sin_f32(u[1]), _cos_sin_f32(u[3])
    return torch.stack([ra * ca, ra * sa, rb * cb], -1).double()


def _fma(a, b, c):
    d = lambda v: v.double() if torch.is_tensor(v) else np.float32(v).item()  # noqa: E731
    return (d(a) * d(b) + d(c)).float()


def _log_f32(u):
    """ln u as the mantissa's 2 atanh series, each operation rounded to FP32."""
    m, e = torch.frexp(u)
    low = m * 2.0 <= float.fromhex("0x1.6a09e6p+0")  # mantissa to [sqrt(1/2), sqrt(2)]
    m, e = torch.where(low, m * 2.0, m), e - low.int()
    t = (m - 1.0) / (m + 1.0)
    t2 = t * t
    p = _fma(t2, float.fromhex("0x1.c71c72p-4"), float.fromhex("0x1.24924ap-3"))
    for k in ("0x1.99999ap-3", "0x1.555556p-2", "0x1p0"):
        p = _fma(p, t2, float.fromhex(k))
    return _fma(e.float(), float.fromhex("0x1.62e430p-1"), t * p * 2.0)


def _cos_sin_f32(u):
    """cos and sin of 2 pi u by quarter turns and Taylor polynomials in FP32."""
    q = torch.round(u * 4.0)
    f = (u - q * 0.25) * float.fromhex("0x1.921fb6p+2")
    f2 = f * f
    s = _fma(f2, float.fromhex("0x1.71de3ap-19"), float.fromhex("-0x1.a01a02p-13"))
    for k in ("0x1.111112p-7", "-0x1.555556p-3"):
        s = _fma(s, f2, float.fromhex(k))
    s = _fma(f * f2, s, f)
    c = _fma(f2, float.fromhex("-0x1.27e4fcp-22"), float.fromhex("0x1.a01a02p-16"))
    for k in ("-0x1.6c16c2p-10", "0x1.555556p-5", "-0x1p-1", "0x1p0"):
        c = _fma(c, f2, float.fromhex(k))
    k = q.long() & 3
    return (torch.where(k == 0, c, torch.where(k == 1, -s, torch.where(k == 2, -c, s))),
            torch.where(k == 0, s, torch.where(k == 1, c, torch.where(k == 2, -s, -c))))


def _oriented(x, box, i, j):
    """Each pair as (own, partner, the partner's periodic shift): the instance
    whose partner lies lexicographically above its own molecule, the one that
    the half list holds.  Near a periodic face the two instances see different
    weights."""
    shift = box[i] * torch.round((x[i] - x[j]) / box[i])
    d = x[j] + shift - x[i]
    above = (d[:, 0] > 0) | ((d[:, 0] == 0) & ((d[:, 1] > 0) | ((d[:, 1] == 0) & (d[:, 2] > 0))))
    return torch.where(above, i, j), torch.where(above, j, i), torch.where(above[:, None], shift, -shift)


def _adress_force(x, pairs, weights, eps, sig, count, replica):
    """Weighted pair forces with the drift force; per-replica energies; the
    half pair energies of pairs with a hybrid member."""
    i, j, shift = pairs
    li, gi = weights(x[:, 0][i], i)
    lj, gj = weights(x[:, 0][j] + shift[:, 0], j)
    d = x[i] - x[j] - shift
    r2 = (d * d).sum(-1)
    k = torch.nonzero(((li > 0) | (lj > 0)) & (r2 <= RC * RC))[:, 0]
    i, j, li, lj, gi, gj, d, r2 = i[k], j[k], li[k], lj[k], gi[k], gj[k], d[k], r2[k]
    f, e = _lj(r2, CAP_ADRESS, eps, sig)
    w = 0.5 * (li + lj)
    g = d * (f * w)[:, None]
    hi, hj = (li > 0) & (li < 1), (lj > 0) & (lj < 1)
    V = torch.where(hi | hj, 0.5 * e, torch.zeros_like(e))
    F = torch.zeros_like(x).index_add(0, i, g).index_add(0, j, -g)
    drift = torch.zeros_like(x[:, 0]).index_add(0, i, -V * gi).index_add(0, j, -V * gj)
    E = torch.zeros(count, dtype=torch.float64, device=x.device).index_add(0, replica[i], (e * w).detach())
    samples = (torch.cat([replica[i][hi], replica[j][hj]]), torch.cat([li[hi], lj[hj]]).detach(),
               torch.cat([V[hi], V[hj]]).detach())
    return torch.cat([(F[:, 0] + drift)[:, None], F[:, 1:]], 1), E, samples


def _bin200(lam):
    return torch.clamp((lam.detach() * 200).floor().long(), 0, 199)


def _exact_adress(replicas, hy_width, steps, interval, table=None, eps=1.0, sig=1.0, bin_width=TF_BIN, frozen=False,
                  on_step=None):
    """Langevin AdResS trajectories of independent single-site replicas."""
    dev = "cuda"
    R = len(replicas)
    x = torch.cat([torch.from_numpy(r["pos"]) for r in replicas]).to(dev)
    v = torch.cat([torch.from_numpy(r["vel"]) for r in replicas]).to(dev)
    sizes = [len(r["pos"]) for r in replicas]
    start = np.concatenate([[0], np.cumsum(sizes)])
    rep = torch.repeat_interleave(torch.arange(R), torch.tensor(sizes)).to(dev)
    box = torch.tensor(np.array([r["L"] for r in replicas]), device=dev)[rep]
    at = torch.tensor([r["at"] for r in replicas], dtype=torch.float64, device=dev)[rep]
    index = torch.cat([torch.arange(n) for n in sizes]).to(dev)
    c1, c2 = math.exp(-DT), math.sqrt(1 - math.exp(-2 * DT))
    nbins = [int(math.ceil(r["L"][0] / bin_width)) for r in replicas]
    inv = torch.tensor([b / r["L"][0] for b, r in zip(nbins, replicas)], dtype=torch.float64, device=dev)[rep]
    nb = torch.tensor(nbins, device=dev)[rep]
    F = torch.zeros_like(x)
    mean = None if frozen else torch.zeros((R, 200), dtype=torch.float64, device=dev)
    density = torch.zeros(nbins[0], dtype=torch.float64, device=dev)
    energies = []
    pairs = None

    def weights(px, idx):
        return _slab(px, 0.5 * box[:, 0][idx], at[idx], hy_width)

    for st in range(steps):
        v = v + 0.5 * DT * F
        x = x + 0.5 * DT * v
        noise = torch.cat([_noise(r["seed"], st, index[start[k]:start[k + 1]]) for k, r in enumerate(replicas)])
        v = v * c1 + c2 * noise
        x = x + 0.5 * DT * v
        if st % interval == 0:
            with torch.no_grad():
                shift = torch.where(x >= box, -box, torch.where(x < 0, box, torch.zeros_like(box)))
            x = x + shift
            with torch.no_grad():
                parts = [_pairs(x[start[k]:start[k + 1]], r["L"], LIST) for k, r in enumerate(replicas)]
                pairs = _oriented(x, box, *[torch.cat([p[q] + int(start[k]) for k, p in enumerate(parts)])
                                            for q in (0, 1)])
        F, E, (srep, slam, sV) = _adress_force(x, pairs, weights, eps, sig, R, rep)
        lam, grad = weights(x[:, 0], slice(None))
        hyb = (lam > 0) & (lam < 1)
        if not frozen:
            F[:, 0] += torch.where(hyb, mean[rep, _bin200(lam)] * grad, torch.zeros_like(grad))
            if st == 0:  # the first run is sampled and updates the compensation mean
                tot = torch.zeros(R * 200, dtype=torch.float64, device=dev).index_add_(0, srep * 200 + _bin200(slam), sV)
                cnt = torch.bincount((rep * 200 + _bin200(lam))[hyb], minlength=R * 200).double()
                mean = torch.where(cnt > 0, tot / torch.clamp(cnt, min=1) / 11.0, torch.zeros_like(tot)).reshape(R, 200)
        b = torch.floor(x.detach()[:, 0] * inv).long()
        ok = (b >= 0) & (b < nb)
        if table is not None:
            F = torch.cat([(F[:, 0] + torch.where(ok, table[torch.where(ok, b, 0)], 0.0))[:, None], F[:, 1:]], 1)
        if R == 1:
            density += torch.bincount(b[ok], minlength=nbins[0]).double()
        v = v + 0.5 * DT * F
        energies.append(E)
        if on_step is not None:
            on_step(st, x)
    return x, v, F, torch.stack(energies), density


def _exact_diff(case, seed):
    pos, vel, L = _gas_inputs(case, seed)
    bins = int(math.ceil(L[0] / (L[0] / 100)))
    table = torch.tensor(_table(seed, bins), device="cuda", requires_grad=True)
    eps = torch.tensor(1.0, dtype=torch.float64, device="cuda", requires_grad=True)
    sig = torch.tensor(1.0, dtype=torch.float64, device="cuda", requires_grad=True)
    width = L[0] / 128
    span = int(math.ceil(6.0 / width)) + 1
    o = torch.arange(-span, span + 1, device="cuda")
    rho = [torch.zeros(128, dtype=torch.float64, device="cuda")]

    def on_step(st, x):
        if st < case["steps"] - case["window"]:
            return
        b = torch.remainder(torch.floor(x.detach()[:, :1] / width).long() + o, 128)
        d = x[:, :1] - (b + 0.5) * width
        d = d - L[0] * torch.round(d.detach() / L[0])
        k = torch.where(d.detach().abs() <= 6.0, torch.exp(-0.5 * d * d) / math.sqrt(2 * math.pi), torch.zeros_like(d))
        rho[0] = rho[0].index_add(0, b.reshape(-1), k.reshape(-1))

    rep = {"pos": pos, "vel": vel, "L": L, "at": case["at"], "seed": NOISE_SEED}
    _exact_adress([rep], HYBRID["diff"], case["steps"], 5, table, eps, sig, L[0] / 100, True, on_step)
    area = L[1] * L[2]
    loss = ((rho[0] / (case["window"] * area) - len(pos) / (L[0] * area)) ** 2).sum()
    loss.backward()
    return {"loss": float(loss), "table": table.grad, "epsilon": float(eps.grad), "sigma": float(sig.grad)}


def _exact_actions(case, seed):
    pos, _, L = _gas_inputs(case, seed)
    k = case["sites"]
    apos, w = _molecule_sites(pos, k, seed)
    n = len(pos)
    a = torch.from_numpy(apos).cuda().reshape(n, k, 3)
    w = torch.from_numpy(w).cuda().reshape(n, k)
    Lt = torch.from_numpy(L).cuda()
    x = (a * w[:, :, None]).sum(1)
    shift = torch.where(x >= Lt, -Lt, torch.where(x < 0, Lt, torch.zeros_like(Lt)))
    x, a = x + shift, a + shift[:, None, :]
    lam, grad = _slab(x[:, 0], float(L[0] / 2), case["at"], HYBRID["actions"])
    i, j = _pairs(x, L, LIST)
    act = (lam[i] > 0) | (lam[j] > 0)
    i, j = i[act], j[act]
    image = Lt * torch.round((x[i] - x[j]) / Lt)
    F = torch.zeros_like(a)
    hy = (lam > 0) & (lam < 1)
    vsum = torch.zeros_like(lam)
    E = 0.0
    for p in range(k):
        for q in range(k):
            d = a[i, p] - a[j, q] - image
            r2 = (d * d).sum(-1)
            near = r2 <= RC * RC
            I, J, d, r2 = i[near], j[near], d[near], r2[near]
            f, e = _lj(r2, CAP_ADRESS)
            wt = 0.5 * (lam[I] + lam[J])
            g = d * (f * wt)[:, None]
            F[:, p].index_add_(0, I, g)
            F[:, q].index_add_(0, J, -g)
            E += float((e * wt).sum())
            V = torch.where(hy[I] | hy[J], 0.5 * e, torch.zeros_like(e))
            vsum.index_add_(0, I, V)
            vsum.index_add_(0, J, V)
    F[:, :, 0] += w * (-vsum * grad)[:, None]
    bins = _bins(L)
    b = torch.floor(a[:, :, 0] * (bins / L[0])).long()
    ok = (b >= 0) & (b < bins)
    F[:, :, 0] += torch.where(ok, torch.from_numpy(_table(seed, bins)).cuda()[torch.where(ok, b, 0)], 0.0)
    return {"energy": E, "force": F.reshape(-1, 3)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("nve", "loop"):
        return _exact_lj(case, seed)
    if kind == "actions":
        return _exact_actions(case, seed)
    if kind == "diff":
        return _exact_diff(case, seed)
    if kind == "adress":
        pos, vel, L = _gas_inputs(case, seed)
        table = torch.from_numpy(_table(seed, _bins(L))).cuda()
        rep = [{"pos": pos, "vel": vel, "L": L, "at": case["at"], "seed": NOISE_SEED}]
        x, v, F, e, density = _exact_adress(rep, HYBRID["adress"], case["steps"], 10, table)
        return {"energy": e[:, 0], "pos": x, "vel": v, "force": F, "table": table, "density": density}
    reps = [{"pos": p, "vel": v, "L": L, "at": at, "seed": 10000 + r}
            for r, (p, v, L, at) in enumerate(_replicas(case, seed))]
    x, v, F, e, _ = _exact_adress(reps, HYBRID["batch"], case["steps"], 10)
    return {"energy": e, "pos": x, "vel": v, "force": F}
