"""Timed cases of the GCMC energy path.

What a program does with this library, through `raspa2_b200.native` (the ctypes
binding of include/raspa_gpu.h):

- "points":   energies of bead positions (the trial loops of CBMC), 1 to 64 a call;
- "displace": the calls of an accepted translation: the pair-energy difference,
              the Ewald Fourier difference, its acceptance and the new position;
- "rescore":  a configuration is uploaded and its total energy recomputed (a
              restart, a drift check, a served job's admission);
- "grid":     an energy grid (LJ or Coulomb) is built from the framework;
- "lookup":   an energy grid is interpolated at points held on the host;
- "engine":   a block of MC moves of many boxes: upload of every configuration,
              the moves, and every state read back.

Frameworks have the density, charges and cavity of the synthetic systems of
`raspa2_b200.systems`, on a jittered lattice, so that they are made quickly.
"""
import dataclasses
import itertools
import math

import numpy as np
import torch

from raspa2_b200 import native, systems, units

MAXMOL = 384                # molecule capacity of an engine's box
DENSITY = 0.0894            # framework atoms per cubic Angstrom (the CO2 systems)
PRECISION = {"fp64": native.RGPU_FP64, "mixed": native.RGPU_MIXED, "mixed_cc64": native.RGPU_MIXED_CC64}


# --------------------------------------------------------------------------
# cases

def listed():
    return [
        # one position of an uncharged molecule in the 3456-atom methane box: the call the drop-in
        # bridge makes for every trial of the reference's own loop
        dict(name="point_fp64", kind="points", model="methane", precision="fp64", n=1, atoms=3456, cell=40.0,
             load=0.3, tri=False),
        # the 20 beads of 10 orientation trials of CO2 in the 1536-atom box
        dict(name="trials_fp64", kind="points", model="co2", precision="fp64", n=20, atoms=1536, cell=25.8,
             load=0.6, tri=False),
        # an odd number of trials in a triclinic cell
        dict(name="trials_fp64_triclinic", kind="points", model="co2", precision="fp64", n=31, atoms=2000,
             cell=29.0, load=0.6, tri=True),
        # the largest batch a call takes, in the largest box, mixed precision
        dict(name="trials_mixed_64", kind="points", model="co2", precision="mixed", n=64, atoms=4096, cell=36.0,
             load=1.0, tri=False),
        # an accepted translation and the one back, one move at a time from the host
        dict(name="displace_fp64", kind="displace", model="co2", precision="fp64", atoms=1536, cell=25.8, kmax=8,
             load=0.6, tri=False),
        # a large loaded box recomputed from scratch
        dict(name="rescore_4096", kind="rescore", model="co2", atoms=4096, cell=36.0, kmax=10, load=1.0, tri=False),
        # energy grids: hexane's framework at 0.4 A, and a Coulomb grid with an odd number of points
        dict(name="grid_lj", kind="grid", model="hexane", coulomb=False, atoms=4096, cell=40.0, points=101,
             tri=False),
        dict(name="grid_coulomb", kind="grid", model="co2", coulomb=True, atoms=1536, cell=25.8, points=77,
             tri=False),
        # lookups of host positions
        dict(name="lookup_100k", kind="lookup", model="hexane", atoms=1200, cell=26.0, points=65, n=99991),
        # one box alone (the plain single-system run)
        dict(name="engine_fp64_one", kind="engine", model="co2", precision="fp64", boxes=1, atoms=1536, cell=25.8,
             kmax=8, load=0.6, moves=200, threads=512, tri=False),
        # the batched workload: boxes of 512 to 4096 atoms, mixed precision
        dict(name="engine_mixed_64", kind="engine", model="co2", precision="mixed", boxes=64, atoms=4096, cell=36.0,
             kmax=10, load=0.8, moves=1000, threads=1024, tri=False),
        # flexible chains over shared energy grids
        dict(name="engine_hexane_32", kind="engine", model="hexane", precision="mixed", boxes=32, atoms=1200,
             cell=26.0, kmax=0, load=0.4, moves=100, threads=512, tri=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo=300, hi=4096):
    """An atom count and the cell that gives it the CO2 systems' density (at least twice the cut-off)."""
    n = _log(rng, lo, hi)
    return n, round(max(24.1, (n / DENSITY) ** (1.0 / 3.0)), 2)


def draw(rng):
    kind = rng.choice(["points", "points", "displace", "rescore", "grid", "lookup", "engine", "engine"])
    n, cell = _box(rng)
    load = round(rng.uniform(0.1, 1.0), 3)
    tri = rng.random() < 0.2
    if kind == "points":
        model = rng.choice(["methane", "co2", "co2"])
        return dict(kind=kind, model=model, precision=rng.choice(["fp64", "fp64", "mixed"]), n=_log(rng, 1, 64),
                    atoms=n, cell=cell, load=load, tri=tri)
    if kind == "displace":
        return dict(kind=kind, model="co2", precision=rng.choice(["fp64", "fp64", "mixed"]), atoms=n, cell=cell,
                    kmax=rng.randint(6, 10), load=load, tri=tri)
    if kind == "rescore":
        return dict(kind=kind, model="co2", atoms=n, cell=cell, kmax=rng.randint(6, 10), load=load, tri=tri)
    if kind == "grid":
        coulomb = rng.random() < 0.4
        return dict(kind=kind, model="co2" if coulomb else rng.choice(["methane", "hexane", "co2"]), coulomb=coulomb,
                    atoms=n, cell=cell, points=2 * rng.randint(15, 38) + 1, tri=tri)
    if kind == "lookup":
        return dict(kind=kind, model="hexane", atoms=_log(rng, 300, 1200), cell=26.0, points=2 * rng.randint(20, 32) + 1,
                    n=_log(rng, 1, 100000))
    model = rng.choice(["co2", "co2", "methane", "hexane"])
    boxes = _log(rng, 1, 48)
    if model == "hexane":
        boxes = min(boxes, 32)
        return dict(kind=kind, model=model, precision="mixed", boxes=boxes, atoms=_log(rng, 600, 1200), cell=26.0,
                    kmax=0, load=round(0.4 * load, 3), moves=rng.randint(50, 100), threads=512, tri=False)
    precision = rng.choice(["fp64", "mixed", "mixed", "mixed_cc64"])
    # FP64 engines have at most 512 threads
    return dict(kind=kind, model=model, precision=precision, boxes=boxes, atoms=n, cell=cell,
                kmax=rng.randint(6, 10) if model == "co2" else 0, load=load, moves=rng.randint(50, 200),
                threads=512 if precision == "fp64" or boxes < 16 else 1024, tri=tri)


# --------------------------------------------------------------------------
# inputs

MOLECULE = {"methane": systems.METHANE, "co2": systems.CO2, "hexane": systems.HEXANE}
ANGLES = (80.0, 95.0, 110.0)


def _lattice(m):
    g = (np.arange(m) + 0.5) / m
    return np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)


def _pore(cell):
    """Radius of the cavity around the cell's centre (systems.VOID_FRACTION of a cube)."""
    return cell * (3.0 * systems.VOID_FRACTION / (4.0 * math.pi)) ** (1.0 / 3.0)


def _framework(rng, n, cell):
    """n fractional positions in the wall around the cavity: sites of the coarsest lattice that has n of them
    there, each jittered by up to 6 % of the lattice constant."""
    r = _pore(cell) / cell
    m = int((n / (1.0 - systems.VOID_FRACTION)) ** (1.0 / 3.0))
    while True:
        s = _lattice(m)
        s = s[np.sum((s - 0.5) ** 2, axis=1) >= r * r]
        if len(s) >= n:
            break
        m += 1
    s = s[rng.permutation(len(s))[:n]]
    return np.round(np.mod(s + rng.uniform(-0.06, 0.06, s.shape) / m, 1.0), 12)


def _system(case, rng, i=0, atoms=None, cell=None, kmax=None):
    n, c = atoms or case["atoms"], cell or case["cell"]
    model = case["model"]
    frac = _framework(rng, n, c)
    mol = MOLECULE[model]
    charged = model == "co2"
    if charged:
        q = np.rint(rng.uniform(-1.2, 1.2, n) * 1e8).astype(np.int64)
        q -= q.sum() // n
        q[-1] -= q.sum()
        q = q * 1e-8
    else:
        q = np.zeros(n)
    types = ["Sifw"] * (n // 3) + ["Ofw"] * (n - n // 3)
    types = [types[k] for k in rng.permutation(n)]
    moves = systems.MoveMix(translation=1.0, rotation=0.0 if model == "methane" else 1.0, swap_insert=1.0,
                            swap_delete=1.0, reinsertion=1.0 if model == "hexane" else 0.0)
    lengths = np.array([c, c, c]) if not case.get("tri") else np.array([c * 1.10, c * 1.12, c * 1.14])
    return systems.System(
        name=f"{model}_{i}", unit_cell=lengths, unit_cells=np.array([1, 1, 1]), frac=frac, uc_types=types,
        uc_charges=q, molecule=mol, temperature=(273.0, 298.0, 323.0)[i % 3] if model != "hexane" else 433.0,
        pressure=float(10.0 ** rng.uniform(4.0, 6.5)), cutoff=12.0, ewald=charged, alpha=0.265,
        kmax=(kmax or case.get("kmax") or 6,) * 3, trials=16 if model == "hexane" else 10,
        trials_first_bead=8 if model == "hexane" else 10, moves=moves, seed=i,
        ideal_gas_rosenbluth=systems.chain_ideal_gas_estimate(mol, 433.0) if model == "hexane" else 1.0,
        cell_angles=ANGLES if case.get("tri") else (90.0, 90.0, 90.0))


def _chain(rng, start):
    """A hexane with all-trans dihedrals in a random direction."""
    x = systems.HEXANE.positions
    q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    return start + (x - x.mean(0)) @ q.T


def _molecules(rng, s, load):
    """Molecules on a jittered lattice of the cavity, `load` of its sites taken, apart from one another."""
    c = s.unit_cell
    gap = {"methane": 4.1, "CO2": 4.2, "hexane": 6.5}[s.molecule.name]
    r = (_pore(float(c.min())) - 2.6) * (0.8 if s.triclinic else 1.0)
    m = max(1, int(float(c.min()) / gap))
    f = _lattice(m)
    f = f[np.sum(((f - 0.5) * c) ** 2, axis=1) < r * r]
    f = f[rng.permutation(len(f))[: max(1, int(round(load * len(f))))]]
    x = s.box_point(f + rng.uniform(-0.05, 0.05, f.shape) / m)
    ref = s.molecule.positions - s.molecule.positions[s.molecule.starting_bead]
    out = []
    for p in x:
        if not s.molecule.rigid:
            out.append(_chain(rng, p))
        elif len(ref) == 1:
            out.append(p[None, :])
        else:
            # of 16 random orientations the one furthest from the molecules placed so far
            u = rng.normal(size=(16, 1, 3))
            t = p + np.linalg.norm(ref, axis=1)[:, None] * np.sign(ref[:, 2:3]) * (u / np.linalg.norm(u, axis=2, keepdims=True))
            if out:
                y = np.array(out)
                y = y[np.sum((y[:, s.molecule.starting_bead] - p) ** 2, axis=1) < 49.0].reshape(-1, 3)
                if len(y):
                    t = t[[np.argmax(np.min(np.sum((t[:, :, None] - y) ** 2, axis=3), axis=(1, 2)))]]
            out.append(t[0])
    return np.array(out).reshape(-1, len(ref), 3)


def _in_cavity(rng, s, n):
    """Positions in the cavity and up to its wall."""
    r = (_pore(float(s.unit_cell.min())) - 1.8) * (0.75 if s.triclinic else 1.0)
    out = np.empty((0, 3))
    while len(out) < n:
        u = rng.uniform(-1.0, 1.0, (4 * n + 8, 3))
        out = np.concatenate([out, u[np.sum(u * u, axis=1) < 1.0]])
    return s.box_point(np.full(3, 0.5)) + r * out[:n]


def _loaded(case, seed):
    rng = np.random.default_rng(seed)
    s = _system(case, rng)
    mols = _molecules(rng, s, case["load"])
    return rng, s, mols


def _points_input(case, seed):
    rng, s, mols = _loaded(case, seed)
    n, na = case["n"], s.molecule.n_atoms
    return s, mols, _in_cavity(rng, s, n), rng.integers(0, na, n), rng.integers(-1, len(mols), n)


def _displace_input(case, seed):
    rng, s, mols = _loaded(case, seed)
    m = int(rng.integers(0, len(mols)))
    return s, mols, m, mols[m] + rng.uniform(-0.2, 0.2, 3)


def _grid_geometry(case, s):
    p = case["points"]
    npts = np.array([p, p, p], np.int32)
    if s.triclinic:
        mat = s.unit_cell_matrix
        return npts, np.abs(mat).sum(axis=1), np.minimum(mat, 0.0).sum(axis=1)
    return npts, np.asarray(s.unit_cell, float), np.zeros(3)


def _probe(s):
    return int(s.molecule_types()[0])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "points":
        s, mols, xyz, atom, excl = _points_input(case, seed)
        g = native.GpuSystem(s, maxmol=512, seed=seed)
        g.set_adsorbates(mols)
        return dict(kind=kind, g=g, args=(xyz, atom.astype(np.int32), excl.astype(np.int32), PRECISION[case["precision"]]))
    if kind == "displace":
        s, mols, m, new = _displace_input(case, seed)
        g = native.GpuSystem(s, maxmol=512, seed=seed)
        g.set_adsorbates(mols)
        return dict(kind=kind, g=g, m=m, new=new, old=mols[m].copy(), precision=PRECISION[case["precision"]])
    if kind == "rescore":
        _, s, mols = _loaded(case, seed)
        return dict(kind=kind, g=native.GpuSystem(s, maxmol=512, seed=seed), mols=mols)
    if kind == "grid":
        s = _system(case, np.random.default_rng(seed))
        npts, size, shift = _grid_geometry(case, s)
        out = torch.empty(tuple(int(x) + 1 for x in npts) + (8,), dtype=torch.float32, device="cuda")
        g = native.GpuSystem(s, maxmol=8, seed=seed)
        return dict(kind=kind, g=g, coulomb=case["coulomb"], type=_probe(s), geom=(npts, size, shift), out=out)
    if kind == "lookup":
        rng = np.random.default_rng(seed)
        s = _system(case, rng)
        npts, size, shift = _grid_geometry(case, s)
        grid = _lj_grid(s, _probe(s), npts, size, shift).float().contiguous()
        xyz = s.box_point(rng.uniform(-0.5, 1.5, (case["n"], 3)))
        return dict(kind=kind, grid=grid, geom=(npts, size, shift, np.asarray(s.unit_cell, float)), xyz=xyz)
    return _engine_state(case, seed)


def _engine_state(case, seed):
    rng = np.random.default_rng(seed)
    frames, hexane = {}, case["model"] == "hexane"
    gs, conf = [], []
    keep = []
    for i in range(case["boxes"]):
        # boxes of uneven size: from an eighth of the largest one's atoms up to it (hexane: one framework)
        k = 0 if hexane else i % 8
        if k not in frames:
            n = case["atoms"] if k == 0 else max(min(case["atoms"], 300), int(case["atoms"] * (8 - k) / 8))
            cell = case["cell"] if k == 0 else max(24.1, min(case["cell"], (n / DENSITY) ** (1.0 / 3.0)))
            kmax = None if not case["kmax"] else max(6, case["kmax"] - (k + 1) // 2)
            frames[k] = _system(case, rng, k, n, cell, kmax)
            if hexane:
                s = frames[k]
                npts, size, shift = _grid_geometry(dict(points=65), s)
                keep = [npts, size, shift, {t: _lj_grid(s, t, npts, size, shift).float().contiguous()
                                            for t in sorted(set(s.molecule_types().tolist()))}]
        s = dataclasses.replace(frames[k], pressure=float(10.0 ** rng.uniform(4.0, 6.5)))
        mols = _molecules(rng, s, case["load"] * rng.uniform(0.3, 1.0))
        g = native.GpuSystem(s, maxmol=MAXMOL, seed=seed, stream_id=i)
        if hexane:
            g.set_grids([keep[3][int(t)].data_ptr() for t in s.molecule_types()], keep[0], keep[1], keep[2],
                        np.asarray(s.unit_cell, float))
        gs.append(g)
        conf.append(mols)
    eng = native.Engine(gs, precision=PRECISION[case["precision"]], threads=case["threads"])
    return dict(kind="engine", eng=eng, conf=conf, moves=case["moves"], keep=keep)


def run(state):
    kind = state["kind"]
    if kind == "points":
        return state["g"].bead_energies(*state["args"])
    if kind == "displace":
        g, m, p = state["g"], state["m"], state["precision"]
        out = []
        for x in (state["new"], state["old"]):
            overlap, du = g.move_difference(m, x, p)
            dew = g.ewald_difference(m, x, p)
            g.ewald_accept()
            g.update_molecule(m, x)
            out.append(dict(overlap=overlap, pair=du, fourier=dew))
        return out
    if kind == "rescore":
        state["g"].set_adsorbates(state["mols"])
        return state["g"].total_energy()
    if kind == "grid":
        g, (npts, size, shift), out = state["g"], state["geom"], state["out"]
        if state["coulomb"]:
            g.grid_build_coulomb(npts, size, shift, out.data_ptr())
        else:
            g.grid_build(state["type"], npts, size, shift, out.data_ptr())
        return out
    if kind == "lookup":
        return native.grid_interpolate(state["grid"].data_ptr(), *state["geom"], state["xyz"])
    eng = state["eng"]
    eng.set_adsorbates(state["conf"])
    eng.run(state["moves"])
    st = eng.get_states()
    xyz = np.zeros((len(st), MAXMOL) + state["conf"][0].shape[1:])
    for d, x in zip(st, xyz):
        x[:d["nmol"]] = d["xyz"]
    return dict(energy=np.stack([d["energy"] for d in st]),
                # attempts and acceptances of each move type, moves, overlaps
                counters=np.stack([np.concatenate([d["counters"][:10], d["counters"][18:20]]) for d in st]),
                nmol=np.array([d["nmol"] for d in st]), status=np.array([d["status"] for d in st]),
                xyz=xyz)


# --------------------------------------------------------------------------
# what a pass cannot do without

def _incut(atoms, cell):
    """Framework atoms inside the cut-off of a position, on average."""
    return atoms / cell ** 3 * (4.0 / 3.0) * math.pi * 12.0 ** 3


def _nk(k):
    return len(systems.kvector_indices((k, k, k)))


def work(case):
    kind, model = case["kind"], case["model"]
    pair = 49.0 if model == "co2" else 25.0       # FLOP of a pair inside the cut-off
    if kind == "grid":
        p = (case["points"] + 1) ** 3
        return {"bytes": 32.0 * p + 32.0 * case["atoms"],
                "flops": p * _incut(case["atoms"], case["cell"]) * (90.0 if case["coulomb"] else 60.0)}
    if kind == "lookup":
        grid = 32.0 * (case["points"] + 1) ** 3
        return {"bytes": min(grid, 256.0 * case["n"]) + 32.0 * case["n"], "flops": 200.0 * case["n"]}
    r = _pore(case["cell"]) - 2.6
    nmol = case["load"] * 4.0 / 3.0 * math.pi * r ** 3 / {"methane": 4.1, "co2": 4.2, "hexane": 6.5}[model] ** 3
    nads = nmol * MOLECULE[model].n_atoms
    near = _incut(case["atoms"], case["cell"]) + 0.5 * nads
    fw = 32.0 * case["atoms"]
    if kind == "points":
        return {"bytes": fw + 32.0 * nads + 64.0 * case["n"], "flops": case["n"] * near * pair}
    if kind == "displace":
        nk = _nk(case["kmax"])
        return {"bytes": 2 * (fw + 32.0 * nads + 56.0 * nk), "flops": 2 * (6 * near * pair + nk * (6 * 10.0 + 12.0))}
    if kind == "rescore":
        nk = _nk(case["kmax"])
        return {"bytes": fw + 56.0 * nads + 44.0 * nk, "flops": nads * near * pair + nk * (10.0 * nads + 12.0)}
    # per move: half displacements (old and new beads), half insertions and deletions (all trials)
    beads = {"methane": 6.0, "co2": 18.0, "hexane": 60.0}[model]
    nk = _nk(case["kmax"]) if case["kmax"] else 0
    scale = 0.55 if model != "hexane" else 1.0    # the boxes' mean size against the largest's
    moves = case["moves"] * case["boxes"]
    if model == "hexane":
        per = beads * (200.0 + 0.5 * 0.6 * nads * pair)
    else:
        per = beads * near * pair + scale * nk * 72.0
    return {"bytes": case["boxes"] * (scale * fw + 48.0 * nads + 44.0 * nk), "flops": moves * per}


# --------------------------------------------------------------------------
# the same results in 64 bits, from plain torch

def _t(x):
    return torch.as_tensor(np.asarray(x, float), dtype=torch.float64, device="cuda" if torch.cuda.is_available() else "cpu")


def _image(s, d):
    """Minimum image of difference vectors d[..., 3]."""
    h = _t(s.box_matrix)
    f = d @ torch.linalg.inv(h).T
    return (f - torch.round(f)) @ h.T


def _pair_sums(s, x, atom, y, ytype, yq, skip=None):
    """LJ and real-space charge energies of beads x with atoms y (skip[i, j]: pairs left out)."""
    eps, sig2, shift = s.lj_tables()
    t, q = s.molecule_types()[atom], s.molecule.charges()[atom]
    e, s2, sh = (_t(v[t[:, None], ytype[None, :]]) for v in (eps, sig2, shift))
    r2 = (_image(s, x[:, None, :] - y[None, :, :]) ** 2).sum(-1)
    inside = r2 < s.cutoff ** 2
    if skip is not None:
        inside &= ~skip
    w = (s2 / r2) ** 3
    zero = torch.zeros((), dtype=torch.float64, device=r2.device)
    lj = torch.where(inside, 4.0 * e * (w * (w - 1.0)) - sh, zero).sum(1)
    if not s.ewald:
        return lj, torch.zeros_like(lj)
    r = torch.sqrt(r2)
    qq = units.COULOMBIC_CONVERSION_FACTOR * _t(q)[:, None] * _t(yq)[None, :]
    return lj, torch.where(inside, qq * torch.erfc(s.alpha * r) / r, zero).sum(1)


def _bead_energies(s, mols, xyz, atom, excl):
    fw, ft, fq = s.framework()
    na = s.molecule.n_atoms
    x = _t(xyz)
    hv, hc = _pair_sums(s, x, atom, _t(fw), ft, fq)
    k = np.arange(len(mols) * na)
    skip = torch.as_tensor(np.asarray(excl)[:, None] == (k // na)[None, :], device=x.device)
    av, ac = _pair_sums(s, x, atom, _t(mols).reshape(-1, 3), s.molecule_types()[k % na], s.molecule.charges()[k % na],
                        skip)
    return torch.stack([hv, hc, av, ac], 1)


def _structure_factor(s, x, q):
    k = _t(systems.kvector_indices(s.kmax))
    a = 2.0 * math.pi * (x @ torch.linalg.inv(_t(s.box_matrix)).T) @ k.T
    return torch.complex((q[:, None] * torch.cos(a)).sum(0), (q[:, None] * torch.sin(a)).sum(0))


def _kfactor(s):
    n = _t(systems.kvector_indices(s.kmax))
    k2 = (2.0 * math.pi * n @ torch.linalg.inv(_t(s.box_matrix))).square().sum(1)
    pre = torch.where(n[:, 0] == 0, 2.0, 4.0).double() * math.pi / s.volume
    return units.COULOMBIC_CONVERSION_FACTOR * pre * torch.exp(-0.25 / s.alpha ** 2 * k2) / k2


def _exclusion(s, x):
    """Intramolecular K q q erf(alpha r) / r of molecules x[m, atoms, 3]."""
    q, e = s.molecule.charges(), 0.0
    for a, b in itertools.combinations(range(len(q)), 2):
        r = torch.linalg.norm(x[:, a] - x[:, b], dim=1)
        e = e + units.COULOMBIC_CONVERSION_FACTOR * q[a] * q[b] * torch.erf(s.alpha * r) / r
    return e.sum()


def _lj_grid(s, probe, npts, size, shift):
    """The LJ energy of the probe with the framework and its derivatives at the grid's points, scaled to the
    grid's cells, in 64 bits."""
    eps, sig2, sh = s.lj_tables()
    fw, ft, _ = s.framework()
    x = _grid_points(npts, size, shift)
    e, s2, u0 = (_t(v[probe, ft]) for v in (eps, sig2, sh))

    def terms(r2):
        w = (s2 / r2) ** 3
        return (4.0 * e * (w * (w - 1.0)) - u0, 24.0 * e * (w * (1.0 - 2.0 * w)) / r2,
                96.0 * e * (w * (7.0 * w - 2.0)) / r2 ** 2, 384.0 * e * (w * (5.0 - 28.0 * w)) / r2 ** 4)
    return _grid_values(s, x, _t(fw), terms, size / npts, 0.0).reshape(tuple(int(n) + 1 for n in npts) + (8,))


def _coulomb_grid(s, npts, size, shift):
    fw, _, fq = s.framework()
    kq, al = units.COULOMBIC_CONVERSION_FACTOR * _t(fq), s.alpha

    def terms(r2):
        r = torch.sqrt(r2)
        c, g, a2 = torch.erfc(al * r), 2.0 * al / math.sqrt(math.pi) * r * torch.exp(-al * al * r2), al * al * r2
        return (kq * c / r, -kq * (g + c) / (r * r2), kq * (g * (3.0 + 2.0 * a2) + 3.0 * c) / (r2 * r2 * r),
                -kq * (g * (15.0 + 10.0 * a2 + 4.0 * a2 * a2) + 15.0 * c) / (r2 ** 3 * r))
    x = _grid_points(npts, size, shift)
    return _grid_values(s, x, _t(fw), terms, size / npts, 1.0).reshape(tuple(int(n) + 1 for n in npts) + (8,))


def _grid_points(npts, size, shift):
    ax = [_t(np.arange(int(n) + 1) * l / int(n) + o) for n, l, o in zip(npts, size, shift)]
    return torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)


def _grid_values(s, x, y, terms, delta, closest):
    out = torch.empty((len(x), 8), dtype=torch.float64, device=x.device)
    zero = torch.zeros((), dtype=torch.float64, device=x.device)
    box = None if s.triclinic else _t(s.box)
    step = max(1, 40_000_000 // len(y))
    for i in range(0, len(x), step):
        d = x[i:i + step, None, :] - y[None, :, :]
        d = _image(s, d) if box is None else d - box * torch.round(d / box)
        dx, dy, dz = d.unbind(-1)
        r2 = dx * dx + dy * dy + dz * dz
        u, f1, f2, f3 = (torch.where(r2 < s.cutoff ** 2, v, zero) for v in terms(r2))
        o = torch.stack([u.sum(1)] + [(v * w).sum(1) for v, w in (
            (f1, dx), (f1, dy), (f1, dz), (f2, dx * dy), (f2, dx * dz), (f2, dy * dz), (f3, dx * dy * dz))], 1)
        big = o[:, 0] > units.ENERGY_OVERLAP_CRITERIA
        if closest:
            big = big | (r2.min(1).values < closest)
        cap = torch.cat([torch.full_like(o[:, :1], 2.0 * units.ENERGY_OVERLAP_CRITERIA),
                         o[:, 1:4].clamp(-units.ENERGY_OVERLAP_CRITERIA, units.ENERGY_OVERLAP_CRITERIA),
                         torch.zeros_like(o[:, 4:])], 1)
        out[i:i + step] = torch.where(big[:, None], cap, o)
    dx, dy, dz = (float(v) for v in delta)
    return out * _t([1.0, dx, dy, dz, dx * dy, dx * dz, dy * dz, dx * dy * dz])


def _hermite(t):
    return ((1 - 3 * t ** 2 + 2 * t ** 3, 3 * t ** 2 - 2 * t ** 3), (t - 2 * t ** 2 + t ** 3, t ** 3 - t ** 2))


def _lookup(grid, npts, size, shift, cell, xyz):
    x, c = _t(xyz), _t(cell)
    x = x - c * torch.trunc(x / c + torch.where(x / c >= 0, 0.5, -0.5))
    x = torch.where(x < 0, x + c, x)
    f = (x - _t(shift)) / _t(size) * _t(npts)
    n = torch.as_tensor(np.asarray(npts), device=x.device)
    i = torch.minimum(f.to(torch.int64).clamp(min=0), n - 1)
    h = _hermite(f - i)                       # h[derivative][corner][:, axis]
    val = torch.zeros(len(x), dtype=torch.float64, device=x.device)
    big = torch.zeros(len(x), dtype=torch.bool, device=x.device)
    order = {(0, 0, 0): 0, (1, 0, 0): 1, (0, 1, 0): 2, (0, 0, 1): 3, (1, 1, 0): 4, (1, 0, 1): 5, (0, 1, 1): 6,
             (1, 1, 1): 7}
    for cx, cy, cz in itertools.product((0, 1), repeat=3):
        v = grid[i[:, 0] + cx, i[:, 1] + cy, i[:, 2] + cz].double()
        big |= v[:, 0] > 1e10
        for (ox, oy, oz), k in order.items():
            val += v[:, k] * h[ox][cx][:, 0] * h[oy][cy][:, 1] * h[oz][cz][:, 2]
    return torch.where(big, torch.full_like(val, 1e8), val)


def exact(case, seed):
    kind = case["kind"]
    if kind == "points":
        return _bead_energies(*_points_input(case, seed)).cpu()
    if kind == "displace":
        s, mols, m, new = _displace_input(case, seed)
        na = s.molecule.n_atoms
        atom = np.tile(np.arange(na), 2)
        e = _bead_energies(s, mols, np.concatenate([new, mols[m]]), atom, np.full(2 * na, m))
        pair = e[:na].sum(0) - e[na:].sum(0)
        fw, _, fq = s.framework()
        sf = _structure_factor(s, _t(fw), _t(fq))
        sa = _structure_factor(s, _t(mols).reshape(-1, 3), _t(np.tile(s.molecule.charges(), len(mols))))
        q = _t(s.molecule.charges())
        ds = _structure_factor(s, _t(new), q) - _structure_factor(s, _t(mols[m]), q)
        kf = _kfactor(s)
        ads = (kf * (2.0 * (sa.conj() * ds).real + ds.abs() ** 2)).sum()
        ads = ads - (_exclusion(s, _t(new)[None]) - _exclusion(s, _t(mols[m])[None]))
        four = torch.stack([ads, 2.0 * (kf * (sf.conj() * ds).real).sum(), torch.zeros_like(ads)])
        return [dict(overlap=None, pair=sign * pair.cpu(), fourier=sign * four.cpu()) for sign in (1.0, -1.0)]
    if kind == "rescore":
        _, s, mols = _loaded(case, seed)
        na = s.molecule.n_atoms
        k = np.arange(len(mols) * na)
        parts = [_bead_energies(s, mols, mols.reshape(-1, 3)[c], c % na, c // na) for c in np.array_split(k, len(k) // 64 + 1)]
        hv, hc, av, ac = torch.cat(parts).sum(0)
        fw, _, fq = s.framework()
        sf = _structure_factor(s, _t(fw), _t(fq))
        q = s.molecule.charges()
        sa = _structure_factor(s, _t(mols).reshape(-1, 3), _t(np.tile(q, len(mols))))
        kf = _kfactor(s)
        uion = units.COULOMBIC_CONVERSION_FACTOR * s.alpha / math.sqrt(math.pi) - kf.sum()
        net = len(mols) * q.sum()
        own = units.COULOMBIC_CONVERSION_FACTOR * s.alpha / math.sqrt(math.pi) * (q ** 2).sum() * len(mols)
        af = (kf * sa.abs() ** 2).sum() - _exclusion(s, _t(mols)) - own + uion * net ** 2
        hf = 2.0 * (kf * (sf.conj() * sa).real).sum() + 2.0 * uion * fq.sum() * net
        return torch.stack([hv, 0.5 * av, hc, 0.5 * ac, hf, af]).cpu()
    if kind == "grid":
        s = _system(case, np.random.default_rng(seed))
        geom = _grid_geometry(case, s)
        return _coulomb_grid(s, *geom) if case["coulomb"] else _lj_grid(s, _probe(s), *geom)
    if kind == "lookup":
        st = prepare(case, seed)
        return _lookup(st["grid"], *st["geom"], st["xyz"]).cpu()
    return None     # a Markov chain of moves: no plain computation of it
