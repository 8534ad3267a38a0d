"""Per-call kernels at the sizes where their work split changes, against the
oracle: frameworks of one atom, one tile, a tile and an atom and more tiles
than warps; one position up to the largest call; few and many adsorbates;
orthorhombic and triclinic boxes.

FP64: within 1e-9 of the result (the per-call parity bound) plus 1e-12 of the
sum of the absolute pair terms (FP64 rounding of at most ~1e4 terms that
cancel). Mixed (accuracy: test_gpu_parity): the same bits for a position in
any call of five positions or more.
"""
import dataclasses

import numpy as np
import pytest

from oracle import oracle as O
from raspa2_b200 import native, systems

pytestmark = pytest.mark.gpu


def co2_box(atoms, tri):
    s = systems.co2_system(seed=5, n_atoms=atoms, cell=26.5, kmax=3, layout="uniform")
    if tri:
        s = dataclasses.replace(s, unit_cell=np.array([29.0, 28.0, 30.0]), cell_angles=(80.0, 95.0, 110.0))
    return s


def molecules(rng, s, n):
    u = rng.normal(size=(n, 1, 3))
    u /= np.linalg.norm(u, axis=2, keepdims=True)
    z = np.array([1.16, 0.0, -1.16])[None, :, None]
    return s.box_point(rng.random((n, 1, 3))) + z * u


@pytest.mark.parametrize("tri", [False, True])
@pytest.mark.parametrize("atoms,nmol,n", [(1, 0, 1), (16, 1, 2), (17, 11, 7), (300, 90, 9), (700, 3, 19), (1100, 40, 64),
                                          (33, 200, 33)])
def test_points_at_split_edges(cuda, atoms, nmol, n, tri):
    s = co2_box(atoms, tri)
    rng = np.random.default_rng(atoms + n)
    mols = molecules(rng, s, nmol)
    g = native.GpuSystem(s, maxmol=256)
    g.set_adsorbates(mols)
    o = O.Oracle.from_system(s, maxmol=256)
    o.set_molecules(mols)
    # positions in and around the box, some in their neighbouring images
    xyz = s.box_point(rng.uniform(-1.0, 2.0, (n, 3)))
    atom = rng.integers(0, 3, n)
    excl = rng.integers(-1, max(nmol, 1), n)
    t, q = s.molecule_types(), s.molecule.charges()
    ref = np.array([o.point(int(t[a]), float(q[a]), x, int(e)) for a, x, e in zip(atom, xyz, excl)])
    scale = np.array([o.point_abs(int(t[a]), float(q[a]), x, int(e)) for a, x, e in zip(atom, xyz, excl)])
    got = g.bead_energies(xyz, atom, excl, native.RGPU_FP64)
    assert np.all(np.abs(got - ref) <= 1e-9 * np.abs(ref) + 1e-12 * scale + 1e-8)
    # mixed: from five positions on a position's FP32 sums do not depend on the others of its call
    if n >= 10:
        got = g.bead_energies(xyz, atom, excl, native.RGPU_MIXED)
        h = n // 2
        parts = [g.bead_energies(xyz[k], atom[k], excl[k], native.RGPU_MIXED) for k in (slice(0, h), slice(h, n))]
        np.testing.assert_array_equal(got, np.concatenate(parts))


@pytest.mark.parametrize("tri", [False, True])
@pytest.mark.parametrize("atoms,nmol,kmax", [(1, 1, 1), (16, 5, 2), (40, 6, 6), (300, 43, 10), (96, 210, 4)])
def test_totals_and_fourier_at_split_edges(cuda, atoms, nmol, kmax, tri):
    """Total energies, Fourier differences (insertion, deletion, displacement), acceptance and molecule updates
    where the split over CTAs changes: fewer wave vectors than a block and more than a cluster's, fewer atoms than
    a phase table and more, one position to more positions than CTAs. FP64 bounds as above; the sums of absolute
    terms are those of the oracle."""
    s = dataclasses.replace(co2_box(atoms, tri), kmax=(kmax, kmax, kmax))
    rng = np.random.default_rng(atoms + nmol + kmax)
    mols = molecules(rng, s, nmol + 1)
    mols, extra = mols[:-1], mols[-1]
    g = native.GpuSystem(s, maxmol=256)
    g.set_adsorbates(mols)
    o = O.Oracle.from_system(s, maxmol=256)

    def totals(x):
        o.set_molecules(x)
        ref = np.array(o.total_energy())[:6]
        t, q = s.molecule_types(), s.molecule.charges()
        pair = sum(o.point_abs(int(t[a]), float(q[a]), m[a], i) for i, m in enumerate(x) for a in range(3))
        e = np.asarray(g.total_energy())
        scale = np.array([pair[0], pair[2], pair[1], pair[3], 0.0, 0.0])
        scale[4:] = np.abs(np.array(o.ewald_delta_abs(new=extra)))[:2].max() * (len(x) + 1) ** 2
        assert np.all(np.abs(e - ref) <= 1e-9 * np.abs(ref) + 1e-12 * scale + 1e-7), (e, ref)

    totals(mols)
    new = mols[0] + rng.uniform(-0.3, 0.3, 3)
    for old, x in ((-1, extra), (nmol - 1, None), (0, new)):
        got = g.ewald_difference(old, x)
        prev = None if old < 0 else mols[old]
        ref, size = np.array(o.ewald_delta(old=prev, new=x)[0]), np.abs(np.array(o.ewald_delta_abs(old=prev, new=x)))
        assert np.all(np.abs(got[:2] - ref[:2]) <= 1e-9 * np.abs(ref[:2]) + 1e-12 * size[:2].max() + 1e-8)
    g.ewald_accept()                       # the displacement
    g.update_molecule(0, new)
    moved = mols.copy()
    moved[0] = new
    np.testing.assert_array_equal(g.adsorbates(), moved)
    o.set_molecules(moved)
    got, ref = g.ewald_difference(-1, extra), np.array(o.ewald_delta(new=extra)[0])
    size = np.abs(np.array(o.ewald_delta_abs(new=extra)))[:2].max()
    assert np.all(np.abs(got[:2] - ref[:2]) <= 1e-9 * np.abs(ref[:2]) + 1e-12 * size + 1e-8)
    g.insert_molecule(extra)
    totals(np.concatenate([moved, extra[None]]))
    g.remove_molecule(0)
    totals(np.concatenate([extra[None], moved[1:]]))


@pytest.mark.parametrize("atoms", [128, 4800])
def test_mixed_lists_and_their_overflow(cuda, atoms):
    """The mixed kernel's pair lists from a tile per warp on, and a framework so dense (0.34 atoms per cubic
    Angstrom) that a warp's list overflows and one warp walks the tiles. Random atoms overlap the beads, so the bound
    is the sensitivity of FP32 distances: r^2 within 3e-7 (three rounded products, coordinates of 2e-8 A at
    r > 0.3 A), 6 times that for r^-12, some 5 roundings of the term and its sum: 5e-6 of the absolute terms."""
    s = co2_box(16, False)
    rng = np.random.default_rng(atoms)
    s = dataclasses.replace(s, unit_cell=np.array([24.1, 24.1, 24.1]), frac=np.round(rng.random((atoms, 3)), 12),
                            uc_types=["Sifw"] * (atoms // 2) + ["Ofw"] * (atoms - atoms // 2),
                            uc_charges=np.round(rng.uniform(-1, 1, atoms), 8))
    g = native.GpuSystem(s, maxmol=4)
    o = O.Oracle.from_system(s, maxmol=4)
    xyz, atom = rng.uniform(0.0, 24.1, (9, 3)), rng.integers(0, 3, 9)
    t, q = s.molecule_types(), s.molecule.charges()
    scale = np.array([o.point_abs(int(t[a]), float(q[a]), x, -1) for a, x in zip(atom, xyz)])
    ref, got = (g.bead_energies(xyz, atom, -1, p) for p in (native.RGPU_FP64, native.RGPU_MIXED))
    near = np.max(np.abs(ref), axis=1) < 1e15      # a pair within about 0.3 A gives more
    assert near.sum() >= 3
    assert np.all(np.abs(got - ref)[near] <= 5e-6 * scale[near] + 1e-6)


@pytest.mark.parametrize("tri", [False, True])
def test_energies_after_a_batched_upload(cuda, tri):
    """A batched upload leaves the records that per-call energies read: the same bits as after uploads system by
    system, for no molecule, one, and more atoms than a block has threads."""
    s = co2_box(96, tri)
    rng = np.random.default_rng(7)
    counts = [0, 1, 86, 200]
    mols = [molecules(rng, s, n) for n in counts]
    xyz = s.box_point(rng.random((24, 3)))
    atom, excl = rng.integers(0, 3, 24), np.full(24, -1)
    got = []
    for batched in (False, True):
        gs = [native.GpuSystem(s, maxmol=256, stream_id=i) for i in range(len(counts))]
        e = native.Engine(gs, precision=native.RGPU_MIXED, threads=256, cluster=2)
        if batched:
            for g in gs:
                g.set_adsorbates(molecules(rng, s, 40))
            e.set_adsorbates(mols)
        else:
            for g, x in zip(gs, mols):
                g.set_adsorbates(x)
        got.append([g.bead_energies(xyz, atom, excl, p) for g in gs for p in (native.RGPU_FP64, native.RGPU_MIXED)])
    np.testing.assert_array_equal(np.array(got[0]), np.array(got[1]))


@pytest.mark.parametrize("tri", [False, True])
def test_bead_on_a_charged_framework_atom(cuda, tri):
    """A bead exactly on a framework atom: the real-space charge energy is infinite with the sign of the charges'
    product, and a molecule on a like charge overlaps, also where the atom's type has no LJ (its LJ term, zero
    times infinity, is NaN)."""
    s = co2_box(16, tri)
    rng = np.random.default_rng(3)
    q = np.round(rng.uniform(0.2, 1.0, 16), 8) * np.where(np.arange(16) % 4 < 2, 1.0, -1.0)
    s = dataclasses.replace(s, uc_types=["Sifw", "Dummy"] * 8, uc_charges=q - q.mean())
    pos, _, fq = s.framework()
    n = len(pos)
    lj = np.array(s.uc_types)[:n] == "Sifw"
    g = native.GpuSystem(s, maxmol=4)
    atom = rng.integers(0, 3, n)
    got = g.bead_energies(pos, atom, -1)
    np.testing.assert_array_equal(got[:, 1], np.inf * np.sign(s.molecule.charges()[atom] * fq))
    np.testing.assert_array_equal(got[lj, 0], np.inf)
    # a molecule whose carbon (charge +0.7) sits on an atom, its oxygens on none
    far = s.box_point(np.array([[0.5, 0.5, 0.5]])) + s.molecule.positions
    g.set_adsorbates(far[None])
    for k in range(n):
        overlap, _ = g.move_difference(0, pos[k] + s.molecule.positions - s.molecule.positions[1])
        assert overlap == (bool(lj[k]) or fq[k] > 0), k


@pytest.mark.parametrize("charged", [False, True])
def test_fp64_lj_rounding(cuda, charged):
    """LJ of one pair at exactly representable distances against extended precision. With one rounded quotient
    sigma^2 / r^2 the r^-12 term collects at most 13 units of u = 2^-53 (6 from the quotient, 2 + 2 from the products
    of s^6, 3 from the rest) and, roundings being independent with an rms of 0.43 u, 2.9 u rms; one more rounding of
    1 / r^2 makes that 3.9 u, so 3.3 u tells them apart (4096 pairs give it to 2 %)."""
    s = co2_box(16, False)
    s = dataclasses.replace(s, unit_cell=np.array([32.0, 32.0, 32.0]), frac=np.full((1, 3), 0.25), uc_types=["Sifw"],
                            uc_charges=np.array([0.5 if charged else 0.0]))
    g = native.GpuSystem(s, maxmol=4)
    rng = np.random.default_rng(11)
    d = rng.normal(size=(4096, 3))
    d *= rng.uniform(0.8, 1.6, (4096, 1)) / np.linalg.norm(d, axis=1, keepdims=True)
    d = np.round(d * 4096) / 4096          # r^2 is exact
    got = g.bead_energies(8.0 + d, 0, -1)[:, 0].astype(np.longdouble)
    eps, sig2, shift = (t[s.molecule_types()[0], systems.TYPE_ORDER.index("Sifw")] for t in s.lj_tables())
    s6 = (np.longdouble(sig2) / np.sum(d.astype(np.longdouble) ** 2, axis=1)) ** 3
    ref = 4 * np.longdouble(eps) * (s6 * (s6 - 1)) - np.longdouble(shift)
    err = (got - ref) / ref * 2.0 ** 53
    assert np.max(np.abs(err)) <= 13 * 1.05          # s^6 >= 21: (2 s^6 - 1) / (s^6 - 1) is within 5 % of 2
    assert np.sqrt(np.mean(err ** 2)) <= 3.3


def test_total_energy_with_the_most_wave_vectors(cuda):
    """kmax 20, the largest accepted: 20004 wave vectors in 79 of the 128 blocks that a call's results have room
    for (the bounds of the totals above)."""
    s = dataclasses.replace(co2_box(16, False), kmax=(20, 20, 20))
    assert s.n_kvectors() == 20004 <= 128 * 256
    rng = np.random.default_rng(20)
    mols = molecules(rng, s, 12)
    g = native.GpuSystem(s, maxmol=16)
    g.set_adsorbates(mols)
    o = O.Oracle.from_system(s, maxmol=16)
    o.set_molecules(mols)
    ref, e = np.array(o.total_energy())[:6], np.asarray(g.total_energy())
    size = np.abs(np.array(o.ewald_delta_abs(new=mols[0])))[:2].max() * 13 ** 2
    assert np.all(np.abs(e - ref)[4:] <= 1e-9 * np.abs(ref[4:]) + 1e-12 * size + 1e-7), (e, ref)
