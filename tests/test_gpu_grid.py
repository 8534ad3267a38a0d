"""GPU energy-grid construction and tricubic lookup against the reference's
grid file and InterpolateVDWGrid values (tests/golden/grid_methane.json)."""
import numpy as np
import pytest

from oracle import oracle as O
from raspa2_b200 import native, systems

from golden_cases import load, system_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def grid(cuda):
    import torch
    c = load("grid_methane")
    s = system_of(c)
    g = native.GpuSystem(s, maxmol=4)
    m = c["meta"]
    n = np.array(m["n"])
    buf = torch.zeros(int(np.prod(n + 1)) * 8, dtype=torch.float32, device="cuda")
    t = systems.TYPE_ORDER.index("CH4_sp3")
    g.grid_build(t, n, m["size"], m["shift"], buf.data_ptr())
    torch.cuda.synchronize()
    host = buf.cpu().numpy().reshape(n[0] + 1, n[1] + 1, n[2] + 1, 8)
    return c, s, g, buf, host


def test_grid_matches_reference_file(grid):
    c, s, g, buf, host = grid
    planes = np.moveaxis(host, 3, 0).reshape(8, -1)      # device point-major -> file plane-major
    got = planes[:, np.array(c["sample_index"])].T
    np.testing.assert_allclose(got, np.array(c["sample_values"]), rtol=2e-7, atol=1e-6)
    sums = [float(np.sum(planes[k].astype(np.float64))) for k in range(8)]
    np.testing.assert_allclose(sums, c["plane_sums"], rtol=1e-6)


def test_grid_matches_oracle(grid):
    c, s, g, buf, host = grid
    m = c["meta"]
    o = O.Oracle.from_system(s)
    t = systems.TYPE_ORDER.index("CH4_sp3")
    ref = o.grid_build(t, m["n"], m["size"], m["shift"])
    np.testing.assert_allclose(np.moveaxis(host, 3, 0), ref, rtol=2e-7, atol=1e-5)


def test_interpolation_matches_oracle_on_same_grid(grid):
    """GPU lookup = oracle lookup on the identical (GPU-built) grid."""
    c, s, g, buf, host = grid
    m = c["meta"]
    pts = np.array(c["interp_points"])
    got = native.grid_interpolate(buf.data_ptr(), m["n"], m["size"], m["shift"], m["cell"], pts)
    planes = np.ascontiguousarray(np.moveaxis(host, 3, 0))
    ref = [O.grid_interpolate(planes, m["n"], m["size"], m["shift"], m["cell"], p) for p in pts]
    np.testing.assert_allclose(got, ref, rtol=1e-12, atol=1e-9)


def test_interpolation_matches_reference(grid):
    """Against InterpolateVDWGrid on the reference's own grid file. The two
    grids agree to FP32 rounding (framework summation order differs), and the
    Hermite sum of a cell near the repulsive wall cancels by up to ~100x, so
    the bound is 2e-5 relative (1e-6 absolute floor)."""
    c, s, g, buf, host = grid
    m = c["meta"]
    pts = np.array(c["interp_points"])
    got = native.grid_interpolate(buf.data_ptr(), m["n"], m["size"], m["shift"], m["cell"], pts)
    np.testing.assert_allclose(got, c["interp_ref"], rtol=2e-5, atol=1e-6)


@pytest.mark.parametrize("tri", [False, True])
@pytest.mark.parametrize("npts,coulomb", [((1, 1, 1), False), ((3, 9, 17), False), ((24, 5, 31), True), ((15, 40, 23), False),
                                          ((2, 3, 2), True)])
def test_grid_build_paths_match_oracle(cuda, npts, coulomb, tri):
    """Grids from one cell to fine ones, over staged images and (tile radius beyond the box's reach) over minimum
    images, in the smallest box the cut-off allows, against the oracle's derivatives at every point: FP32 storage
    (6e-8 relative of a value; twice for the products with the FP32 spacings), and where terms cancel 1e-6 of an
    internal energy unit plus 1e-13 of the plane's largest value (FP64 rounding of its terms)."""
    import dataclasses
    import torch
    s = systems.co2_system(seed=9, n_atoms=150, cell=24.0001, kmax=3, layout="uniform")
    size, shift = np.array([24.0001] * 3), np.zeros(3)
    if tri:
        s = dataclasses.replace(s, unit_cell=np.array([26.5, 26.4, 25.0]), cell_angles=(80.0, 95.0, 110.0))
        m = s.unit_cell_matrix
        size, shift = np.abs(m).sum(axis=1), np.minimum(m, 0.0).sum(axis=1)
    g = native.GpuSystem(s, maxmol=4)
    o = O.Oracle.from_system(s, maxmol=4)
    n = np.array(npts, np.int32)
    buf = torch.zeros(int(np.prod(n + 1)) * 8, dtype=torch.float32, device="cuda")
    t = systems.TYPE_ORDER.index("O_co2")
    if coulomb:
        g.grid_build_coulomb(n, size, shift, buf.data_ptr())
        ref = o.grid_build_coulomb(n, size, shift)
    else:
        g.grid_build(t, n, size, shift, buf.data_ptr())
        ref = o.grid_build(t, n, size, shift)
    torch.cuda.synchronize()
    got = np.moveaxis(buf.cpu().numpy().reshape(tuple(n + 1) + (8,)), 3, 0).reshape(8, -1).astype(np.float64)
    ref = np.asarray(ref, np.float64).reshape(8, -1)
    top = np.abs(ref).max(axis=1, keepdims=True)
    assert np.all(np.abs(got - ref) <= 2e-7 * np.abs(ref) + 1e-6 + 1e-13 * top)


@pytest.mark.parametrize("n", [1, 255, 257, 16384, 16385, 131073])
def test_interpolate_across_stage_edges(cuda, n):
    """Lookups of one point, of blocks, staging chunks and the whole stage and one point more, from several threads
    at once (one of them finds the stage in use), against single lookups through the static scratch: the same
    kernel on the same values, so the same bits."""
    import threading
    import torch
    rng = np.random.default_rng(n)
    npts, size, shift = np.array([7, 9, 11], np.int32), np.array([10.0, 11.0, 12.0]), np.zeros(3)
    grid = torch.rand(8 * 10 * 12 * 8, device="cuda")
    xyz = rng.uniform(-20.0, 30.0, (n, 3))
    got = [None] * 3

    def look(i):
        got[i] = native.grid_interpolate(grid.data_ptr(), npts, size, shift, size, xyz)
    torch.cuda.synchronize()
    threads = [threading.Thread(target=look, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    ref = np.concatenate([native.grid_interpolate_noalloc(grid.data_ptr(), npts, size, shift, size, xyz[i:i + 8192])
                          for i in range(0, n, 8192)])
    for g in got:
        np.testing.assert_array_equal(g, ref)


@pytest.mark.parametrize("cell", [10.0, 13.7])
def test_lookups_at_half_cells(cuda, cell):
    """Points at multiples of half a cell and next to them, where the nearest image is a tie: the value at the
    wrapped point, which is in the cell already (within the rounding of the wrap, a few ulp of 4 cells, times the
    slopes of a random grid of a dozen points a side)."""
    import torch
    npts, size, shift = np.array([7, 9, 11], np.int32), np.full(3, cell), np.zeros(3)
    g = torch.rand(8, 10, 12, 8, device="cuda")
    g[-1], g[:, -1], g[:, :, -1] = g[0], g[:, 0], g[:, :, 0]    # periodic: a point may round onto either face
    g[-1] = g[0]
    grid = g.contiguous()
    half = np.concatenate([np.arange(-8, 9) * (0.5 * cell), np.nextafter(np.arange(-8, 9) * (0.5 * cell), 0.0)])
    xyz = np.stack(np.meshgrid(half, half, half[::3]), -1).reshape(-1, 3)
    n = np.trunc(xyz / cell + np.where(xyz >= 0.0, 0.5, -0.5))
    wrapped = xyz - cell * n
    wrapped = np.where(wrapped < 0.0, wrapped + cell, wrapped)
    torch.cuda.synchronize()
    look = [native.grid_interpolate(grid.data_ptr(), npts, size, shift, size, x) for x in (xyz, wrapped)]
    scale = np.abs(look[1]).max()
    assert np.all(np.abs(look[0] - look[1]) <= 1e-12 * scale)


def test_lookup_after_a_device_reset(cuda):
    """Lookups in a process of their own, before and after cudaDeviceReset (which undoes the mapping of the staging
    memory): the same bits, and those of this process."""
    import os
    import subprocess
    import sys
    code = """
import ctypes as C, sys
import numpy as np
from raspa2_b200 import native
rt = C.CDLL("libcudart.so.12")
native.load()
rng = np.random.default_rng(5)
grid = rng.normal(size=9 * 8 * 7 * 8).astype(np.float32)
xyz = rng.uniform(-9.0, 20.0, (40000, 3))
def lookup():
    d = C.c_void_p()
    assert rt.cudaMalloc(C.byref(d), C.c_size_t(grid.nbytes)) == 0
    assert rt.cudaMemcpy(d, grid.ctypes.data_as(C.c_void_p), C.c_size_t(grid.nbytes), 1) == 0
    size = np.array([10.0, 9.0, 8.0])
    return native.grid_interpolate(d.value, [8, 7, 6], size, np.zeros(3), size, xyz)
a = lookup()
assert np.array_equal(lookup(), a)
for _ in range(2):
    assert rt.cudaDeviceReset() == 0
    assert np.array_equal(lookup(), a)
np.save(sys.argv[1], a)
"""
    import tempfile

    import torch
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    with tempfile.TemporaryDirectory() as tmp:
        f = os.path.join(tmp, "a.npy")
        p = subprocess.run([sys.executable, "-c", code, f], cwd=root, capture_output=True, text=True, timeout=120,
                           env=dict(os.environ, PYTHONPATH=root))
        assert p.returncode == 0, p.stdout + p.stderr
        a = np.load(f)
    rng = np.random.default_rng(5)
    grid = torch.from_numpy(rng.normal(size=9 * 8 * 7 * 8).astype(np.float32)).cuda()
    size = np.array([10.0, 9.0, 8.0])
    got = native.grid_interpolate(grid.data_ptr(), [8, 7, 6], size, np.zeros(3), size, rng.uniform(-9.0, 20.0, (40000, 3)))
    np.testing.assert_array_equal(got, a)
