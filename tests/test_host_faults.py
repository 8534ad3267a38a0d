"""Host code of the library on a CUDA runtime without a device (fake/cudart.c, preloaded into a child process):
failing calls, a device reset, index ranges. No kernel runs, so nothing here is about their results."""
import os
import shutil
import subprocess
import sys
import textwrap

import pytest

from raspa2_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    gcc = shutil.which("gcc")
    home = os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))) if gcc else None
    if not home or not os.path.exists(os.path.join(home, "include", "cuda_runtime.h")):
        pytest.skip("no C compiler or CUDA headers")
    so = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    subprocess.check_call([gcc, "-O2", "-shared", "-fPIC", "-I" + os.path.join(home, "include"), "-o", so,
                           os.path.join(HERE, "fake", "cudart.c")])
    return so


PRELUDE = """
import ctypes as C
import numpy as np
from raspa2_b200 import native, systems
fake = C.CDLL(None)
value = lambda name: C.c_int.in_dll(fake, name)
cell = np.array([20.0, 20.0, 20.0])
grid = np.zeros(2 ** 3 * 8 + 4, np.float32)
d_grid = grid.ctypes.data + -grid.ctypes.data % 16
lookup = lambda x: native.grid_interpolate(d_grid, [1, 1, 1], cell, np.zeros(3), cell, x)
"""


def child(fake, code):
    env = dict(os.environ, LD_PRELOAD=fake, PYTHONPATH=ROOT)
    p = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(code)], cwd=ROOT, env=env, capture_output=True,
                       text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr


def test_lookup_after_a_device_reset(fake):
    """The staging memory of grid lookups is not mapped any more after cudaDeviceReset: the next lookup maps it
    again, and no kernel is given an address that is not mapped."""
    child(fake, """
        value("fake_lookup").value = 1
        x = np.arange(3 * 20000.0).reshape(-1, 3)
        for _ in range(3):
            assert np.array_equal(lookup(x), x[:, 0] + 1.0)
            fake.fake_reset()
        assert value("fake_stray").value == 0
    """)


def test_lookup_of_as_many_points_as_an_int_counts(fake):
    """2^31 - 1 positions, the largest count the call takes: every chunk is looked up once and none after the last.
    The arrays are addresses (51 and 17 GB) over a page of zeros and a block of 2^21 results."""
    child(fake, """
        import os
        libc = C.CDLL(None, use_errno=True)
        libc.mmap.restype = C.c_void_p
        libc.mmap.argtypes = [C.c_void_p, C.c_size_t, C.c_int, C.c_int, C.c_int, C.c_long]
        libc.madvise.argtypes = [C.c_void_p, C.c_size_t, C.c_int]
        def addresses(size, prot):                     # private, anonymous, no reserve
            at = libc.mmap(None, size, prot, 0x4022, -1, 0)
            assert at != C.c_void_p(-1).value
            return at
        n, k = 2 ** 31 - 1, 2 ** 21
        x = addresses(24 * 2 ** 31, 1)
        libc.madvise(x, 24 * 2 ** 31, 14)              # the large page of zeros, where there is one
        out = addresses(8 * 2 ** 31, 0)
        fd = os.memfd_create("results")
        os.ftruncate(fd, 8 * k)
        for o in range(0, 8 * 2 ** 31, 8 * k):
            assert libc.mmap(out + o, 8 * k, 3, 0x11, fd, 0) == out + o    # shared, fixed
        value("fake_lookup").value = 1
        size, npts, zero = (C.c_double * 3)(*cell), (C.c_int * 3)(1, 1, 1), (C.c_double * 3)()
        rc = native.load().rgpu_grid_interpolate(C.c_void_p(d_grid), npts, size, zero, size, C.c_int(n), C.c_void_p(x),
                                                 C.c_void_p(out))
        assert rc == 0 and value("fake_stray").value == 0
        assert value("fake_launches").value == 2 ** 31 // 16384
        assert np.array_equal(np.ctypeslib.as_array(C.cast(out, C.POINTER(C.c_double)), (k,)), np.ones(k))
    """)


def test_footprint_is_what_a_system_allocates(fake):
    """The serving front end's estimate of a job's device memory covers what rgpu_system_create and the engine's
    descriptor take, and is not much above it."""
    child(fake, """
        import dataclasses
        from raspa2_b200 import serve
        co2 = systems.co2_system(seed=21, n_atoms=1536, cell=25.8, kmax=8, layout="uniform")
        for s, maxmol in ((systems.tiny_co2_system(), 8), (co2, 64), (co2, 512), (systems.methane_system(seed=3), 512),
                          (dataclasses.replace(co2, unit_cells=np.array([3, 2, 2])), 100),
                          (dataclasses.replace(systems.tiny_co2_system(), cell_angles=(80.0, 95.0, 100.0),
                                               unit_cell=np.array([29.0, 28.0, 30.0])), 20)):
            n = C.c_longlong.in_dll(fake, "fake_device_bytes")
            n.value = 0
            g = native.GpuSystem(s, maxmol=maxmol)
            e = native.Engine([g], threads=256, cluster=1)
            got = serve.system_footprint_bytes(s, maxmol)
            assert n.value <= got <= 1.05 * n.value + 16384, (s.name, n.value, got)
    """)


def test_empty_configurations_launch_no_kernel(fake):
    """No molecule: an upload is two memsets, and an uncharged system's total energy neither launches nor waits."""
    child(fake, """
        for s in (systems.tiny_co2_system(), systems.methane_system(seed=3)):
            g = native.GpuSystem(s, maxmol=8)
            na = s.molecule.n_atoms
            g.set_adsorbates(np.ones((3, na, 3)))
            n = value("fake_launches").value
            g.set_adsorbates(np.zeros((0, na, 3)))
            assert value("fake_launches").value == n
            syncs = value("fake_syncs").value
            g.total_energy()
            assert s.ewald or (value("fake_launches").value, value("fake_syncs").value) == (n, syncs)
    """)


def test_failed_molecule_updates_change_nothing(fake):
    """Where the launch that writes a molecule to the device fails, the host's copy of the configuration stays as the
    device's."""
    child(fake, """
        s = systems.tiny_co2_system()
        g = native.GpuSystem(s, maxmol=8)
        x = np.random.default_rng(1).uniform(0.0, 20.0, (5, 3, 3))
        g.set_adsorbates(x)
        value("fake_fail_launch").value = 1
        for call in (lambda: g.insert_molecule(x[0] + 1.0), lambda: g.remove_molecule(1), lambda: g.remove_molecule(4),
                     lambda: g.update_molecule(2, x[2] + 1.0)):
            try:
                call()
            except native.NativeError:
                pass
            else:
                assert False, "no error"
            assert np.array_equal(g.adsorbates(), x)
        value("fake_fail_launch").value = 0
        g.insert_molecule(x[0] + 1.0)
        g.update_molecule(2, x[2] + 1.0)
        g.remove_molecule(1)
        g.remove_molecule(4)
        assert np.array_equal(g.adsorbates(), np.stack([x[0], x[0] + 1.0, x[2] + 1.0, x[3]]))
    """)
