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
            assert np.array_equal(lookup(x), x[:, 0])
            fake.fake_reset()
        assert value("fake_stray").value == 0
    """)
