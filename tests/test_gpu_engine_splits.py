"""Chains in CTAs of three to sixteen warps, where the warps that work beside a growth's choice take their parts
together or one each: the FP64 engine follows the oracle's trajectory move for move (the bounds of the same
comparison at 64 and 256 threads: FP64 rounding over the trajectory)."""
import numpy as np
import pytest

from oracle import oracle as O
from raspa2_b200 import native, systems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [96, 128, 160, 192, 512])
def test_chain_growth_at_warp_counts(cuda, threads):
    s = systems.hexane_system(seed=4, n_atoms=1200, cell=26.0, pressure=1e6)
    n = 400
    g = native.GpuSystem(s, maxmol=64, seed=777, stream_id=5)
    g.set_adsorbates(np.zeros((0, 6, 3)))
    e = native.Engine([g], precision=native.RGPU_FP64, threads=threads, cluster=2)
    e.run(n)
    e.sync()
    st = g.state()
    o = O.Oracle.from_system(s, maxmol=64)
    o.set_molecules(np.zeros((0, 6, 3)))
    ost = O.MCState()
    o.mc_run(O.mc_params(s, 777, 5), ost, 0, n)
    assert st["status"] == 0
    np.testing.assert_array_equal(st["counters"][0:4], np.array(ost.attempts[:4]))
    np.testing.assert_array_equal(st["counters"][4:8], np.array(ost.accepted[:4]))
    assert st["counters"][18] == ost.attempts[4] and st["counters"][19] == ost.accepted[4]
    assert st["nmol"] == o.nmol
    np.testing.assert_allclose(g.adsorbates(), o.molecules(), rtol=0, atol=1e-9)
    np.testing.assert_allclose(st["energy"][6], ost.u_intra, rtol=1e-9, atol=1e-6)
