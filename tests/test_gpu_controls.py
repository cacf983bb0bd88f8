"""The run controls of a batch: set by one launch for many instances, by small copies for one or
two; either way every instance starts from progress = 0, done = 0 and the given t_max."""
import pytest

import hotspice_b200 as hs
from hotspice_b200.engine import BatchEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 128, 129])
def test_stale_controls_are_reset(n):
    mags = [hs.ASI.IP_Square(1e-6, 9, T=300, E_B=1e-19, seed=5 + i) for i in range(n)]
    for i, mm in enumerate(mags):
        mm.params.UPDATE_SCHEME = hs.Scheme.NEEL
        if i != n - 1 or n == 1:      # one instance may be up to date
            mm._write_counters(progress=7, done=1, t_max=1e-30)
    eng = BatchEngine(mags)
    n0 = [mm.attempted_switches for mm in mags]
    eng.run(3, t_max=float('inf'))
    for mm, a in zip(mags, n0):
        assert mm.attempted_switches == a + 3
    eng.run(3, t_max=2.5)
    assert all(float(mm._read_counters()['t_max']) == 2.5 for mm in mags)
