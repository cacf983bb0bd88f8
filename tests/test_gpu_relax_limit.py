"""A grid barrier of relax() that runs out of time: the call raises, leaves the spins it reached with
their energies, and the object relaxes as before afterwards."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('exchange', [False, True])
def test_relax_wait_limit_runs_out_cleanly(exchange):
    import hotspice_b200 as hs
    from hotspice_b200 import _lib
    lib = _lib.load()
    g = np.random.default_rng(3)
    nx, ny = 260, 200

    def lattice(pattern):
        energies = [hs.DipolarEnergy(cutoff_range=8.3 * 300e-9), hs.ZeemanEnergy(2e-4, 0.3)]
        if exchange:
            energies.append(hs.ExchangeEnergy(J=2e-21))
        return hs.ASI.IP_Pinwheel(300e-9, nx=nx, ny=ny, T=300, E_B=2e-20, moment=1e-15, seed=21, energies=energies,
                                  pattern=pattern)

    mm = lattice(g.integers(0, 2, size=(ny, nx)) * 2 - 1)
    try:
        assert lib.hs_set_wait_limit(1) == _lib.HS_OK
        with pytest.raises(RuntimeError, match='ran out of time'):
            mm.relax()
    finally:
        lib.hs_set_wait_limit(0)
    torch.cuda.synchronize()
    assert mm.status == 0
    dip = mm.get_energy('dipolar')
    E, Ep = dip.E.clone(), dip.E_perp.clone()
    assert bool((mm._mm_dev == mm._m_dev * mm._mom_dev).all())
    mm.update_energy()
    assert bool((dip.E == E).all()) and bool((dip.E_perp == Ep).all())
    twin = lattice(mm.m.cpu().numpy())            # a new object in the same state
    twin._write_counters(rng_call=int(mm._read_counters()['rng_call']))
    mm.relax()
    twin.relax()
    assert mm.relax_sweeps == twin.relax_sweeps > 0 and mm.status == 0
    assert bool((mm.m == twin.m).all()) and bool((mm.E == twin.E).all())
