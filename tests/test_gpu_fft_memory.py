"""A full recompute whose temporary does not fit: 'auto' sums directly, 'fft64' says so."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('kind', ['OOP_Square', 'IP_Pinwheel'])
def test_auto_falls_back_to_the_direct_sum(kind, monkeypatch):
    import hotspice_b200 as hs
    g = np.random.default_rng(2)
    mm = getattr(hs.ASI, kind)(300e-9, nx=60, ny=50, T=300, E_B=2e-20, moment=1e-15, seed=2,
                               pattern=g.integers(0, 2, size=(50, 60)) * 2 - 1, energies=[hs.DipolarEnergy()])
    d = mm.get_energy('dipolar')

    def energies():
        return d.E.clone(), d.E_perp.clone() if mm.in_plane else d.E.clone()

    d.update(method='direct64')
    direct = energies()
    d.update()
    by_fft = energies()
    assert not bool((by_fft[0] == direct[0]).all())          # 'auto' takes the convolution here
    nbytes = mm._lib.hs_fft_scratch_bytes(mm._lattice_struct())
    empty = torch.empty

    def short(*size, **kw):
        if size == (nbytes,):
            raise torch.cuda.OutOfMemoryError('no memory for the temporary')
        return empty(*size, **kw)

    monkeypatch.setattr(torch, 'empty', short)
    d._E.zero_()
    d.update()
    for a, b in zip(energies(), direct):
        assert bool((a == b).all())
    with pytest.raises(torch.cuda.OutOfMemoryError):
        d.update(method='fft64')
