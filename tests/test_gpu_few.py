"""The update of short switch lists (dip_update_few_kernel) against the per-tile kernel, which the same
list takes when its capacity is large, bit for bit: windows that are disjoint, overlap, meet the edges,
wrap, are truncated, exact and mixed in one list, one switch and the longest short list."""
import ctypes
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _lattice(kind, nx, ny, cut, PBC):
    import hotspice_b200 as hs
    cls, a = {'oop': (hs.ASI.OOP_Square, 200e-9), 'pin': (hs.ASI.IP_Pinwheel, 300e-9)}[kind]
    g = np.random.default_rng(nx + ny)
    return cls(a, nx=nx, ny=ny, T=300, E_B=5e-20, moment=1e-15 * g.uniform(0.5, 1.5, size=(ny, nx)), PBC=PBC, seed=4,
               pattern=g.integers(0, 2, size=(ny, nx)) * 2 - 1,
               energies=[hs.DipolarEnergy(cutoff_range=cut * a if cut else math.inf)])


@pytest.mark.parametrize('n', [1, 2, 33, 64])
@pytest.mark.parametrize('kind,nx,ny,cut,PBC', [
    ('oop', 150, 131, 9, False), ('oop', 97, 64, 30, True), ('pin', 130, 94, 8.3, True), ('pin', 200, 111, 16, False),
    ('oop', 40, 30, 0, False), ('oop', 36, 30, 0, True),
])
@pytest.mark.parametrize('semantics', [0, 1])
def test_short_list_equals_long_list_kernel(kind, nx, ny, cut, PBC, n, semantics):
    from hotspice_b200 import _lib
    mm = _lattice(kind, nx, ny, cut, PBC)
    d = mm._dipolar()
    g = np.random.default_rng(n)
    occ = np.flatnonzero(mm.occupation)
    cells = g.choice(occ, size=min(n, occ.size), replace=False)
    n = cells.size
    E0, P0 = d._E.clone(), d._Ep.clone() if d._Ep is not None else None
    out = []
    for cap in (64, 5000):         # 64: the short-list kernel; 5000: the per-tile kernel
        d._E.copy_(E0)
        if P0 is not None:
            d._Ep.copy_(P0)
        t = torch.zeros((3, cap), device=mm.device, dtype=torch.int32)
        t[0, :n] = torch.as_tensor(cells // nx, dtype=torch.int32)
        t[1, :n] = torch.as_tensor(cells % nx, dtype=torch.int32)
        t[2, :n] = torch.as_tensor(g.integers(0, 2, size=n) if cap == 64 else modes, dtype=torch.int32)
        modes = t[2, :n].cpu().numpy()
        s = _lib.HsSwitchList()
        s.y, s.x, s.mode, s.cap = t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), cap
        count = torch.tensor([n], device=mm.device, dtype=torch.int32)
        _lib.check(mm._lib.hs_dipolar_update(mm._lattice_struct(), ctypes.byref(s), count.data_ptr(), 0, semantics, None,
                                             mm._stream()), 'hs_dipolar_update')
        out.append((d._E.clone(), d._Ep.clone() if P0 is not None else d._E.clone()))
    assert bool((out[0][0] == out[1][0]).all()) and bool((out[0][1] == out[1][1]).all())
    assert not bool((out[0][0] == E0).all())
