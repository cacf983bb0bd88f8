"""An update whose switch list has no room, with the number of switches (none) on the device: nothing is read
from the list and the energies stay."""
import pytest
import torch

import hotspice_b200 as hs
from hotspice_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('cutoff', [1.6e-6, 40e-6])      # short windows, and the whole lattice
@pytest.mark.parametrize('semantics', [0, 1])
def test_list_without_room(cutoff, semantics):
    mm = hs.ASI.OOP_Square(200e-9, nx=300, ny=280, T=300, E_B=5e-20, seed=2, energies=[hs.DipolarEnergy(cutoff_range=cutoff)])
    E = mm._dipolar()._E
    before = E.clone()
    s = _lib.HsSwitchList()                               # null pointers, capacity 0
    count = torch.zeros(1, device=mm.device, dtype=torch.int32)
    _lib.check(mm._lib.hs_dipolar_update(mm._lattice_struct(), s, count.data_ptr(), 0, semantics, None, mm._stream()),
               'hs_dipolar_update')
    torch.cuda.synchronize()
    assert torch.equal(E, before)
