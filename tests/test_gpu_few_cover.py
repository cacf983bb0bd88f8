"""Short switch lists whose windows cover each other, wholly or in part: the engine against the step
kernels, bit for bit, and its time beside theirs (each cell is updated once, not once per window)."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _lattice(kind, nx, ny, cut, PBC, persistent):
    import hotspice_b200 as hs
    cls, a = {'oop': (hs.ASI.OOP_Square, 200e-9), 'pin': (hs.ASI.IP_Pinwheel, 300e-9)}[kind]
    g = np.random.default_rng(nx + ny)
    return cls(a, nx=nx, ny=ny, T=300, E_B=5e-20, moment=1e-15, PBC=PBC, seed=4,
               pattern=g.integers(0, 2, size=(ny, nx)) * 2 - 1, params=hs.SimParams(UPDATE_SCHEME='Metropolis'),
               energies=[hs.DipolarEnergy(cutoff_range=cut * a if cut else math.inf)],
               engine=hs.EngineConfig(persistent=persistent, use_graphs=False))


@pytest.mark.parametrize('kind,nx,ny,cut,PBC,r', [
    ('oop', 64, 61, 0, False, 8), ('oop', 130, 70, 0, False, 20), ('pin', 96, 97, 0, False, 16),   # all of the lattice
    ('oop', 64, 60, 0, True, 8), ('oop', 70, 64, 40, True, 9),                 # minimum image
    ('oop', 200, 150, 30, False, 25), ('pin', 160, 131, 20, False, 24), ('pin', 160, 130, 20, True, 24),   # in part
])
def test_engine_equals_step_kernels_where_windows_overlap(kind, nx, ny, cut, PBC, r):
    one, many = (_lattice(kind, nx, ny, cut, PBC, p) for p in (True, False))
    r *= float(np.min(one.dx))
    assert one._grid_plan(r, 'grid')[0].n_sc <= 64
    for mm in (one, many):
        mm.run(40, r=r)
    assert one.switches == many.switches > 0
    assert bool((one.m == many.m).all()) and bool((one.E == many.E).all())
    if one.in_plane:
        assert bool((one.E_perp == many.E_perp).all())


def test_covering_windows_cost_one_pass_per_cell():
    """256 x 256 uncut, some 15 switches a step. A pass per cell and switch takes the engine
    20 to 300 us (on 16 CTAs, on one), the step kernels about 15; a pass per pair of windows took 4.6 ms."""
    us = []
    for persistent in (True, False):
        mm = _lattice('oop', 256, 256, 0, False, persistent)
        r = 20 * float(np.min(mm.dx))
        mm.run(20, r=r)
        best = math.inf
        for _ in range(3):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            mm.run(64, r=r)
            e1.record()
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1) / 64 * 1e3)
        us.append(best)
    print(us)
    assert us[0] < 60 * us[1]
