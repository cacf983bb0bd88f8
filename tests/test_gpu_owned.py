"""Néel steps on owned cells (the engine's path for a uniform temperature without exchange) against
the step kernels, bit for bit, where the ownership changes form: fewer magnets than a chunk, one
past a chunk, several chunks per warp, numbered cells and listed magnets, windows that wrap or span
the lattice, a period longer than the row table, no dipolar energy; and switches decided by the
time that is left."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lattice(kind, nx, ny, cut, PBC=False, zeeman=True, dipolar=True, **kw):
    import hotspice_b200 as hs

    class Holes(hs.ASI.OOP_Square):           # no period: the unit cell is the lattice
        def _get_occupation(self):
            return np.random.default_rng(5).random((self.ny, self.nx)) < 0.6

    cls, a = {'oop': (hs.ASI.OOP_Square, 200e-9), 'pin': (hs.ASI.IP_Pinwheel, 300e-9), 'kag': (hs.ASI.IP_Kagome, 500e-9),
              'hole': (Holes, 200e-9)}[kind]
    g = np.random.default_rng(nx * 1000 + ny)
    energies = ([hs.DipolarEnergy(cutoff_range=cut * a if cut else math.inf)] if dipolar else []) + \
        ([hs.ZeemanEnergy(1e-3, 0.4)] if zeeman else [])
    return cls(a, nx=nx, ny=ny, T=300, E_B=5.5e-20 * g.lognormal(0, 0.05, size=(ny, nx)), moment=1e-15, PBC=PBC, seed=9,
               pattern=g.integers(0, 2, size=(ny, nx)) * 2 - 1, energies=energies, **kw)


def _same(x, y):
    cx, cy = x._read_counters(), y._read_counters()
    for f in ('rng_call', 'attempted', 'switches', 'status', 'steps', 't', 'last_time', 'n_sw'):
        assert cx[f] == cy[f], f
    assert np.array_equal(x.m.cpu().numpy(), y.m.cpu().numpy())
    assert np.array_equal(x.E.cpu().numpy(), y.E.cpu().numpy())
    if x.USE_PERP_ENERGY:
        assert np.array_equal(x.E_perp.cpu().numpy(), y.E_perp.cpu().numpy())


CASES = [('oop', 5, 6, 0, False), ('oop', 33, 1, 0, False), ('oop', 31, 33, 4, False), ('oop', 97, 80, 6, True),
         ('oop', 40, 36, 19, True), ('pin', 66, 50, 5, True), ('pin', 131, 90, 16, False), ('kag', 36, 19, 3, False),
         ('hole', 9, 8, 0, False)]


@pytest.mark.parametrize('cs', [1, 2, 8])
@pytest.mark.parametrize('kind,nx,ny,cut,PBC', CASES)
def test_owned_steps_equal_step_kernels(kind, nx, ny, cut, PBC, cs):
    import hotspice_b200 as hs
    ref = _lattice(kind, nx, ny, cut, PBC, engine=hs.EngineConfig(persistent=False, use_graphs=False))
    own = _lattice(kind, nx, ny, cut, PBC, engine=hs.EngineConfig(cluster_size=cs))
    for mm in (ref, own):
        mm.run(60)
    _same(ref, own)
    for mm in (ref, own):        # a limit that the next few steps reach: the time decides
        mm.progress(t_max=float(own._read_counters()['last_time']) * 2.5, MCsteps_max=40.0 / own.n)
    _same(ref, own)


def test_owned_steps_with_a_long_period_and_without_dipoles():
    import hotspice_b200 as hs
    with pytest.warns(UserWarning, match='unit cell'):
        pair = [_lattice('hole', 70, 66, 0, dipolar=False, engine=hs.EngineConfig(**e))
                for e in (dict(persistent=False, use_graphs=False), dict(cluster_size=4))]
    for mm in pair:
        mm.run(50)
    _same(*pair)
    pair = [_lattice('pin', 40, 40, 0, dipolar=False, engine=hs.EngineConfig(**e))
            for e in (dict(persistent=False, use_graphs=False), dict(cluster_size=2))]
    for mm in pair:
        mm.run(50)
    _same(*pair)
