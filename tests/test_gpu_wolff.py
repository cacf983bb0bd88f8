"""Wolff clusters step by step against the oracle, where the growth changes hands: clusters that stay
on one warp, clusters that outgrow its lists, neighbourhoods that wrap on small lattices, and a mask
of non-square neighbours."""
import numpy as np
import pytest

from cases import build_oracle
from gpu_cases import build_product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('lattice,nx,ny,T,PBC,pattern', [
    ('OOP_Square', 300, 7, 300.0, True, 'random'),      # small clusters
    ('OOP_Square', 40, 36, 140.0, True, 'uniform'),     # clusters of most of the lattice
    ('OOP_Square', 61, 47, 165.0, False, 'random'),     # mixed sizes
    ('OOP_Square', 3, 3, 200.0, True, 'random'),
    ('OOP_Square', 2, 5, 200.0, True, 'random'),        # neighbours that wrap onto themselves
    ('IP_Kagome', 40, 23, 150.0, False, 'uniform'),     # six neighbours, empty cells
])
@pytest.mark.parametrize('engine', [True, False])
def test_wolff_growth_against_oracle(lattice, nx, ny, T, PBC, pattern, engine):
    import hotspice_b200 as hs
    a = 200e-9
    g = np.random.default_rng(nx * ny)
    spec = {'lattice': lattice, 'a': a, 'moment': 1e-15, 'nx': nx, 'ny': ny, 'seed': 51, 'kw': {'PBC': PBC},
            'energies': [{'type': 'exchange', 'J': 1e-21}],
            'params': {'UPDATE_SCHEME': 'Wolff', 'MULTISAMPLING_SCHEME': 'cluster'}}
    m0 = np.ones((ny, nx), dtype=int) if pattern == 'uniform' else g.integers(0, 2, size=(ny, nx)) * 2 - 1
    fx = {'T': T, 'E_B': np.zeros((ny, nx)), 'm0': m0}
    mo = build_oracle('wolff', spec=spec, fx=fx)
    mp = build_product('wolff', spec=spec, fx=fx, engine=hs.EngineConfig(persistent=engine, use_graphs=False))
    sizes = []
    for _ in range(25):
        before = mo.attempted_switches
        mo.update()
        mp.run(1)
        sizes.append(mo.attempted_switches - before)
        c = mp._read_counters()
        assert int(c['attempted']) == mo.attempted_switches and int(c['switches']) == mo.switches
        assert int(c['rng_call']) == mo.rng.call and int(c['status']) == 0
        assert np.array_equal(mp.m.cpu().numpy(), mo.m)
    print(lattice, nx, ny, sizes)
