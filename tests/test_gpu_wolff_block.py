"""Wolff clusters that the whole CTA grows, over tens of layers, against the oracle: every layer's
count of joined cells is read by all warps and set to zero again for a later layer, and a cell that
joins a layer must not count as a neighbour of that layer's other candidates."""
import numpy as np
import pytest

from cases import build_oracle
from gpu_cases import build_product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('lattice,nx,ny,T,PBC', [
    ('OOP_Square', 96, 70, 120.0, True), ('OOP_Square', 1, 400, 20.0, False), ('OOP_Square', 200, 3, 60.0, False),
    ('IP_Kagome', 120, 71, 100.0, False),      # triangles: cells of one layer are neighbours of each other
])
@pytest.mark.parametrize('engine', [True, False])
def test_large_clusters_against_oracle(lattice, nx, ny, T, PBC, engine):
    import hotspice_b200 as hs
    spec = {'lattice': lattice, 'a': 200e-9, 'moment': 1e-15, 'nx': nx, 'ny': ny, 'seed': 33, 'kw': {'PBC': PBC},
            'energies': [{'type': 'exchange', 'J': 1e-21}],
            'params': {'UPDATE_SCHEME': 'Wolff', 'MULTISAMPLING_SCHEME': 'cluster'}}
    fx = {'T': T, 'E_B': np.zeros((ny, nx)), 'm0': np.ones((ny, nx), dtype=int)}
    mo = build_oracle('wolff', spec=spec, fx=fx)
    mp = build_product('wolff', spec=spec, fx=fx, engine=hs.EngineConfig(persistent=engine, use_graphs=False))
    largest = 0
    for _ in range(20):
        before = mo.attempted_switches
        mo.update()
        mp.run(1)
        largest = max(largest, mo.attempted_switches - before)
        c = mp._read_counters()
        assert int(c['attempted']) == mo.attempted_switches and int(c['switches']) == mo.switches
        assert int(c['rng_call']) == mo.rng.call and int(c['status']) == 0
        assert np.array_equal(mp.m.cpu().numpy(), mo.m)
    assert largest > 320      # more than the one-warp lists hold
