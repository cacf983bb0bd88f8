"""Wolff clusters with neighbour masks of up to 27 entries, wide enough to reach beyond small lattices,
against the oracle."""
import numpy as np
import pytest

from cases import build_oracle
from gpu_cases import build_product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shape,nx,ny,PBC', [
    ((3, 9), 40, 36, True), ((9, 3), 40, 36, False), ((1, 27), 60, 9, True), ((27, 1), 9, 60, False),
    ((3, 9), 3, 30, True), ((9, 3), 30, 3, True), ((1, 27), 13, 12, True), ((1, 27), 12, 12, True),
])
@pytest.mark.parametrize('T', [4000.0, 600.0])        # clusters of a few cells, and of most of the lattice
@pytest.mark.parametrize('engine', [True, False])
def test_wide_masks_against_oracle(shape, nx, ny, PBC, T, engine, monkeypatch):
    import hotspice_b200 as hs
    mask = np.ones(shape, dtype=int)
    mask[shape[0] // 2, shape[1] // 2] = 0
    monkeypatch.setattr(hs.ASI.OOP_Square, '_get_nearest_neighbors', lambda self: mask)
    g = np.random.default_rng(nx * ny)
    spec = {'lattice': 'OOP_Square', 'a': 200e-9, 'moment': 1e-15, 'nx': nx, 'ny': ny, 'seed': 51, 'kw': {'PBC': PBC},
            'energies': [{'type': 'exchange', 'J': 1e-21}],
            'params': {'UPDATE_SCHEME': 'Wolff', 'MULTISAMPLING_SCHEME': 'cluster'}}
    fx = {'T': T, 'E_B': np.zeros((ny, nx)), 'm0': g.integers(0, 2, size=(ny, nx)) * 2 - 1}
    mo = build_oracle('wolff', spec=spec, fx=fx)
    for e in mo.energies:
        e.local_interaction = mask
    mp = build_product('wolff', spec=spec, fx=fx, engine=hs.EngineConfig(persistent=engine, use_graphs=False))
    for _ in range(20):
        mo.update()
        mp.run(1)
        c = mp._read_counters()
        assert int(c['attempted']) == mo.attempted_switches and int(c['switches']) == mo.switches
        assert int(c['rng_call']) == mo.rng.call and int(c['status']) == 0
        assert np.array_equal(mp.m.cpu().numpy(), mo.m)
