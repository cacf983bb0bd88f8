"""progress() runs that end by their stop rule where one warp of the step's CTA writes the counters that
the rule reads: Wolff clusters against the oracle, Metropolis steps of at most 32 candidates on
the engine against the step kernels."""
import math

import numpy as np
import pytest

from cases import build_oracle
from gpu_cases import build_product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nx,ny,T', [(60, 44, 300.0), (40, 36, 150.0), (2, 5, 200.0)])
@pytest.mark.parametrize('mc_max', [0.01, 0.6, 2.0])
@pytest.mark.parametrize('engine', [True, False])
def test_wolff_progress_ends_at_the_limit(nx, ny, T, mc_max, engine):
    import hotspice_b200 as hs
    spec = {'lattice': 'OOP_Square', 'a': 200e-9, 'moment': 1e-15, 'nx': nx, 'ny': ny, 'seed': 12, 'kw': {'PBC': True},
            'energies': [{'type': 'exchange', 'J': 1e-21}],
            'params': {'UPDATE_SCHEME': 'Wolff', 'MULTISAMPLING_SCHEME': 'cluster'}}
    fx = {'T': T, 'E_B': np.zeros((ny, nx)), 'm0': np.random.default_rng(5).integers(0, 2, size=(ny, nx)) * 2 - 1}
    mo = build_oracle('wolff', spec=spec, fx=fx)
    mp = build_product('wolff', spec=spec, fx=fx, engine=hs.EngineConfig(persistent=engine))
    for _ in range(3):
        _, mc = mo.progress(t_max=math.inf, MCsteps_max=mc_max)
        _, dmc = mp.progress(t_max=math.inf, MCsteps_max=mc_max)
        c = mp._read_counters()
        assert int(c['attempted']) == mo.attempted_switches and int(c['switches']) == mo.switches
        assert int(c['rng_call']) == mo.rng.call and int(c['status']) == 0
        assert dmc == pytest.approx(mc, rel=1e-12)
        assert np.array_equal(mp.m.cpu().numpy(), mo.m)


@pytest.mark.parametrize('r', [8e-6, 30e-6])          # 20 candidates and two
@pytest.mark.parametrize('limits', [{'t_max': math.inf, 'MCsteps_max': 0.3}, {'t_max': 4e-10, 'MCsteps_max': 4.0}])
@pytest.mark.parametrize('B', [1e-3, 2e-6])          # barriers that make a step's time infinite, and ordinary ones
@pytest.mark.parametrize('cs', [1, 4])
def test_small_grid_metropolis_progress_ends_at_the_limit(r, limits, cs, B):
    import hotspice_b200 as hs
    g = np.random.default_rng(9)
    m0 = g.integers(0, 2, size=(50, 61)) * 2 - 1
    out = []
    for engine in (hs.EngineConfig(persistent=False, use_graphs=False), hs.EngineConfig(cluster_size=cs)):
        mm = hs.ASI.OOP_Square(1e-6, nx=61, ny=50, T=300, E_B=2e-20, moment=1e-15, pattern=m0, seed=3, engine=engine,
                               energies=[hs.DipolarEnergy(cutoff_range=6e-6), hs.ZeemanEnergy(B)],
                               params=hs.SimParams(UPDATE_SCHEME='Metropolis', METROPOLIS_TIME=True))
        plan, _ = mm._grid_plan(r, 'grid')
        assert plan.n_sc <= 32
        ends = [mm.progress(r=r, **limits) for _ in range(3)]
        c = mm._read_counters()
        out.append((ends, {k: c[k] for k in ('attempted', 'switches', 'rng_call', 't', 'status')}, mm.m.cpu().numpy(),
                    mm.E.cpu().numpy()))
        assert int(c['attempted']) > 0
    np.testing.assert_equal(out[0][:2], out[1][:2])
    assert np.array_equal(out[0][2], out[1][2]) and np.array_equal(out[0][3], out[1][3])
