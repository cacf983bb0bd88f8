"""The Poisson-disc sampler's block form (shared memory) against its one-warp form (scratch
memory), at the background grids where the block form changes: a grid so small that a
neighbourhood wraps around it, one bitmap word per lane and its last full size, several words
per lane."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nx,ny,r_cells', [
    (9, 7, 9),          # one cell
    (60, 11, 7),        # 11 x 2 cells: fewer than four rows
    (46, 44, 1),        # 33 x 32 cells: 1,056 points at most, two words in one lane
    (45, 44, 1),        # 32 x 32: one word per lane, all lanes
    (128, 120, 1.2),    # 83 x 78 cells, seven words per lane
    (300, 200, 20),
])
@pytest.mark.parametrize('PBC', [False, True])
def test_block_sampler_equals_warp_sampler(nx, ny, r_cells, PBC, monkeypatch):
    import hotspice_b200 as hs
    import hotspice_b200.engine as E
    a = 200e-9

    def lattice():
        g = np.random.default_rng(nx)
        return hs.ASI.OOP_Square(a, nx=nx, ny=ny, T=300, E_B=5e-20, moment=1.1e-15, PBC=PBC, seed=11,
                                 pattern=g.integers(0, 2, size=(ny, nx)) * 2 - 1,
                                 energies=[hs.DipolarEnergy(cutoff_range=5 * a)],
                                 params=hs.SimParams(UPDATE_SCHEME='Metropolis', MULTISAMPLING_SCHEME='Poisson'))

    block, warp = lattice(), lattice()
    assert E.BatchEngine([block]).run(6, r=r_cells * a)[0].ws > 0
    monkeypatch.setattr(E, 'poisson_workspace', lambda I: 0)
    assert E.BatchEngine([warp]).run(6, r=r_cells * a)[0].ws == 0
    x, y = block._read_counters(), warp._read_counters()
    for f in ('rng_call', 'attempted', 'switches', 'status', 'steps'):
        assert int(x[f]) == int(y[f]), f
    assert int(x['attempted']) > 0 and int(x['status']) == 0
    assert np.array_equal(block.m.cpu().numpy(), warp.m.cpu().numpy())
    assert np.array_equal(block.E.cpu().numpy(), warp.E.cpu().numpy())
