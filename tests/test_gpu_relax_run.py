"""relax() in one cooperative launch (hs_relax_run) against the sweeps launched kernel by kernel
(hs_minimize_all and hs_relax_check), bit for bit: tiles with a rest, several words per row and
several tiles per CTA, windows that are plain, truncated, minimum-image and wider than the lattice,
exchange, a barrier that counts, one channel and two."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lattice(kind, nx, ny, cut, PBC=False, exchange=False, cutoff_switches=20, monopoles=False):
    import hotspice_b200 as hs
    cls, a = {'oop': (hs.ASI.OOP_Square, 200e-9), 'pin': (hs.ASI.IP_Pinwheel, 300e-9), 'kag': (hs.ASI.IP_Kagome, 500e-9)}[kind]
    g = np.random.default_rng(nx * 1000 + ny)
    energies = [hs.DiMonopolarEnergy(d=0.4 * a, small_d=0.15 * a) if monopoles else
                hs.DipolarEnergy(cutoff_range=cut * a if cut else math.inf), hs.ZeemanEnergy(2e-4, 0.3)]
    if exchange:
        energies.append(hs.ExchangeEnergy(J=2e-21))
    return cls(a, nx=nx, ny=ny, T=300, E_B=2e-20 * g.lognormal(0, 0.05, size=(ny, nx)), moment=1e-15, PBC=PBC, seed=21,
               pattern=g.integers(0, 2, size=(ny, nx)) * 2 - 1, energies=energies,
               params=hs.SimParams(SIMULTANEOUS_SWITCHES_CONVOLUTION_OR_SUM_CUTOFF=cutoff_switches))


def _kernel_by_kernel(mm, ignore_barrier):
    from hotspice_b200 import _lib
    L, s, buf = mm._relax_args()
    st, C = mm._stream(), mm._counters.data_ptr()
    n_max = int(math.sqrt(mm.nx ** 2 + mm.ny ** 2))
    _lib.check(mm._lib.hs_relax_begin(L, buf.data_ptr(), buf.numel(), st))
    for _ in range(n_max):
        _lib.check(mm._lib.hs_minimize_all(L, C, s, int(ignore_barrier), 0, buf.data_ptr(), buf.numel(), st))
        _lib.check(mm._lib.hs_relax_check(L, C, n_max, buf.data_ptr(), buf.numel(), st))
    return mm._relax_word(buf, 1)


@pytest.mark.parametrize('kind,nx,ny,cut,PBC,opts', [
    ('oop', 2, 2, 0, False, {}),
    ('oop', 30, 17, 0, False, {}),                                   # uncut, truncated when many switch
    ('oop', 130, 70, 5, True, {}),                                   # minimum image, three words, a rest
    ('oop', 64, 40, 0, True, {'cutoff_switches': 0}),                # folded kernel, truncated and periodic
    ('pin', 131, 61, 8.3, False, {}),
    ('pin', 260, 200, 4, True, {}),
    ('pin', 50, 34, 0, False, {'monopoles': True}),                  # E_perp keeps its sign
    ('kag', 300, 67, 5, False, {}),
    ('kag', 36, 19, 4, False, {'exchange': True}),                   # a second barrier
    ('oop', 700, 300, 2, False, {}),                                 # more tiles than SMs
])
@pytest.mark.parametrize('ignore_barrier', [True, False])
def test_relax_run_equals_kernel_by_kernel(kind, nx, ny, cut, PBC, opts, ignore_barrier):
    one, many = (_lattice(kind, nx, ny, cut, PBC, **opts) for _ in range(2))
    one.relax(ignore_barrier=ignore_barrier)
    sweeps = _kernel_by_kernel(many, ignore_barrier)
    assert one.relax_sweeps == sweeps
    a, b = one._read_counters(), many._read_counters()
    for f in ('rng_call', 'switches', 'attempted', 'status'):
        assert int(a[f]) == int(b[f]), f
    assert np.array_equal(one.m.cpu().numpy(), many.m.cpu().numpy())
    assert np.array_equal(one._mm_dev.cpu().numpy(), many._mm_dev.cpu().numpy())
    assert np.array_equal(one.E.cpu().numpy(), many.E.cpu().numpy())
    if one.USE_PERP_ENERGY:
        assert np.array_equal(one.E_perp.cpu().numpy(), many.E_perp.cpu().numpy())
    print(kind, nx, ny, sweeps, int(a['switches']))
