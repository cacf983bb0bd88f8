"""FP64 fast convolution (hs_dipolar_full_fft) against the FP64 direct sum, at the sizes where
its transforms change form: every odd factor and stage count, tiles with a rest, the longest
line, windows cropped and wrapped, one and two energy channels per transform."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _make(kind, nx, ny, cut=0.0, PBC=False, perp=None, pattern='random'):
    import hotspice_b200 as hs
    cls, a = {'oop': (hs.ASI.OOP_Square, 200e-9), 'tri': (hs.ASI.OOP_Triangle, 400e-9),
              'pin': (hs.ASI.IP_Pinwheel, 300e-9), 'kag': (hs.ASI.IP_Kagome, 500e-9)}[kind]
    kw = {} if perp is None else dict(m_perp_factor=perp)
    g = np.random.default_rng(nx + 31 * ny)
    moment = 1e-15 * g.uniform(0.5, 1.5, size=(ny, nx))
    return cls(a, nx=nx, ny=ny, T=300, E_B=5e-20, moment=moment, pattern=pattern, PBC=PBC, seed=7,
               energies=[hs.DipolarEnergy(cutoff_range=cut * a if cut else math.inf)], **kw)


def _both(mm):
    d = mm._dipolar()
    d.update(method='direct64')
    ref = [d._E.clone()] + ([d._Ep.clone()] if mm.USE_PERP_ENERGY else [])
    d._E.fill_(7.0)
    if d._Ep is not None:
        d._Ep.fill_(7.0)
    d.update(method='fft64')
    got = [d._E.clone()] + ([d._Ep.clone()] if mm.USE_PERP_ENERGY else [])
    return ref, got


@pytest.mark.parametrize('kind,nx,ny,cut,PBC,perp', [
    ('oop', 2, 1, 0, False, None),        # the shortest lengths
    ('oop', 24, 40, 0, False, None),      # 48 and 80: factors 3 and 5
    ('oop', 72, 16, 0, False, None),      # 144 and 32: factor 9, two stages
    ('oop', 257, 150, 0, False, None),    # 576 and 320: three and more stages, one past 512
    ('oop', 512, 33, 0, True, None),      # 1024, folded periodic kernel
    ('oop', 2000, 3, 0, False, None),     # 4096: the longest line, one column per tile
    ('oop', 3, 2000, 0, False, None),     # the longest column
    ('tri', 61, 40, 0, False, None),      # two sublattices sharing a transform
    ('kag', 36, 19, 0, False, 0.0),       # six of them, one channel
    ('kag', 100, 55, 0, False, None),     # six sublattices, two channels
    ('pin', 131, 90, 7, False, None),     # cropped window
    ('pin', 130, 90, 7, True, None),      # minimum image
    ('oop', 40, 36, 16, True, None),      # minimum image, a window nearly as wide as the lattice
])
def test_fft_matches_direct_sum(kind, nx, ny, cut, PBC, perp):
    mm = _make(kind, nx, ny, cut, PBC, perp)
    ref, got = _both(mm)
    d = mm._dipolar()
    ks = d.kernel_set
    # error bounds relative to |K|_2 |m mu|_2, which bounds every sum: the direct sum loses at most
    # one rounding per term, three transforms and the product at most 12 log2(length) of them, and
    # sums below 2^-52 |K|_max |m mu|_max sqrt(#sources) are 0
    terms = min(nx * ny, ks.K[0].size)
    eps = 2.0 ** -53
    mm2 = float(mm._mm_dev.double().norm())
    for r, g, k in zip(ref, got, (ks.K, ks.Kps)):
        # both channels of a site go through one transform
        k2 = max(math.sqrt(float((ks.K[s] ** 2).sum() + (ks.Kps[s] ** 2).sum())) for s in range(len(ks.K)))
        tol = (12 * 24 + terms + 4) * eps * k2 * mm2 * 1.5e-15
        err = float((r - g).abs().max())
        print(kind, nx, ny, err, tol, float(r.abs().max()))
        assert err <= tol
    assert bool((got[0][mm._m_dev == 0] == 0).all())


def test_fft_vanishing_and_nonfinite_sums():
    """A magnet without a partner in reach has exactly no energy; infinities and NaN reach the
    cells that the direct sum gives them to."""
    m = np.zeros((40, 40))
    m[0, 0], m[39, 39], m[39, 0] = 1, -1, 1
    mm = _make('oop', 40, 40, cut=6, pattern=m)
    ref, got = _both(mm)
    assert bool((got[0] == 0).all()) and bool((ref[0] == 0).all())
    for bad in (math.inf, math.nan):
        mm = _make('oop', 40, 30, cut=6)
        mom = np.full((30, 40), 1e-15)
        mom[11, 17] = bad
        mm.moment = mom
        ref, got = _both(mm)
        same = (ref[0] == got[0]) | (ref[0].isnan() & got[0].isnan())
        assert bool(same.all())
        assert int((~ref[0].isfinite()).sum()) < 13 * 13 + 1
