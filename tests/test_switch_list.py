"""The switch list a step writes to: large enough for the step, and alive while a descriptor points to it."""
import gc
import weakref
from types import SimpleNamespace

import pytest
import torch

from hotspice_b200.core import Magnets


def _holder():
    return SimpleNamespace(device=torch.device('cpu'), _graphs={})


@pytest.mark.parametrize('first,then', [(1, 65), (64, 192), (100, 101), (70, 210)])
def test_list_holds_what_was_asked_for(first, then):
    mm = _holder()
    Magnets._switch_list(mm, first)
    mm._graphs['old'] = 1                      # a graph captured with the shorter list
    t, s = Magnets._switch_list(mm, then)
    assert s.cap >= then and t.shape == (3, s.cap) and not mm._graphs
    assert Magnets._switch_list(mm, first)[0] is t        # it only grows


def test_engine_descriptor_keeps_the_list_it_points_to():
    from hotspice_b200 import _lib
    from hotspice_b200.core import Scheme
    from hotspice_b200.engine import BatchEngine
    mm = _holder()
    mm._counters, mm.params = torch.zeros(256, dtype=torch.uint8), SimpleNamespace(UPDATE_SCHEME=Scheme.NEEL)
    buf = torch.zeros(256, dtype=torch.uint8)
    mm._step_args = lambda kw: ('neel', _lib.HsLattice(), Magnets._switch_list(mm, 1)[1], 1e10, buf)
    inst, keep = BatchEngine._describe(None, mm, 10, {})
    first = weakref.ref(mm._sw[0])
    Magnets._switch_list(mm, 5000)             # relax() between two runs
    gc.collect()
    assert first() is not None and inst.sw.y == first()[0].data_ptr()
    del keep
    gc.collect()
    assert first() is None
