"""The switch list a step writes to: large enough for the step, and alive while a descriptor points to it."""
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
