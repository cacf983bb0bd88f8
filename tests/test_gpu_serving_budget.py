"""A serving budget that holds one request: the next one is admitted when the read-out of the one before
has landed, however quickly it does."""
import pytest
import torch

from hotspice_b200 import serving as S

pytestmark = pytest.mark.gpu


def test_memory_of_a_landed_readout_is_free_for_the_next_request(monkeypatch):
    begin = S.Server._retire_begin

    def landed(self, a, end_event):
        out = begin(self, a, end_event)
        torch.cuda.synchronize()
        return out

    monkeypatch.setattr(S.Server, '_retire_begin', landed)
    reqs = [S.SimRequest(rid=i, spec={'lattice': 'IP_Pinwheel', 'n': 40, 'T': 300.0, 'seed': i}, steps=20, arrival=0.0)
            for i in range(4)]
    srv = S.Server(hbm_budget=max(S.footprint_bytes(r.spec) for r in reqs), round_ms=0.05)
    res = srv.serve(reqs, realtime=False)
    assert sorted(r.rid for r in res) == [0, 1, 2, 3]
    assert srv.stats.max_active == 1
