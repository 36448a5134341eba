"""A candidate whose memory runs out only in its first sweep -- where the
moments, the pair values and GMRES's vectors are reserved -- is no candidate
either, and its plan is released; any other error of the sweep is passed on."""
import importlib

import pytest

from conftest import pkg

PKG = "matlab-cuda-efief-vs-cpu_b200"


@pytest.mark.parametrize("ident,passes", [("efie:nomem", False), ("cuda:rt", True)])
def test_sweep_without_memory_is_no_candidate(ident, passes, monkeypatch):
    pkg()
    at, api, nat = (importlib.import_module(PKG + x) for x in (".autotune", ".api", "._native"))
    closed = []

    class Plan:
        Ne = 1234

        def __init__(self, *a, **k):
            pass

        def run(self, freqs):
            raise nat.MexError(ident, "a failed sweep")

        def close(self):
            closed.append(self)

    monkeypatch.setattr(api, "SweepPlan", Plan)
    monkeypatch.setattr(api, "sweep_opts", lambda **kw: kw)
    args = [None, None, list(range(1234))] + [None] * 17
    if passes:
        with pytest.raises(nat.MexError):
            at._time(args, [2e9], 1, batch=64, lu_nb=512)
    else:
        assert at._time(args, [2e9], 1, batch=64, lu_nb=512) == (1234, None)
    assert len(closed) == 1
