"""A sweep of no frequencies returns empty Zin, S11 and currents, whatever the
solver and the sharing of factors, and leaves the plan as it was."""
import numpy as np
import pytest

import efie_oracle as eo
from conftest import pkg, small_design

pytestmark = pytest.mark.gpu
NONE = np.zeros(0)


def _args(p):
    r = p["rwg"]
    return [p["V"], p["F"], r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"], r["rm"],
            r["Ap"], r["Am"], r["len"]]


@pytest.mark.parametrize("kw", [{}, dict(share_factors=1), dict(share_factors=2), dict(nfreq_hint=9),
                                dict(solver="fp64"), dict(refine="classical")])
def test_plan_runs_an_empty_list(kw):
    m = pkg()
    p = eo.build_problem(small_design())
    d = p["design"]
    plan = m.SweepPlan(*_args(p), p["prepack"], d.mu, d.eps, p["patchEdge"], p["groundEdge"], d.V0, p["spread"], d.Z0,
                       opts=m.sweep_opts(**kw))
    before = plan.run(d.freqs)
    Zin, S11, I = plan.run(NONE, return_currents=True)
    assert Zin.shape == S11.shape == (0,) and I.shape == (p["rwg"]["Ne"], 0)
    assert plan.stats["n_freq"] == 0 and plan.stats["n_launches"] == 0
    after = plan.run(d.freqs)
    plan.close()
    assert np.array_equal(before, after)


def test_calls_take_an_empty_list():
    m = pkg()
    p = eo.build_problem(small_design())
    d = p["design"]
    tail = [NONE, d.mu, d.eps, p["patchEdge"], p["groundEdge"], d.V0, p["spread"], d.Z0]
    for Zin, S11 in (m.patch_sweep_fastquad_cuda(*_args(p), p["prepack"], *tail), m.patch_sweep_cuda(*_args(p), *tail)):
        assert Zin.shape == S11.shape == (0,)
