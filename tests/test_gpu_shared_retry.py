"""A frequency of a sweep on shared factors that misses the target is factored
by itself, in its own slot: the rest of the sweep keeps sharing, the count of
shared frequencies leaves it out, and every result stays right."""
import numpy as np
import pytest

import efie_oracle as eo
from conftest import config1_design, pkg

pytestmark = pytest.mark.gpu


def _plan(m, p, nf, **kw):
    r, d = p["rwg"], p["design"]
    return m.SweepPlan(p["V"], p["F"], r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"],
                       r["rm"], r["Ap"], r["Am"], r["len"], p["prepack"], d.mu, d.eps, p["patchEdge"],
                       p["groundEdge"], d.V0, p["spread"], d.Z0, opts=m.sweep_opts(nfreq_hint=nf, **kw))


@pytest.mark.parametrize("share", [0, 4])
@pytest.mark.parametrize("limit", [10, 8, 6])
def test_missed_frequencies_leave_the_others_sharing(share, limit):
    m = pkg()
    p = eo.build_problem(config1_design("grid"))
    freqs = np.linspace(1e9, 8e9, 101)   # wide: a neighbour's factors need up to thirteen steps
    plan = _plan(m, p, len(freqs), share_factors=share)
    Zin, _, I = plan.run(freqs, return_currents=True)
    st = plan.stats
    plan.close()
    assert st["refine_iters_max"] > limit and st["n_shared_factors"] >= 50 and st["n_fp64_fallback"] == 0
    few = _plan(m, p, len(freqs), share_factors=share, refine_max_iter=limit)
    for _ in range(2):   # the second run replays the factorization as a graph
        Zf, _, If = few.run(freqs, return_currents=True)
        sf = few.stats
        assert st["n_shared_factors"] // 2 < sf["n_shared_factors"] < st["n_shared_factors"]
        assert sf["n_fp64_fallback"] == 0 and sf["max_relres"] <= 1e-10
        # both meet a residual of 1e-10; the errors it leaves are bounded by the sweeps' usual 1e-6
        assert np.max(np.abs(Zf - Zin) / np.abs(Zin)) <= 1e-6
        assert np.max(np.linalg.norm(If - I, axis=0) / np.linalg.norm(I, axis=0)) <= 1e-6
    few.close()
