"""Sweeps whose batch cannot hold the frequencies that automatic sharing would
factor run in groups of batches, to the same results, at every batch around
those counts; so do sweeps one frequency longer than they are many."""
import numpy as np
import pytest

import efie_oracle as eo
from conftest import pkg, small_design

pytestmark = pytest.mark.gpu


def _run(p, freqs, **kw):
    m = pkg()
    r, d = p["rwg"], p["design"]
    plan = m.SweepPlan(p["V"], p["F"], r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"],
                       r["rm"], r["Ap"], r["Am"], r["len"], p["prepack"], d.mu, d.eps, p["patchEdge"],
                       p["groundEdge"], d.V0, p["spread"], d.Z0, opts=m.sweep_opts(**kw))
    out = plan.run(freqs, return_currents=True)
    st = plan.stats
    plan.close()
    return out, st


@pytest.fixture(scope="module")
def problem():
    return eo.build_problem(small_design())   # Ne 125: up to 24 frequencies are factored


@pytest.mark.parametrize("nf", [24, 25, 41])
@pytest.mark.parametrize("batch", [1, 2, 8, 9, 23, 24, 32])
def test_any_batch_gives_the_same_sweep(problem, nf, batch):
    freqs = np.linspace(2e9, 3e9, nf)
    (Z0, _, I0), _ = _run(problem, freqs, solver="fp64")
    (Z, _, I), st = _run(problem, freqs, batch=batch)
    assert st["n_fp64_fallback"] == 0 and st["max_relres"] <= 1e-10
    # only a sweep of no more than 24 in one batch is factored whole
    assert (st["n_shared_factors"] > 0) == (batch < nf or nf > 24)
    # residuals of 1e-10 through cond(Z) of this small design, far below the sweeps' 1e-6
    assert np.max(np.abs(Z - Z0) / np.abs(Z0)) <= 1e-6
    assert np.max(np.linalg.norm(I - I0, axis=0) / np.linalg.norm(I0, axis=0)) <= 1e-6
