"""Sweeps whose buffers cannot be had: the moments of a longer sweep fall back
to the pair values where those still fit, a sweep with room for neither ends
in efie:nomem, and later sweeps of the same plan -- short ones too, which had
a buffer before -- are right or end the same way."""
import importlib

import numpy as np
import pytest

import efie_oracle as eo
from conftest import config1_design, pkg

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture
def limit():
    lib = importlib.import_module(pkg().__name__ + "._native").lib()
    yield lib.efie_debug_limit_allocations
    lib.efie_debug_limit_allocations(0)


@pytest.fixture(scope="module")
def problem():
    return eo.build_problem(config1_design(opts=eo.DEFAULT_OPTS_ACCURATE))   # 41 MB of pair values, 78 of moments


def _plan(p):
    m = pkg()
    r, d = p["rwg"], p["design"]
    return m.SweepPlan(p["V"], p["F"], r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"],
                       r["rm"], r["Ap"], r["Am"], r["len"], p["prepack"], d.mu, d.eps, p["patchEdge"],
                       p["groundEdge"], d.V0, p["spread"], d.Z0, opts=m.sweep_opts(batch=8))


SHORT, LONG = np.array([2.1e9, 2.7e9]), np.linspace(2e9, 3e9, 8)


def test_sweep_without_room_for_moments(problem, limit):
    m = pkg()
    plan = _plan(problem)
    short = plan.run(SHORT)[0]
    limit(60 * MB)
    Zp = plan.run(LONG)[0]   # on the pair values
    again = plan.run(SHORT)[0]
    limit(30 * MB)
    with pytest.raises(m.MexError) as e:
        plan.run(LONG)
    assert e.value.identifier == "efie:nomem"
    try:   # the pair values may have gone with the failed sweep
        assert np.max(np.abs(plan.run(SHORT)[0] - short) / np.abs(short)) <= 1e-6
    except m.MexError as e:
        assert e.identifier == "efie:nomem"
    limit(0)
    last = plan.run(SHORT)[0]
    Zm = plan.run(LONG)[0]   # on the moments
    plan.close()
    assert np.max(np.abs(again - short) / np.abs(short)) <= 1e-6
    assert np.max(np.abs(last - short) / np.abs(short)) <= 1e-6
    assert np.max(np.abs(Zm - Zp) / np.abs(Zm)) <= 1e-6   # the sweeps' bound on both


def test_network_after_a_batch_without_room(limit):
    m = pkg()
    sur = importlib.import_module(m.__name__ + ".surrogate")
    net = sur.Surrogate(n_hidden=256, n_layers=4, seed=1)
    r = np.random.default_rng(2)
    X, T = r.uniform(-1, 1, (60000, 5)).astype(np.float32), r.uniform(-1, 1, (60000, 3)).astype(np.float32)
    Y, (loss, grad) = net.forward(X[:100]), net.loss_grad(X[:100], T[:100])
    limit(100 * MB)   # 60000 rows of activations: 614 MB
    with pytest.raises(m.MexError) as e:
        net.loss_grad(X, T)
    assert e.value.identifier == "efie:nomem"
    assert np.array_equal(net.forward(X[:100]), Y)
    limit(0)
    loss2, grad2 = net.loss_grad(X[:100], T[:100])
    assert loss2 == loss and np.array_equal(grad2, grad)
    assert np.isfinite(net.loss_grad(X, T)[0])
