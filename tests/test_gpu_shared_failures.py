"""Failure paths of sweeps long enough to share factors, made on the host: a
singular matrix at every frequency is reported for the first of the caller's
list, and where the waits of every solve run out, the frequencies that need one
are left to the complex128 LU -- all of the first batch; later ones may meet the
target from the combination of solved currents alone -- with nothing left over
for the next sweep."""
import numpy as np
import pytest

import efie_oracle as eo
from conftest import pkg, small_design

pytestmark = pytest.mark.gpu
FREQS = np.linspace(3e9, 2e9, 41)   # falling: the first is the last one solved in order of frequency


def _plan(p, rwg=None, **kw):
    m = pkg()
    r, d = rwg or p["rwg"], p["design"]
    return m.SweepPlan(p["V"], p["F"], r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"],
                       r["rm"], r["Ap"], r["Am"], r["len"], p["prepack"], d.mu, d.eps, p["patchEdge"],
                       p["groundEdge"], d.V0, p["spread"], d.Z0, opts=m.sweep_opts(nfreq_hint=len(FREQS), **kw))


def test_singular_matrix_of_a_long_sweep():
    m = pkg()
    p = eo.build_problem(small_design("grid"))
    r = dict(p["rwg"])
    j = next(e for e in range(r["Ne"]) if e + 1 not in (p["patchEdge"], p["groundEdge"]))
    r["len"] = r["len"].copy()
    r["len"][j] = 0.0
    plan = _plan(p, r)
    with pytest.raises(m.MexError) as e:
        plan.run(FREQS)
    plan.close()
    assert e.value.identifier == "efie:singular" and "frequency index 1 " in str(e.value)


def test_waits_that_run_out_in_a_long_sweep():
    m = pkg()
    nat = __import__(m.__name__ + "._native", fromlist=["x"])
    p = eo.build_problem(small_design("grid"))
    ref = _plan(p, solver="fp64")
    Zr = ref.run(FREQS)[0]
    ref.close()
    plan = _plan(p)
    Z0 = plan.run(FREQS)[0]
    nat.check(nat.lib().efie_debug_set_wait_test(1, 1 << 12))
    try:
        Zt = plan.run(FREQS)[0]
        st = plan.stats
    finally:
        nat.check(nat.lib().efie_debug_set_wait_test(0, 0))
    assert st["n_fp64_fallback"] == st["n_wait_timeouts"] >= 3   # a start needs three solved frequencies
    assert np.max(np.abs(Zt - Zr) / np.abs(Zr)) <= 1e-9   # the FP64 path's bound
    Z1 = plan.run(FREQS)[0]
    assert plan.stats["n_wait_timeouts"] == plan.stats["n_fp64_fallback"] == 0
    plan.close()
    assert np.array_equal(Z1, Z0)
