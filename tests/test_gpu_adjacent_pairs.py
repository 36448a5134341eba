"""The extraction scheme on meshes whose triangles come in any order: the
adjacent pairs are found and ordered whatever the numbering, so the series'
matrices match the oracle's."""
import ctypes as C
import importlib

import numpy as np
import pytest

import efie_oracle as eo
import oracle_c as oc
from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["grid", "reversed", "shuffled"])
def test_series_on_any_triangle_order(order):
    m = pkg()
    nat = importlib.import_module(m.__name__ + "._native")
    V, F, _, _ = m.make_patch_with_ground_mesh(12e-3, 16e-3, 30e-3, 30e-3, 1.6e-3, 5, 4, 7, 6)
    if order == "reversed":
        F = F[::-1]
    if order == "shuffled":
        F = F[np.random.default_rng(4).permutation(len(F))]
    F = np.asfortranarray(F)
    r = m.build_rwg_interior({"V": V, "F": F})
    mu, eps, f = eo.MU0, eo.EPS0, np.array([2.1e9, 2.9e9])
    plan = m.SweepPlan(V, F, r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"], r["rm"],
                       r["Ap"], r["Am"], r["len"], None, mu, eps, 1, r["Ne"], 1.0, 1.5 * float(np.mean(r["len"])), 50.0,
                       opts=m.sweep_opts(scheme="extract", batch=2), rule_order=eo.DUNAVANT7)
    Z = np.zeros((2, r["Ne"], r["Ne"]), dtype=np.complex128)
    terms = C.c_int32()
    nat.check(nat.lib().efie_debug_plan_series(plan._h, f.ctypes.data_as(nat.c_double_p), 2, 0, C.byref(terms),
                                               Z.ctypes.data))
    plan.close()
    assert terms.value > 0
    for q in range(2):
        omega, k, _, _ = eo.physics(f[q], mu, eps)
        Zo = oc.assemble_z_extract(V, F, r, k, omega, mu, eps)
        assert np.abs(Z[q].T - Zo).max() <= 1e-12 * np.abs(Zo).max()   # the assembly's bound
