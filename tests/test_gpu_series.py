"""Sweep assembly from frequency-independent moments against the FP64 oracle:
Z of every frequency within 1e-12 max|Z| (the bound of the per-frequency
assembly), bit-exactly symmetric, for each quadrature rule, term count, medium
and tile remainder, with the moments held whole or a few tiles at a time."""
import ctypes as C
import importlib

import numpy as np
import pytest

import efie_oracle as eo
import oracle_c as oc
from conftest import config1_design, pkg, small_design

pytestmark = pytest.mark.gpu

ONE = dict(quad_order=1, near_sing_eps=1.2, self_subdiv=1, near_subdiv=1, near_order=2, self_alpha=0.2, near_alpha=0.15)
# name -> design, scheme, frequencies (GHz), eps_r
CASES = {
    "even": (lambda: small_design(), "ref", np.linspace(2, 3, 6), 1.0),
    "uneven": (lambda: small_design("reference"), "ref", [0.3, 1.1, 2.9], 1.0),
    "one": (lambda: small_design(npx=3, npy=2, ngx=2, ngy=2), "ref", [2.5], 1.0),
    "tile_less_one": (lambda: small_design(npx=1, npy=5, ngx=2, ngy=5), "ref", [2.0, 2.5], 1.0),
    "lossy_even": (lambda: small_design(), "ref", np.linspace(1, 2, 5), 4.4 * (1 - 0.02j)),
    "lossy_uneven": (eo.reference_sweep_design, "ref", [1.0, 1.31, 1.4], 2.59 * (1 - 1e-4j)),
    "accurate": (lambda: small_design(opts=eo.DEFAULT_OPTS_ACCURATE), "ref", [2.0, 3.0], 1.0),
    "centre_rule": (lambda: small_design(opts=ONE), "ref", [2.0, 3.0], 1.0),
    "high": (lambda: small_design(), "ref", [5.0, 12.0], 1.0),
    "config1": (config1_design, "ref", [2.0, 2.4, 3.0], 1.0),
    "extract": (lambda: small_design(), "extract", np.linspace(2, 3, 4), 1.0),
    "extract_lossy": (lambda: small_design(npx=7, npy=5, ngx=9, ngy=4), "extract", [1.0, 2.7], 3.0 * (1 - 0.05j)),
}


def _plan(p, scheme, nf, eps):
    m = pkg()
    r, d = p["rwg"], p["design"]
    return m.SweepPlan(p["V"], p["F"], r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"],
                       r["rm"], r["Ap"], r["Am"], r["len"], None if scheme == "extract" else p["prepack"], d.mu, eps,
                       p["patchEdge"], p["groundEdge"], d.V0, p["spread"], d.Z0,
                       opts=m.sweep_opts(scheme=scheme, batch=nf), rule_order=eo.DUNAVANT7)


def _series(plan, freqs, tiles):
    nat = importlib.import_module("matlab-cuda-efief-vs-cpu_b200._native")
    f = np.ascontiguousarray(freqs, dtype=np.float64)
    Z = np.zeros((f.size, plan.Ne, plan.Ne), dtype=np.complex128)
    terms = C.c_int32()
    nat.check(nat.lib().efie_debug_plan_series(plan._h, f.ctypes.data_as(nat.c_double_p), f.size, tiles,
                                               C.byref(terms), Z.ctypes.data))
    return Z.transpose(0, 2, 1), terms.value   # column-major slots


@pytest.mark.parametrize("tiles", [0, 5])
@pytest.mark.parametrize("name", list(CASES))
def test_series_z_matches_oracle(name, tiles):
    make, scheme, ghz, er = CASES[name]
    d = make()
    d.eps = eo.EPS0 * er
    p = eo.build_problem(d)
    freqs = np.asarray(ghz, dtype=np.float64) * 1e9
    plan = _plan(p, scheme, len(freqs), d.eps)
    Z, terms = _series(plan, freqs, tiles)
    assert terms > 0
    for f, z in zip(freqs, Z):
        omega, k, _, _ = eo.physics(f, d.mu, d.eps)
        if scheme == "extract":
            zo = oc.assemble_z_extract(p["V"], p["F"], p["rwg"], k, omega, d.mu, d.eps)
        else:
            zo = oc.assemble_z(p["rwg"], p["prepack"], k, omega, d.mu, d.eps)
        assert np.abs(z - zo).max() < 1e-12 * np.abs(zo).max()
        assert np.array_equal(z, z.T)
    plan.close()


@pytest.mark.parametrize("change", ["half", "off_vertex"])
def test_series_takes_any_rwg_side(change):
    """An RWG with one triangle missing, and one whose free vertex is not a vertex of its triangle."""
    p = eo.build_problem(small_design())
    r = {k: np.array(v, copy=True) for k, v in p["rwg"].items()}
    if change == "half":
        r["minusTri"][5] = 0
    else:
        r["rp"][7] += 1e-9 * np.abs(p["V"]).max()
    p = dict(p, rwg=r)
    d = p["design"]
    plan = _plan(p, "ref", 1, d.eps)
    Z, terms = _series(plan, [2.3e9], 0)
    omega, k, _, _ = eo.physics(2.3e9, d.mu, d.eps)
    zo = oc.assemble_z(r, p["prepack"], k, omega, d.mu, d.eps)
    assert terms > 0 and np.abs(Z[0] - zo).max() < 1e-12 * np.abs(zo).max()
    plan.close()


def test_series_leaves_electrically_large_bases_alone():
    p = eo.build_problem(small_design())
    plan = _plan(p, "ref", 1, eo.EPS0)
    _, terms = _series(plan, [90e9], 0)   # k delta over 3
    assert terms == 0
    plan.close()
