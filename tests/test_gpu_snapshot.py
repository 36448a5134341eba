"""Least-squares initial guesses from solved frequencies against numpy: the
guess reaches the smallest residual of its span for every snapshot count and
tile remainder, also with repeated and nearly dependent snapshots, and reads
only Z's upper triangle and diagonal blocks; long sweeps refine their later
frequencies in fewer steps than their first and meet the same target."""
import importlib

import numpy as np
import pytest

import efie_oracle as eo
import oracle_c as oc
from conftest import config1_design, pkg

pytestmark = pytest.mark.gpu


def _guess(Z, xs, b):
    m = pkg()
    nat = importlib.import_module(m.__name__ + "._native")
    N = Z.shape[0]
    Z = np.array(Z, order="F")
    blk = np.arange(N) // 128
    Z[blk[:, None] > blk[None, :]] = np.nan   # the lower triangle outside the diagonal blocks is not read
    xs, b = np.ascontiguousarray(xs), np.ascontiguousarray(b)
    x = np.zeros(N, dtype=np.complex128)
    nat.check(nat.lib().efie_debug_snapshot_guess(nat.context(), N, len(xs), Z.ctypes.data, xs.ctypes.data,
                                                  b.ctypes.data, x.ctypes.data))
    return x


def _problem(N, k, kind, seed=3):
    r = np.random.default_rng(seed)
    c = lambda *s: r.standard_normal(s) + 1j * r.standard_normal(s)  # noqa: E731
    Z = c(N, N) / np.sqrt(N)
    Z = Z + Z.T + 4 * np.eye(N)
    b = r.standard_normal(N).astype(np.complex128)
    if kind == "random":
        xs = c(k, N)
    else:   # solutions of neighbouring matrices: nearly dependent, the first one twice
        D = c(N, N) / np.sqrt(N)
        D = D + D.T
        xs = np.stack([np.linalg.solve(Z + 0.02 * (j - k / 2 + 0.3) * D, b) for j in range(k)])
        xs[-1] = xs[0]
    return Z, xs, b


SIZES = [(1, 1), (31, 3), (127, 4), (128, 5), (129, 8), (255, 9), (257, 12), (300, 13), (384, 15), (500, 16), (1000, 23)]


@pytest.mark.parametrize("N,k,kind", [(*s, x) for s in SIZES for x in ("random", "neighbours")] +
                         [(4200, 15, "random"), (2400, 20, "random")])   # several passes of the stacked reduction
def test_guess_reaches_the_least_residual(N, k, kind):
    Z, xs, b = _problem(N, k, kind)
    x = _guess(Z, xs, b)
    W = Z @ xs.T
    best = np.linalg.norm(b - W @ np.linalg.lstsq(W, b, rcond=1e-13)[0])
    got = np.linalg.norm(b - Z @ x)
    # FP64 Householder least squares; dropped columns (1e-13) leave at most that much of ||b||
    assert got <= best * (1 + 1e-6) + 1e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("spacing", ["even", "random", "repeated"])
def test_long_sweep_shares_a_few_factorizations(spacing):
    m = pkg()
    d = config1_design("grid")
    p = eo.build_problem(d)
    r = p["rwg"]
    freqs = np.linspace(2e9, 3e9, 41)
    if spacing == "random":
        freqs = np.random.default_rng(1).uniform(2e9, 3e9, 41)
    if spacing == "repeated":
        freqs = np.repeat(freqs[::2], 2)
    plan = m.SweepPlan(p["V"], p["F"], r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"],
                       r["rm"], r["Ap"], r["Am"], r["len"], p["prepack"], d.mu, d.eps, p["patchEdge"],
                       p["groundEdge"], d.V0, p["spread"], d.Z0, opts=m.sweep_opts(nfreq_hint=len(freqs)))
    Zin, _, I = plan.run(freqs, return_currents=True)
    st = plan.stats
    plan.close()
    assert 0 < st["n_shared_factors"] < len(freqs) and st["n_fp64_fallback"] == 0 and st["max_relres"] <= 1e-10
    for j in (0, 1, 20, len(freqs) - 1):
        omega, k, _, _ = eo.physics(freqs[j], d.mu, d.eps)
        Z = oc.assemble_z(r, p["prepack"], k, omega, d.mu, d.eps)
        assert np.linalg.norm(p["b"] - Z @ I[:, j]) / np.linalg.norm(p["b"]) < 1e-9
        zo = 1.0 / eo.port_current(np.linalg.solve(Z, p["b"].astype(complex)), p["wP"], p["wG"], r["len"])
        assert abs(Zin[j] - zo) <= 1e-6 * abs(zo)
