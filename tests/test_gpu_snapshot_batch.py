"""Initial guesses of a whole batch against numpy: every slot has a matrix, a
list of snapshots and a count of its own, with fewer and more work items than
SMs; and the guesses of a sweep are good enough to save its steps."""
import importlib

import numpy as np
import pytest

import efie_oracle as eo
from conftest import config1_design, pkg

pytestmark = pytest.mark.gpu
KMAX = 23


@pytest.mark.parametrize("N,counts", [(129, [1, 2, 8]), (300, [9, 15, 3, 1, 12]), (300, [16, 3, 23, 8, 7, 17]),
                                      (260, list(range(1, 16)) * 4), (257, list(range(1, 24)) * 2 + [23] * 18),
                                      (900, [3, 15, 7, 9] * 6), (900, [23, 1, 17, 8] * 6)])
def test_every_slot_reaches_its_least_residual(N, counts):
    nat = importlib.import_module(pkg().__name__ + "._native")
    r = np.random.default_rng(N + len(counts))
    nf, nx = len(counts), 40
    c = lambda *s: r.standard_normal(s) + 1j * r.standard_normal(s)  # noqa: E731
    base, step = c(N, N) / np.sqrt(N), c(N, N) / np.sqrt(N)
    Z = np.empty((nf, N, N), np.complex128)
    for f in range(nf):
        A = base + 0.1 * f * step
        Z[f] = A + A.T + (4 + f) * np.eye(N)   # symmetric, so either storage order
    xs, b = c(nx, N), r.standard_normal(N).astype(np.complex128)
    pos = np.array([r.permutation(nx)[:KMAX] for _ in range(nf)], np.int32)
    k = np.array(counts, np.int32)
    blk = np.arange(N) // 128
    Zd = Z.copy()
    Zd[:, blk[:, None] < blk[None, :]] = np.nan   # column-major: outside the upper triangle and the diagonal blocks
    x = np.zeros((nf, N), np.complex128)
    nat.check(nat.lib().efie_debug_snapshot_guesses(nat.context(), N, nf, nx, k.ctypes.data, pos.ctypes.data,
                                                    Zd.ctypes.data, xs.ctypes.data, b.ctypes.data, x.ctypes.data))
    for f in range(nf):
        X = xs[pos[f, :k[f]]].T
        best = X @ np.linalg.lstsq(Z[f] @ X, b, rcond=None)[0]
        # well conditioned: the FP64 solutions agree far below this
        assert np.linalg.norm(x[f] - best) <= 1e-9 * np.linalg.norm(best)


def test_guesses_save_a_sweeps_steps():
    m = pkg()
    p = eo.build_problem(config1_design("grid"))
    r, d = p["rwg"], p["design"]
    freqs = np.linspace(2e9, 3e9, 101)
    plan = m.SweepPlan(p["V"], p["F"], r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"],
                       r["rm"], r["Ap"], r["Am"], r["len"], p["prepack"], d.mu, d.eps, p["patchEdge"],
                       p["groundEdge"], d.V0, p["spread"], d.Z0, opts=m.sweep_opts(nfreq_hint=len(freqs)))
    plan.run(freqs)
    st = plan.stats
    trsv = st["classes"]["trsv"]["launches"] // 2   # two solves a step
    batches = -(-(len(freqs) - 15) // 32) + 1
    plan.close()
    # the first batch starts from zero (its steps are at most refine_iters_max); a start that
    # carries the currents to 1e-11 leaves the others two steps a batch, and one that does not, five or more
    assert st["n_shared_factors"] >= 75
    assert trsv <= st["refine_iters_max"] + 2 * batches
