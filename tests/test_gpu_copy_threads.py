"""Host threads that assemble on one context at the same time each get their
own matrix, bit for bit what a call alone returns."""
import threading

import numpy as np
import pytest

import efie_oracle as eo
from conftest import pkg, small_design

pytestmark = pytest.mark.gpu


def test_threads_of_one_context_get_their_own_matrix():
    m = pkg()
    calls = []
    for cells in ((10, 8, 14, 13), (11, 9, 15, 15), (12, 10, 16, 16)):   # 9 to 18 MB: several pieces each
        npx, npy, ngx, ngy = cells
        p = eo.build_problem(small_design(npx=npx, npy=npy, ngx=ngx, ngy=ngy))
        r, d = p["rwg"], p["design"]
        omega, k, _, _ = eo.physics(2.5e9, d.mu, d.eps)
        exc = np.array([p["patchEdge"], p["groundEdge"], d.V0, p["spread"], 0.2])
        args = (p["V"], p["F"], r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"],
                r["rm"], r["Ap"], r["Am"], r["len"], k, omega, d.mu, d.eps, exc)
        calls.append((args, m.gassemble_ZV_EFIE_RWG_DIFF_GPU_FAST(*args)[0]))
    wrong = []

    def work(args, Z):
        for _ in range(8):
            if not np.array_equal(m.gassemble_ZV_EFIE_RWG_DIFF_GPU_FAST(*args)[0], Z):
                wrong.append(len(Z))

    threads = [threading.Thread(target=work, args=c) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
