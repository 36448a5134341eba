"""The staging buffers of large results belong to a context and grow with its
results: matrices of rising and falling size through contexts of their own
equal those of the process's context."""
import ctypes as C
import importlib

import numpy as np
import pytest

import efie_oracle as eo
from conftest import pkg, small_design

pytestmark = pytest.mark.gpu
CELLS = [(4, 3, 6, 6), (10, 8, 14, 13), (16, 12, 20, 20), (11, 9, 15, 15), (22, 17, 27, 27), (10, 8, 14, 13)]


def _z(ctx, p):
    m = pkg()
    nat = importlib.import_module(m.__name__ + "._native")
    api = importlib.import_module(m.__name__ + ".api")
    r, d = p["rwg"], p["design"]
    omega, k, _, _ = eo.physics(2.5e9, d.mu, d.eps)
    mar = api._Marshal()
    mesh = mar.mesh(p["V"], p["F"], r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"],
                    r["rm"], r["Ap"], r["Am"], r["len"])
    exc = np.array([p["patchEdge"], p["groundEdge"], d.V0, p["spread"], 0.2])
    Z, V = np.full((r["Ne"], r["Ne"]), np.nan, np.complex128, order="F"), np.zeros(r["Ne"], np.complex128)
    nat.check(nat.lib().efie_gassemble_zv(ctx, C.byref(mesh), api._cscalar(k), omega, d.mu, api._cscalar(d.eps),
                                          exc.ctypes.data_as(nat.c_double_p), Z.ctypes.data, V.ctypes.data))
    return Z


def test_results_of_any_size_through_contexts_of_their_own():
    nat = importlib.import_module(pkg().__name__ + "._native")
    problems = [eo.build_problem(small_design(npx=a, npy=b, ngx=c, ngy=d)) for a, b, c, d in CELLS]
    want = [_z(nat.context(), p) for p in problems]
    for order in (range(len(CELLS)), reversed(range(len(CELLS)))):
        ctx = nat.new_context()
        for i in order:
            assert np.array_equal(_z(ctx, problems[i]), want[i])
        nat.destroy_context(ctx)
