"""Results brought to pageable host memory in pieces by several threads: every
byte of Z arrives, and none outside it, whatever the destination's alignment,
from sizes below the threshold of that path to several rounds of its buffers."""
import ctypes as C
import importlib

import numpy as np
import pytest

import efie_oracle as eo
from conftest import pkg, small_design

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.mark.parametrize("cells", [(8, 6, 12, 10), (10, 8, 14, 13), (11, 9, 15, 15), (22, 17, 27, 27)])
@pytest.mark.parametrize("offset", [0, 16, 2 * MB - 16])
def test_z_arrives_whole_at_any_alignment(cells, offset):
    m = pkg()
    nat = importlib.import_module(m.__name__ + "._native")
    api = importlib.import_module(m.__name__ + ".api")
    npx, npy, ngx, ngy = cells
    p = eo.build_problem(small_design(npx=npx, npy=npy, ngx=ngx, ngy=ngy))
    r, d = p["rwg"], p["design"]
    omega, k, _, _ = eo.physics(2.5e9, d.mu, d.eps)
    mar = api._Marshal()
    mesh = mar.mesh(p["V"], p["F"], r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"],
                    r["rm"], r["Ap"], r["Am"], r["len"])
    Ne = r["Ne"]
    exc = np.array([p["patchEdge"], p["groundEdge"], d.V0, p["spread"], 0.2])
    V = np.zeros(Ne, np.complex128)
    n = 16 * Ne * Ne
    buf = np.full(n + 6 * MB, 0xA5, np.uint8)
    base = -buf.ctypes.data % (2 * MB) + offset   # from a 2 MB boundary
    nat.check(nat.lib().efie_gassemble_zv(nat.context(), C.byref(mesh), api._cscalar(k), omega, d.mu, api._cscalar(d.eps),
                                          exc.ctypes.data_as(nat.c_double_p), buf.ctypes.data + base, V.ctypes.data))
    Z = buf[base:base + n].view(np.complex128).reshape(Ne, Ne)
    assert np.all(buf[:base] == 0xA5) and np.all(buf[base + n:] == 0xA5)
    # the centroid matrix is symmetric to rounding, so a missing or misplaced piece shows
    assert np.abs(Z - Z.T).max() <= 1e-12 * np.abs(Z).max()
    assert np.abs(np.diag(Z)).min() > 0
