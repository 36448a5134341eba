"""The one-point sweep of a mesh most of whose triangles carry no basis
function: its memory follows the unknowns, not the triangles' pairs."""
import numpy as np
import pytest

import efie_oracle as eo
from conftest import pkg, small_design

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("idle", [0, 400, 600000])   # the pairs of 600000 triangles do not fit the device
def test_idle_triangles_change_nothing(idle):
    m = pkg()
    p = eo.build_problem(small_design())
    r, d = p["rwg"], p["design"]
    F = np.asfortranarray(np.vstack([p["F"], np.tile(p["F"][:1], (idle, 1))]))
    tail = [r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"], r["rm"], r["Ap"], r["Am"],
            r["len"], d.freqs, d.mu, d.eps, p["patchEdge"], p["groundEdge"], d.V0, p["spread"], d.Z0]
    Z0 = m.patch_sweep_cuda(p["V"], p["F"], *tail)[0]
    Z = m.patch_sweep_cuda(p["V"], F, *tail)[0]
    assert np.max(np.abs(Z - Z0) / np.abs(Z0)) <= 1e-6   # the sweeps' bound: 400 and 600000 take another assembly
