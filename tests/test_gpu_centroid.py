"""The one-point sweep as a plan like any other, and with RWG areas that are
not their triangles' (which keeps the assembly that weighs each side by its own
area), against the FP64 oracle of the centroid rule."""
import numpy as np
import pytest

import efie_oracle as eo
import oracle_c as oc
from conftest import config1_design, pkg, small_design

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("areas", ["triangles", "scaled"])
@pytest.mark.parametrize("design,nf", [("small", 1), ("small", 4), ("small", 9), ("lossy", 7), ("config1", 21)])
def test_centroid_sweep_matches_oracle(design, nf, areas):
    m = pkg()
    d = config1_design() if design == "config1" else small_design()
    if design == "lossy":
        d.eps = eo.EPS0 * 3.0 * (1 - 0.03j)
    p = eo.build_problem(d)
    r = {k: np.array(v, copy=True) for k, v in p["rwg"].items()}
    if areas == "scaled":
        r["Ap"] *= 1.001
    freqs = np.linspace(2e9, 3e9, nf)
    st = {}
    Zin, S11 = m.patch_sweep_cuda(p["V"], p["F"], r["edge"], r["plusTri"], r["minusTri"], r["plusSign"],
                                  r["minusSign"], r["rp"], r["rm"], r["Ap"], r["Am"], r["len"], freqs, d.mu, d.eps,
                                  p["patchEdge"], p["groundEdge"], d.V0, p["spread"], d.Z0, stats=st)
    assert st["n_fp64_fallback"] == 0 and st["max_relres"] <= 1e-10
    for j in {0, nf // 2, nf - 1}:
        omega, k, _, _ = eo.physics(freqs[j], d.mu, d.eps)
        Z = oc.assemble_centroid(p["V"], p["F"], r, 0.2, k, omega, d.mu, d.eps)
        x = np.linalg.solve(Z, p["b"].astype(complex))
        zo = d.V0 / (x[p["patchEdge"] - 1] - x[p["groundEdge"] - 1])
        assert abs(Zin[j] - zo) <= 1e-6 * abs(zo)
        assert abs(S11[j] - (zo - d.Z0) / (zo + d.Z0)) <= 1e-6
