"""A prepack's caches and nearMat are laid out on the device: the assembly
from them matches the FP64 oracle for symmetric, one-sided, empty and full near
relations, and for triangle counts off the scan's block sizes."""
import numpy as np
import pytest

import efie_oracle as eo
import oracle_c as oc
from conftest import pkg, small_design

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(1, 1, 1, 1), (4, 3, 6, 6), (7, 5, 9, 11)])
@pytest.mark.parametrize("near", ["as_built", "one_sided", "none", "all", "values", "one_sided_late"])
def test_assembly_from_any_near_matrix(cells, near):
    m = pkg()
    npx, npy, ngx, ngy = cells
    p = eo.build_problem(small_design(npx=npx, npy=npy, ngx=ngx, ngy=ngy))
    pre = dict(p["prepack"])
    nm = np.array(pre["nearMat"], order="F")
    if near == "one_sided":
        nm[np.triu_indices(nm.shape[0], 1)] = 0
    elif near == "none":
        nm[:] = 0
    elif near == "all":
        nm[:] = 1
    elif near == "values":
        nm[nm != 0] = 7   # any non-zero byte means near
    elif near == "one_sided_late":
        nm[-1, 0] = 1 - nm[-1, 0]   # a single entry without its mirror image
    pre["nearMat"] = nm
    r, d = p["rwg"], p["design"]
    omega, k, _, _ = eo.physics(2.5e9, d.mu, d.eps)
    exc = np.array([p["patchEdge"], p["groundEdge"], d.V0, p["spread"]])
    Z, _ = m.ggassemble_ZV_EFIE_RWG_DIFF_GPU_FAST(
        p["V"], p["F"], r["edge"], r["plusTri"], r["minusTri"], r["plusSign"], r["minusSign"], r["rp"], r["rm"],
        r["Ap"], r["Am"], r["len"], pre, k, omega, d.mu, d.eps, exc)
    Zo = oc.assemble_z(r, pre, k, omega, d.mu, d.eps)
    assert np.abs(Z - Zo).max() <= 1e-12 * np.abs(Zo).max()
