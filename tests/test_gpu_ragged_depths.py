"""B operands formed in the product against staged ones, bit for bit, in
energies whose block rows are no multiple of 16 and that do run on the tensor
cores (28 rows and more with split precision, 33 and more in FP64): the
stacked tiles up to 64 rows and the plain ones above; the numbers against the
oracle."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from skkr_budapest_gb300 import api
from skkr_budapest_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _problem(n):
    if n in (54, 90):
        spec, ie = dataclasses.replace(W.rel_pl3_l2(), pl=n // 18, nsets=[2] * 20), 12
    else:
        spec, ie = dataclasses.replace(W.plain_fcc(nset=2), pl=n // 9), 8
    ep = W.energy_problem(dataclasses.replace(spec, nprc=2), ie)
    assert ep.n_pl == n
    return ep


@pytest.mark.parametrize("n", [36, 45, 54, 63, 72, 81, 90, 117])
@pytest.mark.parametrize("precision,tol", [("mixed", 1e-9), ("fp64", 1e-10)])
def test_fused_and_staged_operands_agree(n, precision, tol):
    ep = _problem(n)
    out = []
    for fused in (True, False):
        ctx = api.Context.for_problem(ep, precision)
        try:
            ctx.set_fused_split(fused)
            out.append(ctx.cpacoord(ep))
        finally:
            ctx.close()
        assert out[-1]["status"] == 0 and out[-1]["max_refine_resid"] > 0.0  # (the tensor cores ran)
    for key in ("tauc", "taua", "taub", "tminv"):
        assert np.array_equal(out[0][key], out[1][key]), key
    o = O.cpacoord(ep, nthreads=8)
    assert np.linalg.norm(out[0]["tauc"] - o["tauc"]) < tol * np.linalg.norm(o["tauc"])
