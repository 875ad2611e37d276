"""FP64 contexts above 32 rows, whose products and inverses run on the tensor
cores with eight slices per operand: against the oracle at the FP64 path's
1e-10, at the sizes where the form changes (33 rows and more, one or two
depth halves, the block inverse above 128, odd sizes above it)."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from skkr_budapest_gb300 import api
from skkr_budapest_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _problem(kind, pl, lmax, ie=10, nprc=3):
    if kind == "bdg":
        spec = W.bdg_bcc(nsets=[1] * 64, lmax=lmax, pl=pl)
    elif kind == "rel":
        spec = W.rel_bcc(nsets=[2] * 24)
    else:
        spec = W.plain_fcc(nset=2)
    spec = dataclasses.replace(spec, pl=pl, lmax=lmax, nprc=nprc)
    return W.energy_problem(spec, ie)


# rows n_PL = pl x basis: 27 (FP64 pipe), 36, 54, 64, 72, 128; 135 (odd above
# 128: Gauss-Jordan), 144 (two halves of 72) and 256
@pytest.mark.parametrize("kind,pl,lmax,n", [("fcc", 3, 2, 27), ("fcc", 4, 2, 36), ("rel", 3, 2, 54), ("rel", 2, 3, 64),
                                            ("rel", 4, 2, 72), ("rel", 4, 3, 128), ("fcc", 15, 2, 135),
                                            ("bdg", 4, 2, 144), ("bdg", 4, 3, 256)])
def test_fp64_context_matches_the_oracle(kind, pl, lmax, n):
    ep = _problem(kind, pl, lmax, nprc=1 if n == 135 else 3)
    assert ep.n_pl == n
    g, o = api.cpacoord(ep), O.cpacoord(ep, nthreads=8)
    assert g["status"] == 0 and o["status"] == 0
    assert g["max_dec_iters"] == o["max_dec_iters"] and g["cpa_iterations"] == o["cpa_iterations"]
    for key in ("tauc", "taua", "taub", "tminv"):
        assert rel(g[key], o[key]) < 1e-10, (key, rel(g[key], o[key]))


def test_graphs_and_host_loop_agree_bit_for_bit():
    ep = _problem("bdg", 4, 2)
    out = []
    for on in (True, False):
        ctx = api.Context.for_problem(ep, "fp64")
        try:
            ctx.set_graphs(on)
            out.append(ctx.cpacoord(ep))
        finally:
            ctx.close()
    assert np.array_equal(out[0]["tauc"], out[1]["tauc"])


def test_a_nan_energy_is_reported_not_returned():
    ep = _problem("rel", 4, 2)
    t = ep.tminvl.copy()
    t[0, 1, 2] = np.nan
    r = api.cpacoord(dataclasses.replace(ep, tminvl=t), check=False)
    assert r["status"] != 0
