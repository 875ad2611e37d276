"""Split-precision contexts of small blocks, which run on the FP64 pipe: the
FP64 context's results bit for bit up to 27 rows, the oracle's to 1e-9 on
both sides of the line and for BdG (whose layout differs: 1e-10 of FP64's)."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from skkr_budapest_gb300 import api
from skkr_budapest_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,pl,lmax,n", [("fcc", 1, 1, 4), ("fcc", 2, 2, 18), ("fcc", 3, 2, 27), ("fcc", 2, 3, 32),
                                            ("rel", 1, 2, 18), ("bdg", 1, 1, 16)])
def test_small_blocks(kind, pl, lmax, n):
    spec = {"fcc": lambda: W.plain_fcc(nset=3), "rel": lambda: W.rel_bcc(nsets=[3] * 24),
            "bdg": lambda: W.bdg_bcc(nsets=[2] * 64, lmax=lmax, pl=pl)}[kind]()
    ep = W.energy_problem(dataclasses.replace(spec, pl=pl, lmax=lmax), 8)
    assert ep.n_pl == n
    g, f, o = api.cpacoord(ep, "mixed"), api.cpacoord(ep), O.cpacoord(ep, nthreads=8)
    for key in ("tauc", "taua"):
        if n <= 27 and kind != "bdg":
            assert np.array_equal(g[key], f[key])
        assert np.linalg.norm(g[key] - f[key]) < 1e-10 * np.linalg.norm(f[key])
        assert np.linalg.norm(g[key] - o[key]) < 1e-9 * np.linalg.norm(o[key])
