"""The batched tau2d sweeps where the diagonal inverses fall into one and
several batches: 1 to 5 principal layers, one class of point-group operations
and one class an operation (t^-1 without the stacking's symmetry), against the
oracle at the FP64 path's 1e-10 and the split precision's 1e-9.  Rows n_PL 18
(FP64 pipe), 36 and 54 (stacked tiles), 72."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from skkr_budapest_gb300 import api
from skkr_budapest_gb300 import synth as S
from skkr_budapest_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _problem(kind, nprc, classes):
    if kind in ("n18", "n36"):
        spec, ie = dataclasses.replace(W.plain_fcc(nset=2), pl=2 if kind == "n18" else 4), 6
    elif kind == "n54":
        spec, ie = dataclasses.replace(W.rel_pl3_l2(), nsets=[2] * 20), 10
    else:
        spec, ie = dataclasses.replace(W.rel_bcc(nsets=[1] * 24), lmax=2), 8
    ep = W.energy_problem(dataclasses.replace(spec, nprc=nprc), ie)
    if classes > 1:
        rng = np.random.default_rng(nprc)
        t = ep.tminv
        e = rng.normal(size=t.shape) + 1j * rng.normal(size=t.shape)
        t = t + 1e-2 * np.abs(t).max() * e / t.shape[-1]
        ep = dataclasses.replace(ep, tminv=t, tminva=t.copy(), tminvb=t.copy())
    return ep


@pytest.mark.parametrize("kind", ["n18", "n36", "n54", "n72"])
@pytest.mark.parametrize("nprc", [1, 2, 4, 5])
@pytest.mark.parametrize("classes", [1, 8])
def test_energy(kind, nprc, classes):
    ep = _problem(kind, nprc, classes)
    o = O.cpacoord(ep, nthreads=8)
    assert o["status"] == 0
    for precision, tol in (("fp64", 1e-10), ("mixed", 1e-9)):
        g = api.cpacoord(ep, precision)
        assert g["status"] == 0
        assert np.linalg.norm(g["tauc"] - o["tauc"]) < tol * np.linalg.norm(o["tauc"]), precision


@pytest.mark.parametrize("kind,nprc,classes", [("n36", 4, 8), ("n36", 5, 1), ("n18", 4, 8), ("n72", 2, 8)])
def test_tauij(kind, nprc, classes):
    ep = _problem(kind, nprc, classes)
    n = ep.nintfc
    a = 6.8 if kind != "n72" else 6.0
    cvec = np.array([[0.5 * ((int(ep.ninprc[0]) + i) % 2) * a] * 2 for i in range(n)])
    pairs = [(0, 0, 0, n - 1), (1, 0, 0, 0), (0, -1, n - 1, 1), (1, 1, n // 2, n // 2)]
    a0 = [op[:2, :2].T.ravel() for op in S.c4v_ops()]
    o = O.tauij(ep, pairs, [a, 0.0], [0.0, a], cvec, a0, nthreads=8)
    scale = max(np.linalg.norm(t) for t in o["tau_ij"])
    for precision, tol in (("fp64", 1e-10), ("mixed", 1e-9)):
        ctx = api.Context.for_problem(ep, precision)
        try:
            g = ctx.tauij(ep, pairs, [a, 0.0], [0.0, a], cvec, a0)
        finally:
            ctx.close()
        for key in ("tau_ij", "tau_ji"):
            for x, y in zip(g[key], o[key]):
                assert np.linalg.norm(x - y) < tol * scale, (precision, key)
