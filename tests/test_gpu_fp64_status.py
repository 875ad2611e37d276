"""The status of an FP64 energy shows the checks of its tensor-core inverses:
the largest accepted residual (at most 1e-9) where they ran, nothing on the
FP64 pipe."""
import dataclasses

import pytest

from skkr_budapest_gb300 import api
from skkr_budapest_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _problem(kind):
    if kind == "bdg":
        return W.energy_problem(W.bdg_bcc(nsets=[1] * 64, lmax=2), 10)                             # 144 rows
    if kind == "rel":
        return W.energy_problem(dataclasses.replace(W.rel_bcc(nsets=[1] * 24), lmax=2), 8)         # 72
    return W.energy_problem(dataclasses.replace(W.plain_fcc(nset=2), pl=4 if kind == "fcc" else 2), 8)  # 36, 18


def _status(ep, pipe=False):
    ctx = api.Context.for_problem(ep, "fp64")
    try:
        ctx.set_fp64_pipe(pipe)
        r = ctx.cpacoord(ep)
    finally:
        ctx.close()
    return r


@pytest.mark.parametrize("kind", ["fcc", "rel", "bdg"])
def test_accepted_residual_is_reported(kind):
    r = _status(_problem(kind))
    assert 0.0 < r["max_refine_resid"] <= 1e-9 and r["inv_fallbacks"] >= 0


@pytest.mark.parametrize("kind,pipe", [("rel", True), ("bdg", True), ("small", False)])
def test_the_pipe_has_none(kind, pipe):
    r = _status(_problem(kind), pipe)
    assert r["max_refine_resid"] == 0.0 and r["inv_fallbacks"] == 0 and r["inv_refined"] == 0
