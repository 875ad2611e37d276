"""FP64 contexts above 32 rows whose t^-1 is strongly graded over the channels:
the tensor cores' eight slices hold elements relative to their row's or
column's largest, so such blocks run on the FP64 pipe, and the small elements
of tau keep FP64's digits.  One k point and the identity alone, so that no
element of tau vanishes by symmetry."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from skkr_budapest_gb300 import api
from skkr_budapest_gb300 import workloads as W

pytestmark = pytest.mark.gpu
K = np.array([[0.11, 0.07]])


def _spec(kind):
    if kind == "fcc":
        return dataclasses.replace(W.plain_fcc(nset=2), pl=4), 8               # 36 rows
    if kind == "pl3":
        return W.rel_pl3_l2(), 2                                               # 54
    if kind == "rel":
        return dataclasses.replace(W.rel_bcc(nsets=[1] * 24), lmax=2), 8       # 72
    return W.bdg_bcc(nsets=[1] * 64, lmax=2), 10                               # 144


def _problem(kind, power):
    """t^-1 within the highest l scaled by 2^power."""
    spec, ie = _spec(kind)
    ep = W.energy_problem(spec, ie, 1)
    l_of = [l for l in range(ep.lmax + 1) for _ in range((2 * l + 1) * (2 if ep.irel else 1))]
    top = np.array(l_of * (2 if ep.irel == 2 else 1)) == ep.lmax
    up = np.where(top[:, None] & top[None, :], 2.0 ** power, 1.0)
    t = {f: getattr(ep, f) * up for f in ("tminvl", "tminvr", "tminv", "tminva", "tminvb")}
    return dataclasses.replace(ep.with_k(K, np.ones(1)), lg=ep.lg[:1], rg=ep.rg[:1], **t)


def _run(ep, precision="fp64", pipe=False):
    ctx = api.Context.for_problem(ep, precision)
    try:
        ctx.set_fp64_pipe(pipe)
        r = ctx.cpacoord(ep)
    finally:
        ctx.close()
    assert r["status"] == 0
    return r["tauc"]


@pytest.mark.parametrize("kind", ["fcc", "pl3", "rel", "bdg"])
def test_graded_blocks_run_on_the_pipe_even_ones_do_not(kind):
    graded, even = _problem(kind, 16), _problem(kind, 0)
    assert np.array_equal(_run(graded), _run(graded, pipe=True))
    a, b = _run(even), _run(even, pipe=True)
    assert not np.array_equal(a, b)
    assert np.linalg.norm(a - b) < 1e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("kind", ["fcc", "pl3", "rel"])
def test_small_elements_keep_their_digits(kind):
    """The median error of an element against the CPU's elimination: 1e-15 a
    side by FP64, above 1e-12 by slices at this grading."""
    ep = _problem(kind, 20)
    o = O.cpacoord(ep, nthreads=4)["tauc"]
    err = np.abs(_run(ep) - o) / np.abs(o)
    assert np.median(err) < 1e-13


def test_fp64_parts_of_a_split_precision_context():
    """This near the axis the decimation of a split-precision energy runs in
    FP64, with the same choice of engine."""
    ep = _problem("bdg", 16)
    assert abs(ep.ce.imag) < 2e-4
    assert np.array_equal(_run(ep, "mixed"), _run(ep, "mixed", pipe=True))
