"""Sliced products of up to 64 rows, whose real and imaginary parts share one
tile: sizes around its column halves and the odd ones of the interfaces, and a
whole energy with the B operands formed in the product or split first."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from skkr_budapest_gb300 import api, native
from skkr_budapest_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 18, 30, 36, 47, 48, 54, 63])
@pytest.mark.parametrize("slices", [3, 4, 6, 8])
def test_products(n, slices):
    """Row and column scales are below twice the largest parts; 2K terms, each
    off by (S + 2) 2^(-8 S) of the scales, and numpy's rounding; past six
    slices the sums round into the sixth level's unit, 2^-54."""
    rng = np.random.default_rng(10 * n + slices)
    a, b = (rng.normal(size=(160, n, n)) + 1j * rng.normal(size=(160, n, n)) for _ in range(2))
    c = native.zgemm_batch(a, b, precision="mixed", slices=slices)
    ra = np.maximum(np.abs(a.real), np.abs(a.imag)).max(-1)[..., :, None]
    cb = np.maximum(np.abs(b.real), np.abs(b.imag)).max(-2)[..., None, :]
    bound = 4 * ra * cb * (2 * n * ((slices + 2) * 2.0 ** (-8 * slices) + 2.0 ** -52) + 2.0 ** -54)
    d = c - a @ b
    assert (np.maximum(np.abs(d.real), np.abs(d.imag)) <= bound).all()


@pytest.mark.parametrize("pl,lmax", [(2, 2), (3, 2), (2, 3), (4, 1)])
def test_energies_with_either_split(pl, lmax):
    """n = 36, 54, 64 and 32: bit for bit the same, and the oracle's to the split precision's 1e-9."""
    spec = dataclasses.replace(W.rel_pl3_l2(), pl=pl, lmax=lmax, nsets=[3] * 20)
    ep = W.energy_problem(spec, 12)
    out = []
    for fused in (True, False):
        ctx = api.Context.for_problem(ep, "mixed")
        try:
            ctx.set_fused_split(fused)
            out.append(ctx.cpacoord(ep))
        finally:
            ctx.close()
    assert np.array_equal(out[0]["tauc"], out[1]["tauc"])
    o = O.cpacoord(ep, nthreads=8)
    assert np.linalg.norm(out[0]["tauc"] - o["tauc"]) < 1e-9 * np.linalg.norm(o["tauc"])
