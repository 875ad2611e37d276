"""Screened to physical tau (phystau, phystau2) at every basis size, from one
row to the 64 of the superconducting lmax = 3 basis, against the matrix
formula in numpy, and from several threads at once."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from skkr_budapest_gb300 import native

pytestmark = pytest.mark.gpu


def crand(rng, *s):
    return rng.normal(size=s) + 1j * rng.normal(size=s)


def basis(irel, lmax):
    """l of every basis function, and the number of screening constants (BdG: electrons, then holes)."""
    if irel == 0:
        return np.repeat(np.arange(lmax + 1), 2 * np.arange(lmax + 1) + 1), lmax + 1
    l = np.concatenate([[q] * (2 if q == 0 else 4 * q + 2) for q in range(lmax + 1)])
    return (np.concatenate([l, l + lmax + 1]), 2 * (lmax + 1)) if irel == 2 else (l, lmax + 1)


def bound(l, t, r):
    """Two sums of n terms: 4 n eps of the product of the norms."""
    return 4 * len(t) * 2.3e-16 * np.linalg.norm(l) * np.linalg.norm(t) * np.linalg.norm(r)


@pytest.mark.parametrize("irel", [0, 1, 2])
@pytest.mark.parametrize("lmax", [0, 1, 2, 3])
def test_against_numpy(irel, lmax):
    rng = np.random.default_rng(10 * irel + lmax)
    l, nal = basis(irel, lmax)
    n = len(l)
    tau, t1, t2 = crand(rng, n, n), crand(rng, n, n), crand(rng, n, n)
    a1, a2 = crand(rng, nal), crand(rng, nal)
    one = np.eye(n)
    left, right = one + a1[l][:, None] * t1, one + t1 * a1[l][None, :]
    want = left @ tau @ right - (np.diag(a1[l]) + a1[l][:, None] * t1 * a1[l][None, :])
    assert np.linalg.norm(native.phystau(tau, t1, a1, lmax, irel) - want) < bound(left, tau, right) + 1e-14
    right2 = one + t2 * a2[l][None, :]
    got = native.phystau2(tau, t1, a1, t2, a2, lmax, irel)
    assert np.linalg.norm(got - left @ tau @ right2) < bound(left, tau, right2) + 1e-14


def test_threads():
    rng = np.random.default_rng(7)
    l, nal = basis(1, 3)
    n = len(l)
    args = [(crand(rng, n, n), crand(rng, n, n), crand(rng, nal)) for _ in range(40)]
    alone = [native.phystau(*a, 3, 1) for a in args]
    with ThreadPoolExecutor(8) as ex:
        both = list(ex.map(lambda a: native.phystau(*a, 3, 1), args))
    assert all(np.array_equal(x, y) for x, y in zip(alone, both))
