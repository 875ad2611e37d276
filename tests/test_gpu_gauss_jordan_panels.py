"""The FP32 Gauss-Jordan in panels of eight rows (the start of every
split-precision inverse) through zinv_batch: sizes around a panel, a size
class and the largest, matrices that need pivoting in every row, and batches
in which one item is lost."""
import numpy as np
import pytest

from skkr_budapest_gb300 import native

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 7, 8, 9, 31, 32, 33, 56, 63, 64, 65, 72, 95, 96, 97, 120, 127, 128]


def crand(rng, *s):
    return rng.normal(size=s) + 1j * rng.normal(size=s)


def close(x, a):
    """Both inverses carry a few cond(A) x 1e-16: 1e-14 cond, by each matrix's own."""
    for xi, ai in zip(x, a):
        ref = np.linalg.inv(ai)
        err = np.linalg.norm(xi - ref) / np.linalg.norm(ref)
        if err > 1e-14 * np.linalg.cond(ai):
            return False
    return True


@pytest.mark.parametrize("n", SIZES)
def test_sizes(n):
    rng = np.random.default_rng(n)
    a = crand(rng, 5, n, n) + 3 * np.eye(n)
    x, resid = native.zinv_batch(a, precision="mixed")
    assert close(x, a) and resid < 1e-5


@pytest.mark.parametrize("n", [8, 33, 64, 90, 128])
def test_pivots_away_from_the_diagonal(n):
    """Permuted rows leave no usable pivot on the diagonal."""
    rng = np.random.default_rng(100 + n)
    a = np.stack([(crand(rng, n, n) * 0.1 / np.sqrt(n) + np.diag(np.exp(2j * np.pi * rng.random(n))))[rng.permutation(n)]
                  for _ in range(4)])
    x, resid = native.zinv_batch(a, precision="mixed")
    assert close(x, a) and resid < 1e-5


@pytest.mark.parametrize("n", [20, 64, 100, 128])
def test_a_lost_item_leaves_the_others(n):
    """A NaN, an infinite or a singular item ends as non-finite; its neighbours
    are inverted as if alone."""
    rng = np.random.default_rng(200 + n)
    a = crand(rng, 6, n, n) + 3 * np.eye(n)
    b = a.copy()
    b[1, n // 2, n // 3] = np.nan
    b[3] = np.inf
    b[4] = 0.0
    x, _ = native.zinv_batch(b, precision="mixed")
    good = [0, 2, 5]
    assert close(x[good], a[good])
    assert not np.isfinite(x[[1, 3, 4]]).all(axis=(1, 2)).any()
