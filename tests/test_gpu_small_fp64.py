"""FP64 products and inverses of small blocks at the edges of their thread
layouts (16, 32, 48, 64 rows), against numpy."""
import numpy as np
import pytest

from skkr_budapest_gb300 import native

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def crand(rng, *s):
    return rng.normal(size=s) + 1j * rng.normal(size=s)


@pytest.mark.parametrize("batch", [1, 400])
@pytest.mark.parametrize("n", [1, 2, 9, 16, 17, 18, 31, 32, 33, 48, 49, 63, 64, 65])
def test_products(n, batch):
    rng = np.random.default_rng(n)
    a, b = crand(rng, batch, n, n), crand(rng, batch, n, n)
    c = native.zgemm_batch(a, b)
    # two roundings per real term, n complex terms, on either side
    assert (np.abs(c - a @ b) <= 8 * n * EPS * (np.abs(a) @ np.abs(b))).all()


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 18, 24, 25, 32, 33, 48, 49, 64, 65])
def test_inverses(n):
    rng = np.random.default_rng(1000 + n)
    a = crand(rng, 40, n, n)
    a[3] = a[3][:, ::-1] * np.eye(n)[::-1]          # a permutation of a diagonal: every step pivots off the diagonal
    x = native.gjinv_batch(a)
    for i in range(len(a)):
        # Gauss-Jordan with row pivoting: n eps cond times a modest growth
        tol = 20 * n * EPS * np.linalg.cond(a[i])
        assert np.linalg.norm(x[i] - np.linalg.inv(a[i])) <= tol * np.linalg.norm(x[i]), i


@pytest.mark.parametrize("scale", [1e-200, 1e200])
def test_inverse_where_squares_leave_the_range(scale):
    rng = np.random.default_rng(7)
    a = crand(rng, 3, 20, 20)
    x = native.gjinv_batch(a * scale)
    ref = np.linalg.inv(a)
    assert np.linalg.norm(x * scale - ref) < 1e-11 * np.linalg.norm(ref)


def test_nan_matrix_leaves_its_neighbours_alone():
    rng = np.random.default_rng(8)
    a = crand(rng, 3, 18, 18)
    ref = np.linalg.inv(a)
    a[1, 4, :] = np.nan
    x = native.gjinv_batch(a)
    assert np.isnan(x[1]).any()
    assert np.linalg.norm(x[[0, 2]] - ref[[0, 2]]) < 1e-11 * np.linalg.norm(ref[[0, 2]])
