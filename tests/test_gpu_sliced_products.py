"""The persistent sliced product at the edges of its tiles (128 rows, 32
complex columns, k-blocks of 16) and rings, against numpy, and its handling of
infinities and NaN."""
import numpy as np
import pytest

from skkr_budapest_gb300 import native

pytestmark = pytest.mark.gpu


def crand(rng, *s):
    return rng.normal(size=s) + 1j * rng.normal(size=s)


def bound(a, b, slices):
    """Largest error of C_ij, from the largest |Re|, |Im| of row i of A and of
    column j of B (their power-of-two scales are below twice these): 2K real
    terms, each off by both operands' rounding and the dropped slice pairs,
    (S + 2) 2^(-DB S) of the scales; the levels past the sixth round into its
    unit; and numpy's own rounding."""
    k = a.shape[-1]
    db = 8 if k <= 128 else 7
    ra = np.maximum(np.abs(a.real), np.abs(a.imag)).max(-1)
    cb = np.maximum(np.abs(b.real), np.abs(b.imag)).max(-2)
    per_term = (slices + 2) * 2.0 ** (-db * slices) + 2.0 ** -52
    unit = 2.0 ** (-2 * (db - 1) - 5 * db) if slices > 6 else 0.0
    return 4.0 * ra[..., :, None] * cb[..., None, :] * (2 * k * per_term + unit)


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 64, 65, 127, 128, 129, 200, 256])
@pytest.mark.parametrize("slices", [3, 4, 5, 6, 7, 8])
def test_products_at_tile_edges(n, slices):
    rng = np.random.default_rng(100 * n + slices)
    batch = 200 if n in (33, 65) else 3          # 200: several tiles for every SM
    a, b = crand(rng, batch, n, n), crand(rng, batch, n, n)
    c = native.zgemm_batch(a, b, precision="mixed", slices=slices)
    err = np.maximum(np.abs((c - a @ b).real), np.abs((c - a @ b).imag))
    assert (err <= bound(a, b, slices)).all(), (err / bound(a, b, slices)).max()


@pytest.mark.parametrize("slices", [3, 6, 8])
def test_infinities_and_nan_stay_in_their_row_and_column(slices):
    rng = np.random.default_rng(slices)
    a, b = crand(rng, 3, 40, 40), crand(rng, 3, 40, 40)
    ref = a @ b
    a[1, 5, 7] = np.nan
    a[1, 6, 0] = np.inf
    b[1, 3, 35] = complex(0.0, -np.inf)
    c = native.zgemm_batch(a, b, precision="mixed", slices=slices)
    bad = np.zeros((3, 40, 40), bool)
    bad[1, 5:7, :] = True
    bad[1, :, 35] = True
    assert np.isnan(c[bad]).all()
    assert np.isfinite(c[~bad]).all()
    assert np.abs((c - ref)[~bad]).max() < (1e-4 if slices == 3 else 1e-10)
