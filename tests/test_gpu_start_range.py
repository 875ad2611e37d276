"""The FP32 start of the inverses over its range of scales: |pivot|^2 and its
reciprocal stay FP32 numbers down to subnormal ones, so a matrix whose
elements are near 2^63.3 (|pivot|^2 near 2^126.6, its reciprocal subnormal)
starts as any other and is accepted after the Newton steps, not handed to the
FP64 elimination."""
import numpy as np
import pytest

from skkr_budapest_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 32, 64, 96, 128])
@pytest.mark.parametrize("log2", [-62.0, -30.0, 0.0, 40.0, 63.3])
def test_scaled_matrices_are_accepted(n, log2):
    rng = np.random.default_rng(n)
    noise = rng.normal(size=(4, n, n)) + 1j * rng.normal(size=(4, n, n))
    a = (np.eye(n) + 0.02 / np.sqrt(n) * noise) * 2.0 ** log2
    x, resid = native.zinv_batch(a, precision="mixed")
    ref = np.linalg.inv(a)
    # (condition below 1.2: a few hundred roundings of the product sums)
    assert (np.linalg.norm(x - ref, axis=(1, 2)) < 1e-14 * np.linalg.norm(ref, axis=(1, 2))).all()
    # the largest accepted residual: 0 when every item went to the FP64 elimination, and NaN or more than the limit never
    assert 0.0 < resid <= 1e-6
