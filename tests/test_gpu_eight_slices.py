"""Products with eight slices, the tensor-core form of FP64: the error of an
output is that of the digits left out, also where the output is far below the
scales of its row and column (entries graded along the summed index, the large
of one operand against the small of the other).

The bound, in units of sigma_i tau_j (powers of two above the row's and the
column's largest real or imaginary part), per real sum of K' = 2K terms and
for eight-bit digits, uniform in [-127, 128] (variance 5461): the seven slice
pairs of level 8 leave 2^-78 5461 sqrt(7 K'), quantising the operands 2^-62;
together 2^-60.15 at K = 128.  Eight times that (some 1e5 outputs are looked
at) is 2^-57.  Seven-bit digits (K > 128; variance 1365): 2^-68 1365
sqrt(7 K') and 2^-53.5 give 2^-51.5 at K = 256, bound 2^-48.5.  The
rounding to double comes on top, of a sum that is itself rounded to half of
that place where it is largest: 1.5 x 2^-53 of the output."""
import numpy as np
import pytest

from skkr_budapest_gb300 import native

pytestmark = pytest.mark.gpu


def scale(m, axis):
    big = np.maximum(np.abs(m.real), np.abs(m.imag)).max(axis=axis)
    return np.where(big > 0, np.ldexp(1.0, np.frexp(big)[1]), 0.0)


@pytest.mark.parametrize("n", [1, 33, 54, 64, 65, 96, 128, 200])
@pytest.mark.parametrize("decades", [0, 6, 12, 18])
def test_error_is_that_of_the_digits_left_out(n, decades):
    rng = np.random.default_rng(1000 * decades + n)
    g = np.logspace(0, -decades, n)
    m = 1 if n > 96 else 2
    a = (rng.normal(size=(m, n, n)) + 1j * rng.normal(size=(m, n, n))) * g[None, None, :]
    b = (rng.normal(size=(m, n, n)) + 1j * rng.normal(size=(m, n, n))) * g[::-1][None, :, None]
    c = native.zgemm_batch(a, b, precision="mixed", slices=8)
    for x, y, z in zip(a, b, c):
        ref = x.astype(np.clongdouble) @ y.astype(np.clongdouble)
        st = scale(x, 1)[:, None] * scale(y, 0)[None, :]
        bound = 2.0 ** -57 if n <= 128 else 2.0 ** -48.5
        for p, q in ((z.real, ref.real), (z.imag, ref.imag)):
            assert (np.abs(p - q) <= bound * st + 1.5 * 2.0 ** -53 * np.abs(q)).all()
