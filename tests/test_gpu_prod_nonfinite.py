"""A NaN or infinite coefficient in a product reaches the entries it has a part
in, |m - m1| <= lmax and |n - n1| <= lmax, and no others: those equal the
product with the coefficient set to zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def coefficients(B, seed):
    rng = np.random.default_rng(seed)
    k = np.abs(np.arange(2 * B - 1) - (B - 1))
    keep = (np.maximum(k[:, None], k[None, :])[:, :, None] <= np.arange(B)) / (2.0 * np.arange(B) + 1)
    return (rng.standard_normal((2 * B - 1, 2 * B - 1, B)) + 1j * rng.standard_normal((2 * B - 1, 2 * B - 1, B))) * keep


@pytest.mark.parametrize('bad', [np.nan, np.inf])
@pytest.mark.parametrize('left', [True, False])
@pytest.mark.parametrize('B', [2, 3, 4, 6, 7, 12, 13, 32])
def test_bad_coefficient_stays_in_its_support(hp, B, left, bad):
    lmax = B - 1
    m = np.arange(-lmax, B)
    for m1, n1 in [(lmax, -lmax), (0, lmax), (-lmax, 0), (1, -1)]:
        F, G = coefficients(B, 1), coefficients(B, 2)
        X = F if left else G
        X[m1 + lmax, n1 + lmax, lmax] = 0
        clean = hp.fftSO3_prod(F, G)
        X[m1 + lmax, n1 + lmax, lmax] = bad
        out = hp.fftSO3_prod(F, G)
        free = (np.abs(m - m1) > lmax)[:, None] | (np.abs(m - n1) > lmax)[None, :]
        assert np.array_equal(out[free], clean[free])
        keep = np.maximum(np.abs(m)[:, None], np.abs(m)[None, :])[:, :, None] <= np.arange(B)
        assert not np.isfinite(out[~free][keep[~free]]).any()
