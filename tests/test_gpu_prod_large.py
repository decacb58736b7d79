"""The Clebsch-Gordan product at bandlimits beyond the direct oracle's reach: the
degrees below B of the pointwise product of the two functions, through the
oracle's transforms at the bandlimit (3B - 1) / 2 that holds them exactly.
Tolerance 1e-12 relative L2, the bar of the library's other product tests."""
import numpy as np
import pytest

from oracle import so3

pytestmark = pytest.mark.gpu


def coefficients(B, seed):
    rng = np.random.default_rng(seed)
    k = np.abs(np.arange(2 * B - 1) - (B - 1))
    keep = (np.maximum(k[:, None], k[None, :])[:, :, None] <= np.arange(B)) / (2.0 * np.arange(B) + 1)
    return (rng.standard_normal((2 * B - 1, 2 * B - 1, B)) + 1j * rng.standard_normal((2 * B - 1, 2 * B - 1, B))) * keep


def pointwise(F, G, B):
    Bg = (3 * B - 1) // 2
    o = Bg - B

    def function(X):
        P = np.zeros((2 * Bg - 1, 2 * Bg - 1, Bg, 1, 1), complex)
        P[o:o + 2 * B - 1, o:o + 2 * B - 1, :B, 0, 0] = X
        return so3.ifftSO3R_backward(P, real=False)

    H = so3.fftSO3R_forward(function(F) * function(G))
    return H[o:o + 2 * B - 1, o:o + 2 * B - 1, :B, 0, 0]


@pytest.mark.parametrize('B', [9, 11, 16, 20, 25, 31, 32])
def test_product(hp, B):
    F, G = coefficients(B, 1), coefficients(B, 2)
    keep = np.maximum(*np.abs(np.mgrid[1 - B:B, 1 - B:B]))[:, :, None] <= np.arange(B)
    ref = pointwise(F, G, B) * keep
    out = hp.fftSO3_prod(F, G)
    assert np.linalg.norm((out - ref).ravel()) < 1e-12 * np.linalg.norm(ref.ravel())
