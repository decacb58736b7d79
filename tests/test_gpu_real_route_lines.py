"""Real-harmonic transforms of HP_REAL plans on both sides of the lines between
the direct sums and the complex rows: the two sides agree function by function
(1e-12 relative L2, the bar of the library's real-harmonic tests), and both with
the oracle."""
import numpy as np
import pytest

from oracle import real_harmonics as rh

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm((np.asarray(a) - np.asarray(b)).ravel()) / np.linalg.norm(np.asarray(b).ravel()))


def direct_and_rows(call, x, nb):
    """The first nb functions as one batch (the last size of the direct sums) and with one more."""
    a, b = call(x[..., :nb]), call(x[..., :nb + 1])
    for k in range(nb):
        assert rel(b[..., k], a[..., k]) < 1e-12
    return b


@pytest.mark.parametrize('B,nb', [(2, 450), (3, 200), (5, 72), (6, 50), (7, 36), (8, 16)])
def test_forward(hp, B, nb):
    f = np.random.default_rng(B).standard_normal((2 * B, 2 * B, 2 * B, nb + 1))
    F = direct_and_rows(hp.Plan(B, 2, 2, hp.HP_FP64, hp.HP_REAL).real_forward, f, nb)
    for k in (0, nb):
        assert rel(F[..., k], rh.forward(f[..., k])) < 1e-12


@pytest.mark.parametrize('B,nb', [(2, 1000), (3, 444), (5, 160), (6, 72), (7, 53), (8, 40)])
def test_backward(hp, B, nb):
    F = np.random.default_rng(B).standard_normal((2 * B - 1, 2 * B - 1, B, nb + 1))
    keep = np.maximum(*np.abs(np.mgrid[1 - B:B, 1 - B:B]))[:, :, None] <= np.arange(B)
    f = direct_and_rows(hp.Plan(B, 2, 2, hp.HP_FP64, hp.HP_REAL).real_backward, F, nb)
    for k in (0, nb):
        assert rel(f[..., k], rh.backward(F[..., k] * keep)) < 1e-12


def test_first_bandlimit_without_direct_sums(hp):
    f = np.random.default_rng(9).standard_normal((18, 18, 18, 1))
    plan = hp.Plan(9, 2, 2, hp.HP_FP64, hp.HP_REAL)
    F = plan.real_forward(f)
    assert rel(F[..., 0], rh.forward(f[..., 0])) < 1e-12
    assert rel(plan.real_backward(F)[..., 0], rh.backward(rh.forward(f[..., 0]))) < 1e-12
