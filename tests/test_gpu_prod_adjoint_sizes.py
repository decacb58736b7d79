"""The node-convolution product and the line passes of the adjoint at the sizes
where they can go wrong, against the oracle: the smallest bandlimits, a group of
outputs that is not full, batches cut into several launches, omega grids off
the 2/3/5 sizes, groups of lines that are not full, 2-D grids above 32 points.
Tolerances: 1e-10 relative L2, the library's FP64 bar (1e-12 for the product,
the bar of its other tests).
"""
import numpy as np
import pytest

from oracle import adjoint as adj
from oracle import pendulum as pd
from oracle import so3

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return float(np.linalg.norm((a - b).ravel()) / max(np.linalg.norm(b.ravel()), 1e-300))


def coefficients(B, xs, seed):
    rng = np.random.default_rng(seed)
    k = np.abs(np.arange(2 * B - 1) - (B - 1))
    keep = (np.maximum(k[:, None], k[None, :])[:, :, None] <= np.arange(B)) / (2.0 * np.arange(B) + 1)
    F = rng.standard_normal((2 * B - 1, 2 * B - 1, B) + xs) + 1j * rng.standard_normal((2 * B - 1, 2 * B - 1, B) + xs)
    return F * keep.reshape(keep.shape + (1,) * len(xs))


@pytest.mark.parametrize('B,batch', [(2, 1), (3, 2), (4, 3), (6, 1), (7, 2), (10, 1)])
def test_product(hp, B, batch):
    F, G = coefficients(B, (batch,), 1), coefficients(B, (batch,), 2)
    out = hp.fftSO3_prod(F, G)
    for b in range(batch):
        assert rel(out[..., b], so3.fftSO3_prod(F[..., b], G[..., b])) < 1e-12


def test_product_ignores_entries_outside_the_degree(hp):
    """Inputs outside |m|, |n| <= l are not coefficients: whatever they hold, the product is the same."""
    F, G = coefficients(5, (), 3), coefficients(5, (), 4)
    bad = F + np.where(F == 0, np.nan, 0)
    assert np.array_equal(hp.fftSO3_prod(bad, G), hp.fftSO3_prod(F, G))


def test_product_batches_over_several_launches(hp):
    """B = 20: one launch holds 188 products; each equals the product formed alone."""
    F, G = coefficients(20, (190,), 5), coefficients(20, (190,), 6)
    out = hp.fftSO3_prod(F, G)
    for b in (0, 187, 188, 189):
        assert np.array_equal(out[..., b], hp.fftSO3_prod(F[..., b], G[..., b]))


@pytest.mark.parametrize('B,Bx,ndim', [(2, 2, 3), (3, 5, 3), (4, 4, 3), (3, 7, 3), (2, 3, 2), (3, 17, 2), (4, 20, 2)])
def test_adjoint_gradients(hp, B, Bx, ndim):
    P = pd.pendulum_3d(B, Bx, L=4.0) if ndim == 3 else pd.pendulum_reduced(B, Bx)
    gyro = (0.0, 0.0, 0.0)
    if ndim == 3:
        J = np.diag(P.params['J'])
        gyro = ((J[1] - J[2]) / J[0], (J[2] - J[0]) / J[1], (J[0] - J[1]) / J[2])
    plan = hp.Plan(B, Bx, ndim, hp.HP_FP64, hp.HP_REAL)
    plan.set_model(P.L, P.b, P.G, P.MR, gyro)
    xs = (2 * Bx,) * ndim
    F0 = so3.fftSO3R_forward(so3.ifftSO3R_backward(coefficients(B, xs, 7), real=True))
    lamT = coefficients(B, xs, 8)
    lam_ref, g_ref, _ = adj.euler_adjoint(F0, lamT, P, 1e-3, 3)
    lam0, g = plan.adjoint(F0, lamT, 3, 1e-3, 2)
    assert rel(lam0, lam_ref) < 1e-10
    # every parameter against the largest gradient of its kind
    for kind in ('b', 'gyro', 'gscale') if ndim == 3 else ('b', 'gscale'):
        ref = np.array([g_ref[(kind, i)] for i in range(ndim)])
        assert np.abs(np.asarray(g[kind])[:ndim] - ref).max() < 1e-9 * np.abs(ref).max(), kind
    ref = np.array([[g_ref[('G', min(i, j), max(i, j))] for j in range(ndim)] for i in range(ndim)])
    assert np.abs(g['G'][:ndim, :ndim] - ref).max() < 1e-9 * np.abs(ref).max()
