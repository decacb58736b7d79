"""Gravity tiles that small bandlimits and 2-D grids do not reach: the adjoint's
dot pass at its 8- and 4-point tiles (B >= 15 and B >= 24), the adjoint of mixed
plans (FP32 taps of W Grav W^-1), and the 3-D derivative on both sides of the
block count that chooses its tile, at bandlimits whose widest tile is 32, 16, 8
and 4 points.  Against the oracle: 1e-10 relative L2 in FP64, 1e-6 in mixed plans;
gradients against the largest of their kind, 1e-9 and 1e-5 (sums of products of
two such fields)."""
import numpy as np
import pytest

from oracle import adjoint as adj
from oracle import pendulum as pd
from oracle import so3

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


def coefficients(B, xs, seed):
    rng = np.random.default_rng(seed)
    k = np.abs(np.arange(2 * B - 1) - (B - 1))
    keep = (np.maximum(k[:, None], k[None, :])[:, :, None] <= np.arange(B)) / (2.0 * np.arange(B) + 1)
    F = rng.standard_normal((2 * B - 1, 2 * B - 1, B) + xs) + 1j * rng.standard_normal((2 * B - 1, 2 * B - 1, B) + xs)
    return F * keep.reshape(keep.shape + (1,) * len(xs))


def model(hp, B, Bx, ndim, precision):
    P = pd.pendulum_3d(B, Bx, L=4.0) if ndim == 3 else pd.pendulum_reduced(B, Bx)
    gyro = (0.0, 0.0, 0.0)
    if ndim == 3:
        J = np.diag(P.params['J'])
        gyro = ((J[1] - J[2]) / J[0], (J[2] - J[0]) / J[1], (J[0] - J[1]) / J[2])
    plan = hp.Plan(B, Bx, ndim, precision, hp.HP_REAL)
    plan.set_model(P.L, P.b, P.G, P.MR, gyro)
    return P, plan


def real_coefficients(B, xs, seed):
    F = coefficients(B, xs, seed)
    G = F[::-1, ::-1]                                # the projection on real densities: (F + C F) / 2
    for a in range(3, F.ndim):
        G = np.roll(np.flip(G, a), 1, a)
    k = np.arange(2 * B - 1)
    sign = (-1.0) ** (k[:, None] - k[None, :])
    return (F + sign.reshape(sign.shape + (1,) * (F.ndim - 2)) * np.conj(G)) / 2


@pytest.mark.parametrize('B,Bx,ndim,precision', [(14, 2, 2, 0), (15, 2, 2, 0), (15, 3, 2, 0), (23, 2, 2, 0), (24, 2, 2, 0),
                                                 (4, 3, 3, 1), (7, 2, 2, 1), (15, 2, 2, 1), (24, 2, 2, 1)])
def test_adjoint(hp, B, Bx, ndim, precision):
    P, plan = model(hp, B, Bx, ndim, precision)
    xs = (2 * Bx,) * ndim
    F0, lamT = real_coefficients(B, xs, 7), coefficients(B, xs, 8)
    lam_ref, g_ref, _ = adj.euler_adjoint(F0, lamT, P, 1e-3, 2)
    lam0, g = plan.adjoint(F0, lamT, 2, 1e-3, 2)
    assert rel(lam0, lam_ref) < (1e-6 if precision else 1e-10)
    tol = 1e-5 if precision else 1e-9
    for kind in ('b', 'gyro', 'gscale') if ndim == 3 else ('b', 'gscale'):
        ref = np.array([g_ref[(kind, i)] for i in range(ndim)])
        assert np.abs(np.asarray(g[kind])[:ndim] - ref).max() < tol * np.abs(ref).max(), kind
    ref = np.array([[g_ref[('G', min(i, j), max(i, j))] for j in range(ndim)] for i in range(ndim)])
    assert np.abs(g['G'][:ndim, :ndim] - ref).max() < tol * np.abs(ref).max()


@pytest.mark.parametrize('precision', [0, 1])
@pytest.mark.parametrize('B,Bx,ndim', [(8, 4, 3), (10, 4, 3), (10, 5, 3), (18, 2, 3), (19, 2, 3), (22, 2, 3), (23, 2, 2),
                                       (24, 2, 3), (25, 2, 2), (30, 2, 2), (31, 2, 2), (32, 2, 2)])
def test_derivative(hp, B, Bx, ndim, precision):
    P, plan = model(hp, B, Bx, ndim, precision)
    F = real_coefficients(B, (2 * Bx,) * ndim, 4)
    assert rel(plan.derivative(F), pd.derivative_fast(F, P)) < (1e-6 if precision else 1e-10)
