"""The synthesis of small bandlimits on both sides of the line between one kernel
and two (B^3 times the omega points), real and complex, against the oracle: 1e-10
relative L2 in FP64, 1e-6 in mixed plans.  A density buffer off a 16-byte boundary
takes the plain stores, with the same values (B = 7: the two-pass and one-pass
kernels)."""
import numpy as np
import pytest

from oracle import so3

pytestmark = pytest.mark.gpu

SIZES = [(2, 2, 2), (2, 6, 2), (3, 2, 3), (4, 5, 2), (4, 5, 3), (4, 6, 3), (5, 11, 2), (5, 12, 2), (5, 6, 3), (5, 7, 3),
         (6, 2, 2), (6, 8, 2), (6, 9, 2), (6, 5, 3), (6, 6, 3)]


def coefficients(B, Bx, ndim, real, seed):
    rng = np.random.default_rng(seed)
    shape = (2 * B - 1, 2 * B - 1, B) + (2 * Bx,) * ndim
    k = np.arange(2 * B - 1) - (B - 1)
    keep = (np.maximum(np.abs(k)[:, None], np.abs(k)[None, :])[:, :, None] <= np.arange(B)) / (2 * np.arange(B) + 1)
    F = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) * keep.reshape(keep.shape + (1,) * ndim)
    if real:                                         # (F + C F) / 2
        G = F[::-1, ::-1]
        for a in range(3, F.ndim):
            G = np.roll(np.flip(G, a), 1, a)
        F = (F + ((-1.0) ** (k[:, None] - k[None, :])).reshape((2 * B - 1, 2 * B - 1, 1) + (1,) * ndim) * np.conj(G)) / 2
    return F


@pytest.mark.parametrize('precision', [0, 1])
@pytest.mark.parametrize('real', [True, False])
@pytest.mark.parametrize('B,Bx,ndim', SIZES)
def test_density(hp, B, Bx, ndim, real, precision):
    F = coefficients(B, Bx, ndim, real, B + Bx)
    plan = hp.Plan(B, Bx, ndim, precision, hp.HP_REAL if real else hp.HP_COMPLEX)
    ref = so3.ifftSO3R_backward(F, real=real)
    assert np.linalg.norm((plan.backward(F) - ref).ravel()) < (1e-6 if precision else 1e-10) * np.linalg.norm(ref.ravel())


@pytest.mark.parametrize('real', [True, False])
@pytest.mark.parametrize('precision', [0, 1])
@pytest.mark.parametrize('B', [5, 7])
def test_unaligned_density_buffer(hp, B, precision, real):
    import torch
    Bx = 3
    st = hp.State(hp.Plan(B, Bx, 2, precision, hp.HP_REAL if real else hp.HP_COMPLEX))
    st.load(coefficients(B, Bx, 2, real, 1))
    n = (2 * B) ** 3 * (2 * Bx) ** 2 * (1 if real else 2)
    a, b = (torch.zeros(n + 8, dtype=torch.float32 if precision else torch.float64, device='cuda') for _ in range(2))
    st.density_into(a.data_ptr())
    # one value of the density, or half a complex FP64 one, which alone is 16 bytes
    off = 2 if precision and not real else 1
    st.density_into(b.data_ptr() + off * b.element_size())
    torch.cuda.synchronize()
    assert torch.equal(a[:n], b[off:off + n])
