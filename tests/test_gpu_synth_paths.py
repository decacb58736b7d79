"""The synthesis kernels at the edges of their ranges, against the oracle.

Real plans take the one-pass kernel (coefficient batches prefetched to shared
memory, nodes paired with their mirrors) from B = 6 (FP32) or 7 (FP64) up to
the bandlimit whose tables still fit, everything else and all complex plans
the two-pass kernels, whose omega points go in chunks.  The sizes are both
sides of every such line, the smallest and largest bandlimits, odd and even
ones, a last group of nodes that is not full (B = 15, 16), a grid of one batch,
and grids that leave a remainder after the last whole chunk (B = 20 complex
FP64: 64 points of 100; B = 32: 32 of 36).

Tolerances are the transform bars of the library: 1e-10 relative L2 in FP64,
1e-6 in mixed plans.
"""
import numpy as np
import pytest

from oracle import pendulum as pd
from oracle import so3

pytestmark = pytest.mark.gpu

TOL = {0: 1e-10, 1: 1e-6}
REAL = [(2, 2, 2), (3, 3, 2), (5, 3, 3), (6, 2, 2), (6, 3, 3), (7, 3, 2), (8, 2, 3), (9, 3, 2), (13, 2, 2), (15, 3, 2),
        (16, 2, 3), (17, 3, 2), (18, 2, 2), (32, 2, 2)]
COMPLEX = [(2, 2, 2), (3, 3, 3), (7, 3, 2), (16, 4, 2), (20, 5, 2), (32, 3, 2)]


def rel(a, b):
    return float(np.linalg.norm((np.asarray(a) - np.asarray(b)).ravel()) / np.linalg.norm(np.asarray(b).ravel()))


def random_coefficients(B, Bx, ndim, seed):
    rng = np.random.default_rng(seed)
    shape = (2 * B - 1, 2 * B - 1, B) + (2 * Bx,) * ndim
    F = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    k = np.abs(np.arange(2 * B - 1) - (B - 1))
    l = np.arange(B)
    keep = (np.maximum(k[:, None], k[None, :])[:, :, None] <= l) / (2 * l + 1)
    return F * keep.reshape(keep.shape + (1,) * ndim)


@pytest.mark.parametrize('precision', [0, 1])
@pytest.mark.parametrize('B,Bx,ndim', REAL)
def test_real_synthesis(hp, B, Bx, ndim, precision):
    f, _ = pd.seeded_density(B, Bx, ndim, 8.0, seed=B)
    F = so3.fftSO3R_forward(f)
    plan = hp.Plan(B, Bx, ndim, precision, hp.HP_REAL)
    assert rel(plan.backward(F), so3.ifftSO3R_backward(F, real=True)) < TOL[precision]


@pytest.mark.parametrize('precision', [0, 1])
@pytest.mark.parametrize('B,Bx,ndim', COMPLEX)
def test_complex_synthesis(hp, B, Bx, ndim, precision):
    F = random_coefficients(B, Bx, ndim, seed=B)
    plan = hp.Plan(B, Bx, ndim, precision, hp.HP_COMPLEX)
    assert rel(plan.backward(F), so3.ifftSO3R_backward(F, real=False)) < TOL[precision]


@pytest.mark.parametrize('B,symmetry', [(8, 0), (15, 0), (20, 0), (6, 1)])
@pytest.mark.parametrize('precision', [0, 1])
def test_unaligned_density_buffer(hp, B, symmetry, precision):
    """A density buffer one value off a 16-byte boundary takes the plain stores; the values are the same."""
    import torch
    Bx = 3
    F = random_coefficients(B, Bx, 2, seed=1)
    st = hp.State(hp.Plan(B, Bx, 2, precision, symmetry))
    st.load(F)
    n = (2 * B) ** 3 * (2 * Bx) ** 2 * (2 if symmetry else 1)
    buf = torch.zeros(2 * n + 8, dtype=torch.float32 if precision else torch.float64, device='cuda')
    step = buf.element_size() * (2 if symmetry else 1)
    st.density_into(buf.data_ptr())
    off = n + (-n) % 4
    st.density_into(buf.data_ptr() + off * buf.element_size() + step)
    torch.cuda.synchronize()
    a, b = buf[:n], buf[off + step // buf.element_size():][:n]
    assert torch.equal(a, b)
