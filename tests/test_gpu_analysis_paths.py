"""The FFT stage of the forward transform at the edges of its tiles, against the
oracle: the smallest and largest bandlimits, lines that are not a multiple of 16
bytes (odd B in FP32: 8-byte copies), omega grids that the tiles (1 to 16 points)
do not divide, real and complex densities, both precisions; and a density buffer
off a 16-byte boundary, which takes plain loads and gives the same coefficients.
Tolerances are the transform bars: 1e-10 relative L2 in FP64, 1e-6 mixed."""
import numpy as np
import pytest

from oracle import pendulum as pd
from oracle import so3

pytestmark = pytest.mark.gpu

TOL = {0: 1e-10, 1: 1e-6}


def rel(a, b):
    return float(np.linalg.norm((np.asarray(a) - np.asarray(b)).ravel()) / np.linalg.norm(np.asarray(b).ravel()))


@pytest.mark.parametrize('precision', [0, 1])
@pytest.mark.parametrize('symmetry', [0, 1])
@pytest.mark.parametrize('B,Bx,ndim', [(2, 2, 2), (3, 3, 3), (4, 5, 2), (9, 3, 2), (17, 3, 2), (24, 2, 2), (32, 3, 2)])
def test_forward(hp, B, Bx, ndim, symmetry, precision):
    f, _ = pd.seeded_density(B, Bx, ndim, 8.0, seed=B)
    if symmetry:
        f = f * np.exp(1j * np.random.default_rng(1).uniform(0, 6, f.shape))
    plan = hp.Plan(B, Bx, ndim, precision, symmetry)
    assert rel(plan.forward(f), so3.fftSO3R_forward(f)) < TOL[precision]


@pytest.mark.parametrize('B,symmetry,precision', [(8, 0, 0), (8, 0, 1), (9, 0, 1), (15, 0, 1), (6, 1, 1)])
def test_unaligned_density_buffer(hp, B, symmetry, precision):
    import torch
    Bx = 3
    n = (2 * B) ** 3 * (2 * Bx) ** 2 * (2 if symmetry else 1)
    g = torch.Generator(device='cuda').manual_seed(2)
    buf = torch.rand(n + 2, dtype=torch.float32 if precision else torch.float64, device='cuda', generator=g)
    off = 2 if symmetry else 1
    a, b = (hp.State(hp.Plan(B, Bx, 2, precision, symmetry)) for _ in range(2))
    a.load_density(buf[off:].data_ptr())
    b.load_density(buf[off:off + n].clone().data_ptr())
    assert np.array_equal(a.store(), b.store())
