"""Real-harmonic transforms of HP_REAL plans (through the complex rows and the
FFT kernels) against the oracle and against the direct sums that complex plans
run: the smallest bandlimits, odd ones, batches that the kernels' tiles (2 to
16 functions) and the 32-function blocks do not divide, device tensors that are
not 16-byte aligned.  Tolerance 1e-12 relative L2, the bar of the library's
other real-harmonic tests."""
import numpy as np
import pytest

from oracle import real_harmonics as rh

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm((np.asarray(a) - np.asarray(b)).ravel()) / np.linalg.norm(np.asarray(b).ravel()))


@pytest.mark.parametrize('B,nb', [(2, 1), (3, 2), (4, 5), (5, 3), (8, 33), (11, 1)])
def test_transforms_vs_oracle(hp, B, nb):
    rng = np.random.default_rng(B)
    f = rng.standard_normal((2 * B, 2 * B, 2 * B, nb))
    plan = hp.Plan(B, 2, 2, hp.HP_FP64, hp.HP_REAL)
    F = plan.real_forward(f)
    g = plan.real_backward(F)
    for b in {0, nb // 2, nb - 1}:
        ref = rh.forward(f[..., b])
        assert rel(F[..., b], ref) < 1e-12
        assert rel(g[..., b], rh.backward(ref)) < 1e-12


@pytest.mark.parametrize('B,nb', [(6, 31), (16, 7), (20, 2)])
def test_both_routes_agree(hp, B, nb):
    rng = np.random.default_rng(B)
    f = rng.standard_normal((2 * B, 2 * B, 2 * B, nb))
    real, cplx = (hp.Plan(B, 2, 2, hp.HP_FP64, sym) for sym in (hp.HP_REAL, hp.HP_COMPLEX))
    F = cplx.real_forward(f)
    assert rel(real.real_forward(f), F) < 1e-12
    F = F + rng.standard_normal(F.shape)          # also values where |m| or |n| > l, which both ignore
    assert rel(real.real_backward(F), cplx.real_backward(F)) < 1e-12


def test_unaligned_tensors(hp):
    import torch
    B, nb = 7, 3
    n, c = (2 * B) ** 3 * nb, (2 * B - 1) ** 2 * B * nb
    plan = hp.Plan(B, 2, 2, hp.HP_FP64, hp.HP_REAL)
    g = torch.Generator(device='cuda').manual_seed(1)
    f = torch.randn(n + 1, dtype=torch.float64, device='cuda', generator=g)
    F, F1 = torch.zeros(c, dtype=torch.float64, device='cuda'), torch.zeros(c + 1, dtype=torch.float64, device='cuda')
    plan.real_forward(f[1:], out=F1[1:])
    plan.real_forward(f[1:].clone(), out=F)
    assert torch.equal(F, F1[1:])
    h, h1 = torch.zeros(n, dtype=torch.float64, device='cuda'), torch.zeros(n + 1, dtype=torch.float64, device='cuda')
    plan.real_backward(F1[1:], out=h1[1:])
    plan.real_backward(F, out=h)
    assert torch.equal(h, h1[1:])
