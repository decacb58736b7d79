"""Kernels that work through their scratch in chunks under a memory budget that
does not hold the usual chunk: the calls go through in smaller ones and their
results are the same bit for bit (a chunk changes no sum), on the first call and
on the next, which keeps the buffer it has."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def coefficients(shape, seed):
    import torch
    g = torch.Generator(device='cuda').manual_seed(seed)
    return torch.randn(int(np.prod(shape)), dtype=torch.complex128, device='cuda', generator=g).view(*shape)


@pytest.mark.parametrize('B,batch,room', [(12, 200, 7 << 20), (4, 300, 1 << 16), (32, 12, 130 << 20)])
def test_products(hp, B, batch, room):
    """room: less than the node sums of a launch take, 58, 2.4 and 72 MB beside the table of 1.7, 0.02 and 95 MB."""
    import torch
    D = 2 * B - 1
    F, G = (coefficients((D, D, B, batch), s) for s in (1, 2))
    ref, out = torch.empty_like(F), torch.empty_like(F)
    hp.Plan(B, 2, 2, 0, 0).prod(F, G, out=ref)
    plan = hp.Plan(B, 2, 2, 0, 0)
    try:
        hp.set_device_budget(hp.device_bytes() + room)
        for _ in range(2):
            out.zero_()
            plan.prod(F, G, out=out)
            assert torch.equal(out, ref)
            held = hp.device_bytes()
            hp.set_device_budget(held)      # what it has is enough now
    finally:
        hp.set_device_budget(0)


@pytest.mark.parametrize('cut', [2, 16])
@pytest.mark.parametrize('precision', [0, 1])
def test_complex_synthesis(hp, precision, cut):
    import torch
    B, N = 20, 10
    rng = np.random.default_rng(3)
    F = rng.standard_normal((39, 39, 20, N, N)) + 1j * rng.standard_normal((39, 39, 20, N, N))
    cplx = torch.complex64 if precision else torch.complex128

    def state():
        st = hp.State(hp.Plan(B, N // 2, 2, precision, hp.HP_COMPLEX))
        st.load(F)
        return st, torch.zeros((2 * B) ** 3 * N * N, dtype=cplx, device='cuda')

    st, ref = state()
    before = hp.device_bytes()
    st.density_into(ref.data_ptr())
    grown = hp.device_bytes() - before
    chunk = 39 * 40 * 40 * (8 if precision else 16) * (128 if precision else 64)   # points of a chunk
    assert grown > chunk
    st, out = state()
    try:
        hp.set_device_budget(hp.device_bytes() + grown - chunk + chunk // cut)
        for _ in range(2):
            out.zero_()
            st.density_into(out.data_ptr())
            torch.cuda.synchronize()
            assert torch.equal(torch.view_as_real(out), torch.view_as_real(ref))
            hp.set_device_budget(hp.device_bytes())
    finally:
        hp.set_device_budget(0)
