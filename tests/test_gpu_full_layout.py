"""Rows to the full coefficient layout, exact: kept entries as loaded, zeros
outside |m|, |n| <= l, and for real plans the m < 0 half from
F^l_{mn}[k] = (-1)^(m-n) conj F^l_{-m,-n}[-k].  Sizes whose omega count is not a
multiple of the eight points of a thread, k1 lines shorter than eight points and
lines that the eight points straddle; the largest bandlimit; both symmetries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('symmetry', [0, 1])
@pytest.mark.parametrize('B,Bx,ndim', [(2, 2, 2), (3, 3, 2), (5, 3, 3), (4, 5, 2), (10, 2, 3), (7, 9, 2), (32, 3, 2)])
def test_load_store(hp, B, Bx, ndim, symmetry):
    plan = hp.Plan(B, Bx, ndim, 0, symmetry)
    rng = np.random.default_rng(B)
    l, m = np.arange(B), np.arange(-(B - 1), B)
    mask = (np.abs(m)[:, None, None] <= l) & (np.abs(m)[None, :, None] <= l)
    F = (rng.standard_normal(plan.F_shape) + 1j * rng.standard_normal(plan.F_shape)).astype(np.complex128)
    want = F * mask.reshape(mask.shape + (1,) * ndim)
    if symmetry == 0:
        k = tuple(range(3, 3 + ndim))
        mirror = np.conj(np.roll(np.flip(want, (0, 1) + k), 1, k))
        sign = (-1.0) ** (m[:, None] - m[None, :])
        mirror *= sign.reshape(sign.shape + (1,) * (1 + ndim))
        want[:B - 1] = mirror[:B - 1]
    st = hp.State(plan)
    st.load(F)
    assert np.array_equal(st.store(), want)
