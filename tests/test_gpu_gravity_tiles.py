"""The gravity pass at the widths of its omega tiles (8, 16 and 32 points, taken
by the blocks and the rows per thread they leave), on both sides of each line, against the
oracle's derivative: 1e-10 relative L2 in FP64, 1e-6 mixed."""
import numpy as np
import pytest

from oracle import pendulum as pd
from oracle import so3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('precision', [0, 1])
@pytest.mark.parametrize('B,Bx', [(2, 2), (4, 8), (6, 3), (8, 11), (8, 12), (8, 16), (9, 16)])
def test_derivative(hp, B, Bx, precision):
    P = pd.pendulum_reduced(B, Bx)
    f, _ = pd.seeded_density(B, Bx, 2, P.L, seed=4)
    F = so3.fftSO3R_forward(f)
    ref = pd.derivative_fast(F, P)
    plan = hp.get_plan(B, Bx, 2, precision, hp.HP_REAL)
    plan.set_model(P.L, P.b, P.G, P.MR)
    out = plan.derivative(F)
    assert np.linalg.norm(out - ref) < (1e-6 if precision else 1e-10) * np.linalg.norm(ref)
