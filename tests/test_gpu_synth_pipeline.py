"""The one-pass synthesis with several omega batches per block: coefficients of
the next batch copied while one is transformed, staging buffers rewritten behind
the bulk copies (or, for a buffer off a 16-byte boundary, behind plain stores),
a last block with fewer batches.  synth_waves = 1 makes few blocks of many
batches; the densities equal the oracle's (1e-10, 1e-6 mixed) and, bit for bit,
those of one batch per block."""
import numpy as np
import pytest

from oracle import pendulum as pd
from oracle import so3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('B,Bx,precision', [(6, 13, 1), (8, 14, 1), (15, 10, 1), (16, 8, 1), (17, 5, 1),
                                            (7, 13, 0), (9, 10, 0), (12, 7, 0), (13, 7, 0), (16, 5, 0)])
def test_many_batches_per_block(hp, B, Bx, precision):
    import torch
    f, _ = pd.seeded_density(B, Bx, 2, 8.0, seed=B)
    F = so3.fftSO3R_forward(f)
    ref = so3.ifftSO3R_backward(F, real=True).ravel(order='F')
    plan = hp.Plan(B, Bx, 2, precision, hp.HP_REAL)
    st = hp.State(plan)
    st.load(F)
    n = (2 * B) ** 3 * (2 * Bx) ** 2
    out = []
    for waves in (1, 64):
        for off in (0, 1):
            plan.set_tune(synth_waves=waves)
            buf = torch.zeros(n + 4, dtype=torch.float32 if precision else torch.float64, device='cuda')
            st.density_into(buf.data_ptr() + off * buf.element_size())
            torch.cuda.synchronize()
            out.append(buf[off:off + n].cpu())
    assert np.linalg.norm(out[0].double().numpy() - ref) < (1e-6 if precision else 1e-10) * np.linalg.norm(ref)
    assert all(torch.equal(x, out[0]) for x in out[1:])
