"""A batch's replayed graph and other calls on its members' plans: the graph
holds addresses of the plans' workspaces, so a call that frees one of those
(grows it or releases it) must end the graph's use.  The replay that must not
happen is seen from the host, by the count of graph launches; the members end
as when stepped alone (1e-12 relative L2, the bar of hybrid batches)."""
import math

import numpy as np
import pytest

from oracle import pendulum as pd

pytestmark = pytest.mark.gpu

PRM = dict(d=0.12, h=0.2, r=0.025, theta_t=5 * math.pi / 180, lambda_max=100.0, epsilon=0.8)


def init(st, seed):
    _, q = pd.seeded_density(3, 2, 2, 3.4, seed=seed)
    st.init_mf_gauss(q['U'], q['s'], q['V'], q['mu'], 0.25 * np.eye(2))


def hybrid_member(hp, precision):
    P = pd.pendulum_reduced(4, 3, L=3.4)
    plan = hp.Plan(4, 3, 2, precision, hp.HP_REAL)
    plan.set_den_model(P.L, P.b, P.G, P.mR)
    coll = hp.Collision(plan, L=P.L, Gd=0.0025 * np.eye(2), nD=10, **PRM)
    st = hp.State(plan)
    init(st, 7)
    return plan, coll, st


def init_other(hp, plan):
    """Frees the plan's transform buffers once the initial density is made."""
    init(hp.State(plan), 8)


def many_real_functions(hp, plan):
    """More functions than the plan has omega points, in FP64."""
    f = np.random.default_rng(1).standard_normal((8, 8, 8, 200))
    plan.real_forward(f)


@pytest.mark.parametrize('precision', [0, 1])
@pytest.mark.parametrize('between,frees', [(init_other, True), (many_real_functions, None)])
def test_replay_after_the_workspace_moved(hp, between, frees, precision):
    plan, coll, st = hybrid_member(hp, precision)
    F0 = st.store()
    st.hybrid_step(coll, 1e-3, 'euler', 11)
    ref = st.store()
    st.load(F0)
    batch = hp.Batch([st], [coll])
    batch.step(1e-3, 'euler', 5)
    n = batch.info()['graph_launches']
    assert n >= 1
    between(hp, plan)
    batch.step(1e-3, 'euler', 2)      # two steps: a live graph replays them, a dropped one is not captured again
    if frees:
        assert batch.info()['graph_launches'] == n
    batch.step(1e-3, 'euler', 4)      # captured again where it was dropped
    assert batch.info()['graph_launches'] > n
    assert np.linalg.norm(st.store() - ref) <= (1e-12 if precision == 0 else 1e-6) * np.linalg.norm(ref)


def test_replay_goes_on_while_nothing_is_freed(hp):
    plan, coll, st = hybrid_member(hp, 0)
    batch = hp.Batch([st], [coll])
    batch.step(1e-3, 'euler', 5)
    n = batch.info()['graph_launches']
    st.store()
    plan.moments(st.store())
    batch.step(1e-3, 'euler', 2)
    assert batch.info()['graph_launches'] == n + 1
