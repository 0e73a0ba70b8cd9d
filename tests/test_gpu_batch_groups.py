"""Batches with lane groups: models the groups take (4 and 8 lanes) beside
models they do not (four factors, a third changed species, more than 8
reactions, large networks on warps), of even and uneven sizes, with scores,
statistics and Jacobians.  Every item equals the oracle, and the reduced
outputs equal those of the batch without chunks and groups bit for bit.
"""

import numpy as np
import pytest

from py_stoch_b200 import networks
from test_gpu_kernels import check_batch, model

pytestmark = pytest.mark.gpu


def _mixed():
    big = networks.synthetic_networks(1, seed=4, s_range=(9, 9),
                                      r_range=(40, 40), n_samples=6,
                                      t_range=(0.003, 0.003), x0_max=400)
    return [model(2, 3), model(3, 7), model(4, 6), model(2, 6, lists=True),
            networks.schlogl(t_end=0.3, n_samples=6), model(2, 12, 6, 0.02),
            networks.telegraph(t_end=2.0, n_samples=5), model(1, 4)] + big


@pytest.mark.parametrize('sizes', [
    [40, 33, 100, 64, 128, 17, 130, 300, 20], [8] * 9,
    [1, 1, 200, 1, 1, 1, 1, 700, 1], [500, 3, 1, 2, 40, 260, 15, 16, 9]])
@pytest.mark.parametrize('method', ['direct', 'tau'])
@pytest.mark.parametrize('score', [False, True])
def test_mixed(torch_cuda, built_lib, oracle_mod, sizes, method, score):
    from py_stoch_b200.batch import Batch
    models, budget = _mixed(), 20000
    kw = dict(method=method, score=score, stats=True, jacobian=score,
              seqhash=True, t_final=True)
    b = Batch(models, sizes, **kw)
    assert b.lane_groups and b._group_items is not None
    b.run(seed=3, step_budget=budget)
    plain = Batch(models, sizes, chunk=0, **kw)
    plain.run(seed=3, step_budget=budget)
    torch_cuda.cuda.synchronize()
    for i, m in enumerate(models):
        o = oracle_mod.simulate(m, sizes[i], 0 if method == 'direct' else 1,
                                seed=3, traj_id_base=int(b.traj_id_base[i]),
                                warp=int(b.mappings[i]) == 2,
                                step_budget=budget)
        check_batch(torch_cuda, b, i, o, sizes[i])
        np.testing.assert_array_equal(b.stats(i).cpu().numpy(),
                                      plain.stats(i).cpu().numpy())
        if score:
            np.testing.assert_array_equal(b.jacobian(i).cpu().numpy(),
                                          plain.jacobian(i).cpu().numpy())


def test_every_trajectory_runs_whatever_the_limits_hold(
        torch_cuda, built_lib, oracle_mod):
    """The spare field of the limits changes nothing."""
    from py_stoch_b200.batch import Batch
    m = model(2, 3)
    b = Batch([m], 100, method='tau', seqhash=True)
    assert b.lane_groups
    b.limits.reserved = 2 << 16 | 16
    b.run(seed=9)
    torch_cuda.cuda.synchronize()
    check_batch(torch_cuda, b, 0, oracle_mod.simulate(m, 100, 1, seed=9),
                100)


@pytest.mark.parametrize('n,block', [(1, 32), (8, 32), (16, 64), (24, 32),
                                     (32, 128), (40, 32), (256, 128)])
def test_group_blocks(torch_cuda, built_lib, n, block):
    from py_stoch_b200.batch import Batch
    b = Batch([model(2, 3)] * 3, n, method='tau')
    assert b._group_block == block
    # each item has at most a trajectory per group of its block
    raw = b._group_items.cpu().numpy().view(np.int64).reshape(-1, 12)
    assert raw[:, 1].max() <= block // 4 and raw[:, 1].sum() == 3 * n
