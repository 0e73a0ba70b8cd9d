"""Networks beyond the register arrays: the one-word-per-reaction form and
its segmented selection at the edges of the segments (33, 40, 41 and 255
reactions), a model it does not take (a third-order reaction), a network that
dies out, thread- and warp-mapped, alone and in a batch; the warp kernel with
the step variates of 32 steps spread over its lanes also below 32 reactions.
Each run equals the oracle.
"""

import numpy as np
import pytest

from py_stoch_b200 import networks
from py_stoch_b200.model import Model

pytestmark = pytest.mark.gpu


def _net(R, third=False, dying=False):
    m = networks.synthetic_networks(1, seed=R, s_range=(9, 9),
                                    r_range=(R, R), n_samples=7,
                                    t_range=(0.01, 0.01), x0_max=800)[0]
    order, net = m.order.copy(), m.net.copy()
    if third:
        order[:, R // 2] = 0
        order[3, R // 2] = 3
    if dying:  # no zeroth-order source, every reaction takes one of each
        order[:, order.sum(axis=0) == 0] = np.eye(9, dtype=np.int32)[:, :1]
        net = -order
    return Model(order, order, net, m.rate, m.x0, m.sample_times,
                 m.out_species)


@pytest.mark.parametrize('R,third,dying', [
    (33, False, False), (40, False, False), (41, False, True),
    (255, False, False), (64, True, False), (20, False, False)])
@pytest.mark.parametrize('mapping', ['thread', 'warp'])
def test_wide_networks(torch_cuda, built_lib, oracle_mod, R, third, dying,
                       mapping):
    from py_stoch_b200.batch import Batch
    from py_stoch_b200.simulator import simulate
    m = _net(R, third, dying)
    n = 70
    for method in ('direct', 'tau'):
        o = oracle_mod.simulate(m, n, 0 if method == 'direct' else 1, seed=R,
                                warp=mapping == 'warp', step_budget=3000)
        r = simulate(m, n, method=method, mapping=mapping, seed=R,
                     seqhash=True, t_final=True, step_budget=3000,
                     sorted_blocks=False)
        b = Batch([m], n, method=method, mapping=mapping, chunk=40,
                  small_batch_warps=False)
        b.run(seed=R, step_budget=3000)
        torch_cuda.cuda.synchronize()
        g = {k: v.cpu().numpy() for k, v in r.items() if k != '_keepalive'}
        np.testing.assert_array_equal(g['samples'], o['samples'])
        np.testing.assert_array_equal(g['status'], o['status'])
        np.testing.assert_array_equal(g['events'], o['events'])
        np.testing.assert_array_equal(g['seqhash'].view(np.uint64),
                                      o['seqhash'])
        np.testing.assert_allclose(g['t_final'], o['t_final'], rtol=1e-12)
        np.testing.assert_array_equal(b.samples(0).cpu().numpy(),
                                      o['samples'])
        np.testing.assert_array_equal(
            b.per_traj('status', 0).cpu().numpy(), o['status'])
