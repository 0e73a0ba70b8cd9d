"""Small packable models through every kernel that takes them: lane groups of
32, 16, 8 and 4 lanes, the direct forms of the thread kernels and of the
mode-sorted scheduler (1, 2 or 3 factor slots) and the first models past
them (four factors, one reaction, five species).  Each run equals the oracle,
with the direct method and tau-leaping, with and without scores, alone and in
a batch.
"""

import numpy as np
import pytest

from py_stoch_b200 import networks
from py_stoch_b200.model import Model

pytestmark = pytest.mark.gpu
T_RTOL = 1e-12
N = 24000           # the thread kernels on up to 148 SMs (162 per SM)


def _model(factors, reactions, S=4, t_end=0.05):
    """A source, a reaction with `factors` reactant factors in all (orders 1;
    1+1; 2+1; 2+2) and first-order conversions, `reactions` in all."""
    pre = np.zeros((S, reactions), np.int64)
    post = np.zeros((S, reactions), np.int64)
    orders = {1: (1, 0), 2: (1, 1), 3: (2, 1), 4: (2, 2)}[factors]
    pre[0, 0], pre[1, 0] = orders
    post[2, 0] = 1
    if orders[1] == 0:
        post[1, 0] = 1
    k = [{1: 0.5, 2: 1e-3, 3: 2e-6, 4: 4e-9}[factors]]
    if reactions > 1:
        post[0, 1] = 3
        k.append(900.0)
    for j in range(2, reactions):
        pre[j % S, j] = 1
        post[(j + 1) % S, j] = 1
        k.append(0.3 + 0.2 * j)
    return Model.mass_action(pre, post, k, [300, 200, 100, 50, 20][:S],
                             np.linspace(0, t_end, 6).astype(np.float32),
                             np.arange(S))


def _compare(g, o, n, score):
    np.testing.assert_array_equal(g['samples'], o['samples'][:, :, :n])
    for key in ('status', 'events', 'seqhash'):
        np.testing.assert_array_equal(g[key], o[key][:n], err_msg=key)
    np.testing.assert_allclose(g['t_final'], o['t_final'][:n], rtol=T_RTOL,
                               atol=0)
    if score:
        np.testing.assert_allclose(g['score'], o['score'][:n], rtol=T_RTOL,
                                   atol=1e-12)


@pytest.mark.parametrize('factors,reactions,S', [
    (1, 2, 4), (2, 3, 4), (3, 4, 4), (4, 4, 4), (1, 6, 4), (3, 6, 5),
    (2, 8, 5), (4, 8, 4), (2, 1, 4)])
@pytest.mark.parametrize('method', ['direct', 'tau'])
def test_small_models(torch_cuda, built_lib, oracle_mod, factors, reactions,
                      S, method):
    from py_stoch_b200.batch import Batch
    from py_stoch_b200.simulator import simulate
    m = _model(factors, reactions, S)
    o = oracle_mod.simulate(m, N, 0 if method == 'direct' else 1,
                            seed=factors)

    def check(n, score, **kw):
        r = simulate(m, n, method=method, seed=factors, seqhash=True,
                     t_final=True, score=score, **kw)
        torch_cuda.cuda.synchronize()
        g = {k: v.cpu().numpy() for k, v in r.items() if k != '_keepalive'}
        g['seqhash'] = g['seqhash'].view(np.uint64)
        _compare(g, o, n, score)

    # (runs of these sizes take 32, 32, 16, 8 and 4 or 8 lanes on 148 SMs,
    # the largest a thread per trajectory)
    for n in (1, 300, 1700, 3001, 9000, N):
        check(n, n in (300, 3001, N))
    if method == 'tau':
        check(3001, True, geometry={'round_ssa': 20, 'round_leap': 2})
        check(2000, False, sorted_blocks=False)
        check(3001, False, geometry={'sorted_block': 448})
    for n in (130, N):  # lane groups and a thread per trajectory
        b = Batch([m], n, method=method, score=True)
        assert b.lane_groups == (n == 130 or method == 'tau')
        b.lane_groups &= n == 130
        b.run(seed=factors)
        torch_cuda.cuda.synchronize()
        np.testing.assert_array_equal(b.samples(0).cpu().numpy(),
                                      o['samples'][:, :, :n])
        np.testing.assert_allclose(b.score(0).cpu().numpy(),
                                   o['score'][:n], rtol=T_RTOL, atol=1e-12)


@pytest.mark.parametrize('n', [40, 2000, 3000, 9000])
def test_rare_ends_in_lane_groups(torch_cuda, built_lib, oracle_mod, n):
    """What ends a run of steps early: many sample times per step, counts
    that leave the int32 range, absorption, the step budget inside and at
    the edge of a row of steps, fallback rounds shorter than a row."""
    from py_stoch_b200.simulator import simulate
    dense = networks.schlogl(t_end=0.05, n_samples=300)
    grow = Model.mass_action([[1]], [[2]], [40.0], [2**31 - 40],
                             np.float32([0, 1e-10, 3e-10]), [0])
    decay = Model.mass_action([[1, 0], [0, 1]], [[0, 0], [1, 0]], [3.0, 2.0],
                              [30, 20], np.linspace(0, 20, 9).astype(
                                  np.float32), [0, 1])
    for m, kw in ((dense, {}), (grow, {}), (decay, {}),
                  (dense, {'step_budget': 33}), (decay, {'step_budget': 7}),
                  (dense, {'ssa_fallback_steps': 3}),
                  (dense, {'ssa_fallback_steps': 1, 'step_budget': 50})):
        for method in ('direct', 'tau'):
            r = simulate(m, n, method=method, seed=8, seqhash=True,
                         t_final=True, **kw)
            torch_cuda.cuda.synchronize()
            g = {k: v.cpu().numpy() for k, v in r.items()
                 if k != '_keepalive'}
            g['seqhash'] = g['seqhash'].view(np.uint64)
            o = oracle_mod.simulate(m, n, 0 if method == 'direct' else 1,
                                    seed=8, **kw)
            _compare(g, o, n, False)
