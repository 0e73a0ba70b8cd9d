"""Propensities and totals at the ends of the number range, through every
engine: a propensity that overflows to infinity or is NaN (infinity times a
zero count), with and without a positive propensity beside it; finite
propensities whose FP64 sum passes the FP32 range; subnormal propensities.
The rates are finite and so accepted.  Every run is bounded by its step
budget and equals the oracle.  Where the total is NaN and nothing is positive
no reaction can be selected: such a step changes no count.
"""

import numpy as np
import pytest

from py_stoch_b200.model import Model

pytestmark = pytest.mark.gpu
T_RTOL = 1e-12
BUDGET = 40
MANY = 24000        # the thread kernels on up to 148 SMs (162 per SM)


def _model(kind, R, form='direct'):
    """Species A, B, C, D and E; a model of R reactions.  form: 'direct'
    (direct forms), 'packed' (one reaction of four factors), 'lists' (a
    change of 20)."""
    S = 5
    pre, post = np.zeros((S, R), np.int64), np.zeros((S, R), np.int64)
    x0 = [1000000, 0, 0, 0, 0]
    times = np.float32([0, 1, 2])
    k = [1.0] * R

    def rx(j, a, b, rate):
        pre[:, j], post[:, j] = 0, 0
        for i, n in a.items():
            pre[i, j] = n
        for i, n in b.items():
            post[i, j] = n
        k[j] = rate

    # from the last reaction on: propensity 0 (D and E stay at zero)
    for j in range(R):
        rx(j, {3: 1}, {4: 1}, 2.0)
    if form == 'packed':
        rx(R - 1, {3: 2, 4: 2}, {3: 1}, 2.0)
    elif form == 'lists':
        rx(R - 1, {3: 1}, {4: 20}, 2.0)
    if kind == 'nan':            # A + B -> A: inf * 0
        rx(0, {0: 1, 1: 1}, {0: 1}, 1e33)
    elif kind == 'nan_last':
        rx(R - 2, {0: 1, 1: 1}, {0: 1}, 1e33)
    elif kind == 'nan_positive':  # beside a source, before and after
        rx(0, {}, {2: 1}, 5.0)
        rx(1, {0: 1, 1: 1}, {0: 1}, 1e33)
        if R > 3:
            rx(2, {2: 1}, {1: 1}, 40.0)
    elif kind == 'nan_apart':    # the source in another lane's reactions,
        rx(0, {0: 1, 1: 1}, {0: 1}, 1e33)  # after one of propensity 0
        rx(R - 1 if R < 5 else 3, {}, {2: 1}, 5.0)
    elif kind == 'inf':          # A -> A + B
        rx(0, {}, {2: 1}, 5.0)
        rx(1, {0: 1}, {0: 1, 1: 1}, 1e33)
    elif kind == 'late_inf':     # C + A -> A once C comes (fallback steps)
        x0 = [0, 0, 1000000, 0, 0]
        rx(0, {}, {0: 1}, 5.0)
        rx(1, {0: 1, 2: 1}, {2: 1}, 1e33)
    elif kind == 'late_nan':     # with a third factor that stays 0
        x0 = [0, 0, 1000000, 0, 0]
        rx(0, {}, {0: 1}, 5.0)
        rx(1, {0: 1, 2: 1, 3: 1}, {2: 1}, 1e33)
        if R > 3:
            rx(2, {0: 1}, {1: 1}, 1.0)
    elif kind == 'sum':          # finite, the sum beyond FP32
        for j in range(min(R, 3)):
            rx(j, {0: 1}, {0: 1, 1: 1}, 3e32)
        times = np.float32([0, 2e-38, 3e-38])
    elif kind == 'subnormal':    # 1e-44 and 1e-38
        rx(0, {0: 1}, {1: 1}, 1e-44)
        rx(1, {}, {2: 1}, 3e-42)
        times = np.float32([0, 1e38, 3e38])
    return Model.mass_action(pre, post, k, x0, times, np.arange(S))


def _compare(torch, r, o, n):
    torch.cuda.synchronize()
    np.testing.assert_array_equal(r['samples'].cpu().numpy(),
                                  o['samples'][:, :, :n])
    for key in ('status', 'events'):
        np.testing.assert_array_equal(r[key].cpu().numpy(), o[key][:n],
                                      err_msg=key)
    if 'seqhash' in r:
        np.testing.assert_array_equal(
            r['seqhash'].cpu().numpy().view(np.uint64), o['seqhash'][:n])
    if 't_final' in r:
        np.testing.assert_allclose(r['t_final'].cpu().numpy(),
                                   o['t_final'][:n], rtol=T_RTOL)
    if 'score' in r:
        np.testing.assert_allclose(r['score'].cpu().numpy(), o['score'][:n],
                                   rtol=T_RTOL, atol=1e-12)


KINDS = ['nan', 'nan_last', 'nan_positive', 'nan_apart', 'inf', 'late_inf',
         'late_nan', 'sum', 'subnormal']


@pytest.mark.parametrize('kind', KINDS)
@pytest.mark.parametrize('R,form', [
    (2, 'direct'), (3, 'direct'), (4, 'direct'), (7, 'direct'),
    (8, 'direct'), (4, 'packed'), (8, 'packed'), (4, 'lists'),
    (12, 'direct')])
def test_rare_totals_small(torch_cuda, built_lib, oracle_mod, kind, R, form):
    from py_stoch_b200.batch import Batch
    from py_stoch_b200.simulator import simulate
    m = _model(kind, R, form)
    for method in ('direct', 'tau'):
        o = oracle_mod.simulate(m, MANY, 0 if method == 'direct' else 1,
                                seed=R, step_budget=BUDGET)
        # lane groups of 32 and 4 or 8 lanes (the lockstep group for lists),
        # a thread per trajectory
        runs = [(n, {}) for n in (300, 5000, MANY)]
        if method == 'tau':
            runs += [(3000, {'geometry': {'round_ssa': 20,
                                          'round_leap': 2}}),
                     (3000, {'sorted_blocks': False})]
        for n, kw in runs:
            for score in (False, True):
                r = simulate(m, n, method=method, seed=R, seqhash=True,
                             t_final=True, score=score, mapping='thread',
                             step_budget=BUDGET, **kw)
                _compare(torch_cuda, r, o, n)
        for chunk in (0, 128):  # a thread per trajectory, lane groups
            b = Batch([m], 200, method=method, mapping='thread', score=True,
                      chunk=chunk)
            b.run(seed=R, step_budget=BUDGET)
            _compare(torch_cuda, {'samples': b.samples(0),
                                  'status': b.per_traj('status', 0),
                                  'events': b.per_traj('events', 0),
                                  'score': b.score(0)}, o, 200)


@pytest.mark.parametrize('kind', KINDS)
@pytest.mark.parametrize('R,mapping', [(4, 'warp'), (40, 'warp'),
                                       (70, 'warp'), (40, 'thread'),
                                       (70, 'thread')])
@pytest.mark.parametrize('form', ['direct', 'packed'])
def test_rare_totals_wide(torch_cuda, built_lib, oracle_mod, kind, R,
                          mapping, form):
    """Warp-mapped runs and networks beyond the register arrays, with one
    word per reaction ('packed': four factors, as orders 2 + 2)."""
    from py_stoch_b200.batch import Batch
    from py_stoch_b200.simulator import simulate
    m = _model(kind, R, form)
    n = 96
    for method in ('direct', 'tau'):
        o = oracle_mod.simulate(m, n, 0 if method == 'direct' else 1, seed=R,
                                warp=mapping == 'warp', step_budget=BUDGET)
        for score in ((False, True) if mapping == 'warp' else (False,)):
            r = simulate(m, n, method=method, mapping=mapping, seed=R,
                         seqhash=True, t_final=True, score=score,
                         step_budget=BUDGET)
            _compare(torch_cuda, r, o, n)
        b = Batch([m], n, method=method, mapping=mapping,
                  small_batch_warps=False)
        b.run(seed=R, step_budget=BUDGET)
        _compare(torch_cuda, {'samples': b.samples(0),
                              'status': b.per_traj('status', 0),
                              'events': b.per_traj('events', 0)}, o, n)
