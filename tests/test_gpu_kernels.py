"""Packable models of 1 to 8 reactions and 1 to 6 reactant factors through
every kernel that takes them: lane groups of every width, the thread kernels
with direct forms (up to 3 factors), with packed descriptors (4 and more) and
with one reaction, the simple tau loop, the mode-sorted scheduler, and the
batch with and without lane groups.  Models of 9 to 32 reactions, packable
and not, through the thread kernels and the scheduler.  Each run equals the
oracle, with and without scores.
"""

import numpy as np
import pytest

from py_stoch_b200 import _lib, networks
from py_stoch_b200.model import Model

pytestmark = pytest.mark.gpu
T_RTOL = 1e-12
MANY = 24000        # the thread kernels on up to 148 SMs (162 per SM)


def model(factors, R, S=4, t_end=0.05, lists=False, x=1000):
    """Reaction 0 takes `factors` molecules in all of species 0 and 1 (orders
    1; 1+1; 2+1; 2+2; 3+2; 3+3) and turns one of species 0 into one of species
    1; a source; first-order conversions.  lists: a conversion that changes a
    third species, beyond the packed forms.  x: species 0's count; about 1,000
    takes both leaps and fallback steps."""
    pre, post = np.zeros((S, R), np.int64), np.zeros((S, R), np.int64)
    a, b = {1: (1, 0), 2: (1, 1), 3: (2, 1), 4: (2, 2), 5: (3, 2),
            6: (3, 3)}[factors]
    pre[0, 0], pre[1, 0], post[0, 0], post[1, 0] = a, b, a - 1, b + 1
    k = [9.0 * {1: 1, 2: 1, 3: 2, 4: 4, 5: 12, 6: 36}[factors] /
         x ** (factors - 1)]
    if R > 1:
        post[0, 1] = 3
        k.append(2.0 * x)
    for j in range(2, R):
        pre[j % S, j] = 1
        post[(j + 1) % S, j] = 1
        if lists and j == 2:
            post[(j + 2) % S, j] = 1
        k.append(3.0 + 2.0 * j)
    return Model.mass_action(pre, post, k, ([x, x, x // 4] + [20] * S)[:S],
                             np.linspace(0, t_end, 6).astype(np.float32),
                             np.arange(S))


def packable(lib, m):
    return lib.pyst_test_model_packable(m.blob().ctypes.data)


def compare(g, o, n):
    for key, v in g.items():
        if key in ('_keepalive', 'workspace'):
            continue
        v = v.cpu().numpy()
        if key == 'samples':
            np.testing.assert_array_equal(v, o[key][:, :, :n])
        elif key in ('status', 'events'):
            np.testing.assert_array_equal(v, o[key][:n], err_msg=key)
        elif key == 'seqhash':
            np.testing.assert_array_equal(v.view(np.uint64), o[key][:n])
        else:
            np.testing.assert_allclose(v, o[key][:n], rtol=T_RTOL,
                                       atol=1e-12 if key == 'score' else 0,
                                       err_msg=key)


def kernel(m, n, method, score=False, **kw):
    from py_stoch_b200.simulator import run_kernel
    return run_kernel(m, n, method, 'thread', score, **kw)[0]


def check(torch, m, o, n, method, seed, want=None, **kw):
    from py_stoch_b200.simulator import simulate
    route = {k: v for k, v in kw.items()
             if k in ('score', 'geometry', 'sorted_blocks')}
    assert want is None or kernel(m, n, method, **route) == want
    r = simulate(m, n, method=method, seed=seed, seqhash=True, t_final=True,
                 mapping='thread', **kw)
    torch.cuda.synchronize()
    compare(r, o, n)


def check_batch(torch, b, i, o, n):
    g = {'samples': b.samples(i)}
    for k in ('status', 'events', 'seqhash', 't_final'):
        if k in b.out:
            g[k] = b.per_traj(k, i)
    if 'score' in b.out:
        g['score'] = b.score(i)
    compare(g, o, n)


@pytest.mark.parametrize('factors,R,S', [
    (1, 1, 4), (4, 1, 4), (1, 2, 2), (2, 2, 4), (4, 2, 4), (3, 3, 4),
    (5, 3, 3), (1, 4, 4), (3, 4, 4), (4, 4, 4), (6, 4, 5), (2, 5, 4),
    (3, 5, 6), (4, 5, 4), (1, 6, 8), (3, 6, 4), (6, 6, 4), (2, 7, 4),
    (3, 7, 4), (5, 7, 7), (1, 8, 4), (3, 8, 9), (4, 8, 8), (6, 8, 20)])
@pytest.mark.parametrize('method', ['direct', 'tau'])
def test_small_packable(torch_cuda, built_lib, oracle_mod, factors, R, S,
                        method):
    from py_stoch_b200.batch import Batch
    m = model(factors, R, S, x=3000 if factors == 6 else 1000)
    assert packable(built_lib, m) == 1
    seed = 10 * factors + R
    o = oracle_mod.simulate(m, MANY, 0 if method == 'direct' else 1,
                            seed=seed)
    # 32, 32, 16, 8 and 4 or 8 lanes, a thread per trajectory (148 SMs; with
    # 9 or more species 16 or 32 lanes, then a thread)
    for n in (1, 300, 1700, 3001, 9000, MANY):
        want = (_lib.KERNEL_GROUP if n <= 300 else None if n < MANY else
                _lib.KERNEL_THREAD if method == 'direct' else
                _lib.KERNEL_SORTED)
        for score in (False, True):
            check(torch_cuda, m, o, n, method, seed, want, score=score)
    if method == 'tau':
        for score in (False, True):
            for geo in ({'round_ssa': 20, 'round_leap': 2},
                        {'sorted_block': 448}):
                check(torch_cuda, m, o, 2500, method, seed,
                      _lib.KERNEL_SORTED, score=score, geometry=geo)
            check(torch_cuda, m, o, 2500, method, seed, _lib.KERNEL_THREAD,
                  score=score, sorted_blocks=False)
    for chunk in (0, 128):  # a thread per trajectory, lane groups
        for score in (False, True):
            b = Batch([m], 300, method=method, mapping='thread', score=score,
                      seqhash=True, t_final=True, chunk=chunk)
            b.run(seed=seed)
            torch_cuda.cuda.synchronize()
            check_batch(torch_cuda, b, 0, o, 300)


@pytest.mark.parametrize('R', [3, 4, 6, 8, 9, 12, 16, 17, 24, 32])
@pytest.mark.parametrize('lists', [False, True])
@pytest.mark.parametrize('method', ['direct', 'tau'])
def test_register_engine(torch_cuda, built_lib, oracle_mod, R, lists, method):
    """Both forms of the selection (prefix sums kept or added up again)."""
    m = model(2, R, 6, 0.02, lists)
    assert packable(built_lib, m) == (0 if lists else 1)
    n = 3000
    o = oracle_mod.simulate(m, n, 0 if method == 'direct' else 1, seed=R)
    for score in (False, True):
        for kw in ({},) if method == 'direct' else (
                {'sorted_blocks': False}, {'geometry': {'round_ssa': 30}}):
            check(torch_cuda, m, o, n, method, R, score=score, **kw)


def test_ends_under_every_scheduler(torch_cuda, built_lib, oracle_mod):
    """Many sample times per step, counts that leave the int32 range,
    absorption and the step budget, in the thread kernels, the simple tau loop
    and the mode-sorted scheduler (direct forms, packed and lists)."""
    t = np.linspace(0, 20, 9).astype(np.float32)
    decay = [[1, 0], [0, 1]], [[0, 0], [1, 0]]
    grow = [[1, 0], [0, 1]], [[2, 0], [0, 2]]
    models = [
        (networks.schlogl(t_end=0.05, n_samples=300), {}),
        (networks.schlogl(t_end=0.05, n_samples=50), {'step_budget': 33}),
        (Model.mass_action(*decay, [3.0, 2.0], [30, 20], t), {}),
        (Model.mass_action(*decay, [3.0, 2.0], [30, 20], t),
         {'step_budget': 7}),
        (Model.mass_action(*grow, [40.0, 1.0], [2**31 - 40, 7],
                           np.float32([0, 1e-10, 3e-10])), {}),
        # four factors: packed descriptors
        (Model.mass_action([[1, 2], [0, 2]], [[2, 1], [0, 3]], [40.0, 1e-12],
                           [2**31 - 40, 9],
                           np.float32([0, 1e-10, 3e-10])), {}),
        # a change of 20: lists
        (Model.mass_action([[1, 0], [0, 1]], [[21, 0], [0, 0]], [40.0, 1.0],
                           [2**31 - 400, 9],
                           np.float32([0, 1e-10, 3e-10])), {})]
    assert [packable(built_lib, m) for m, _ in models] == [1] * 6 + [0]
    for m, kw in models:
        o = oracle_mod.simulate(m, MANY, 0, seed=8, **kw)
        for score in (False, True):
            check(torch_cuda, m, o, MANY, 'direct', 8, _lib.KERNEL_THREAD,
                  score=score, **kw)
        o = oracle_mod.simulate(m, MANY, 1, seed=8, **kw)
        for score in (False, True):
            for n, geo in ((MANY, {}), (700, {'round_ssa': 3}),
                           (700, {'pool_slots': 1})):
                check(torch_cuda, m, o, n, 'tau', 8, _lib.KERNEL_SORTED,
                      score=score, geometry=geo, **kw)
            check(torch_cuda, m, o, 700, 'tau', 8, _lib.KERNEL_THREAD,
                  score=score, sorted_blocks=False, **kw)


def test_staging_timeout_of_the_kernel_named(torch_cuda, built_lib):
    """Every kernel marks its trajectories when the model's staging gives up
    (the copy itself still lands)."""
    from py_stoch_b200.batch import Batch
    from py_stoch_b200.simulator import simulate
    m = model(2, 3)
    other = model(2, 3, lists=True)
    runs = [(m, 64, 'direct', _lib.KERNEL_GROUP, {}),
            (m, 3000, 'tau', _lib.KERNEL_GROUP, {}),
            (m, MANY, 'direct', _lib.KERNEL_THREAD, {}),
            (m, MANY, 'tau', _lib.KERNEL_SORTED, {}),
            (m, 3000, 'tau', _lib.KERNEL_SORTED,
             {'geometry': {'round_ssa': 40}}),
            (m, 3000, 'tau', _lib.KERNEL_THREAD, {'sorted_blocks': False}),
            (other, 300, 'direct', _lib.KERNEL_LOCKSTEP, {}),
            (other, 3000, 'tau', _lib.KERNEL_SORTED, {})]
    built_lib.pyst_test_set_staging_polls(0)
    try:
        for mm, n, method, want, kw in runs:
            assert kernel(mm, n, method, **kw) == want
            r = simulate(mm, n, method=method, mapping='thread', **kw)
            torch_cuda.cuda.synchronize()
            assert (r['status'].cpu().numpy() == _lib.TRAJ_STAGING).all()
        for chunk in (0, 128):
            b = Batch([m, other], 200, method='tau', chunk=chunk)
            assert b.lane_groups == (chunk > 0)
            b.run(seed=1)
            torch_cuda.cuda.synchronize()
            assert (b.out['status'].cpu().numpy() == _lib.TRAJ_STAGING).all()
    finally:
        built_lib.pyst_test_set_staging_polls(-1)
