"""Workloads on which the engine's speed is judged, through its public entry
points: single-model runs (direct method, tau-leaping, general kinetic laws),
gradients, the gradient reduction by itself, batched sweeps and the drop-in
classes, from a call of a few microseconds of work to the full-size runs.

A case is a dict of plain values.  ``prepare`` builds what a program holds
before the call, ``run`` is one call, ``work`` its bytes and floating-point
operations, ``exact`` the FP64 value of the outputs that have one (the
simulations have none: their outputs are random draws).
"""

import math

import numpy as np
import torch

from py_stoch_b200 import kinetic, networks, sbml, sim_maker
from py_stoch_b200.autograd import sampled_moments, score_backward
from py_stoch_b200.batch import Batch
from py_stoch_b200.model import Model
from py_stoch_b200.shard import KernelOps
from py_stoch_b200.simulator import CuTauLeaping, device_blob, simulate


def listed():
    return [
        # the headline run: plain tau-leaping, every trajectory sampled
        # 200 times
        {'name': 'tau_schlogl_262144', 'kind': 'tau', 'net': 'schlogl',
         'n': 262144, 't_end': 5.0, 'samples': 200},
        # an ordinary tau-leaping run of an odd size, far from filling the
        # GPU: one parameter point of an interactive study
        {'name': 'tau_schlogl_4999', 'kind': 'tau', 'net': 'schlogl',
         'n': 4999, 't_end': 5.0, 'samples': 200},
        # tau-leaping of an oscillating network: leaps of large counts, few
        # fallback steps
        {'name': 'tau_lv_20011', 'kind': 'tau', 'net': 'lv', 'n': 20011,
         't_end': 10.0, 'samples': 100},
        # the reference's Lotka-Volterra direct-method run: few, long
        # trajectories
        {'name': 'direct_lv_1024', 'kind': 'direct', 'net': 'lv', 'n': 1024,
         't_end': 10.0, 'samples': 100},
        # the smallest call: launch, allocation and host work count
        {'name': 'direct_telegraph_32', 'kind': 'direct', 'net': 'telegraph',
         'n': 32, 't_end': 1.0, 'samples': 5},
        # a gradient of sampled moments: forward with scores, backward
        {'name': 'grad_telegraph_1048576', 'kind': 'grad', 'n': 1048576,
         't_end': 50.0, 'samples': 20},
        # the moments and the gradient reduction alone, on samples and
        # scores a run has left on the GPU (a second loss on one run)
        {'name': 'reduce_1048576', 'kind': 'reduce', 'n': 1048576,
         'kappa': 1, 'samples': 20, 'reactions': 6},
        # a parameter sweep in one launch with scores, in-kernel statistics
        # and their Jacobians
        {'name': 'sweep_64x256', 'kind': 'sweep', 'sets': 64, 'n': 256,
         'samples': 50, 'budget': 30000},
        # uneven networks in one launch, enough trajectories to fill the GPU
        # thread by thread
        {'name': 'synthetic_1024x61', 'kind': 'synthetic', 'nets': 1024,
         'n': 61, 'method': 'tau', 'budget': 2000},
        # the same networks in a small batch (large networks then take a
        # warp per trajectory)
        {'name': 'synthetic_150x48', 'kind': 'synthetic', 'nets': 150,
         'n': 48, 'method': 'direct', 'budget': 2000},
        # general kinetic laws (saturation, integer division, square root)
        {'name': 'laws_direct_10007', 'kind': 'laws', 'method': 'direct',
         'n': 10007, 't_end': 1.0, 'samples': 20},
        # the drop-in class from parsed SBML arguments to a NumPy array
        {'name': 'dropin_direct_50000', 'kind': 'dropin', 'gillespie': 1,
         'n': 50000, 't_end': 5, 'samples': 50},
    ]


def _log_int(rng, lo, hi):
    """A whole number in [lo, hi], even over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo),
                                                          math.log(hi)))))))


def _log(rng, lo, hi):
    return round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 3)


def draw(rng):
    kind = rng.choice(['tau', 'tau', 'direct', 'direct', 'grad', 'reduce',
                       'sweep', 'synthetic', 'synthetic', 'laws', 'dropin'])
    c = {'kind': kind}
    if kind == 'tau':
        c['net'] = rng.choice(['schlogl', 'lv'])
        if c['net'] == 'schlogl':
            c.update(n=_log_int(rng, 200, 250000), t_end=_log(rng, 1, 5),
                     samples=_log_int(rng, 10, 200))
        else:
            c.update(n=_log_int(rng, 200, 20000), t_end=_log(rng, 1, 10),
                     samples=_log_int(rng, 10, 100))
    elif kind == 'direct':
        c['net'] = rng.choice(['lv', 'telegraph', 'schlogl'])
        if c['net'] == 'lv':
            n = _log_int(rng, 32, 20000)
            c.update(n=n, t_end=_log(rng, 0.1, max(0.2, min(
                10.0, 10.0 * 4096 / n))), samples=_log_int(rng, 10, 100))
        elif c['net'] == 'telegraph':
            c.update(n=_log_int(rng, 32, 500000), t_end=_log(rng, 1, 50),
                     samples=_log_int(rng, 5, 50))
        else:
            c.update(n=_log_int(rng, 32, 100000), t_end=_log(rng, 0.5, 5),
                     samples=_log_int(rng, 10, 200))
    elif kind == 'grad':
        c.update(n=_log_int(rng, 1000, 1000000), t_end=_log(rng, 5, 50),
                 samples=_log_int(rng, 5, 20))
    elif kind == 'reduce':
        c.update(n=_log_int(rng, 1000, 1000000),
                 kappa=rng.randint(1, 2), samples=_log_int(rng, 5, 50),
                 reactions=rng.randint(2, 32))
    elif kind == 'sweep':
        c.update(sets=_log_int(rng, 8, 64), n=_log_int(rng, 32, 256),
                 samples=_log_int(rng, 10, 50), budget=_log_int(rng, 2000,
                                                                30000))
    elif kind == 'synthetic':
        nets = _log_int(rng, 16, 1024)
        c.update(nets=nets, n=rng.randint(16, 64),
                 method=rng.choice(['tau', 'direct']),
                 budget=_log_int(rng, 200, 2000))
    elif kind == 'laws':
        c.update(method=rng.choice(['direct', 'tau']),
                 n=_log_int(rng, 100, 10000), t_end=_log(rng, 0.1, 1),
                 samples=_log_int(rng, 5, 50))
    else:
        c.update(gillespie=rng.randint(0, 1), n=_log_int(rng, 100, 50000),
                 t_end=rng.randint(1, 5), samples=_log_int(rng, 5, 50))
    return c


def _net(c):
    if c['net'] == 'schlogl':
        return networks.schlogl(t_end=c['t_end'], n_samples=c['samples'])
    if c['net'] == 'lv':
        return networks.lotka_volterra(t_end=c['t_end'],
                                       n_samples=c['samples'])
    return networks.telegraph(t_end=c['t_end'], n_samples=c['samples'])


def _law_model(t_end, samples, scale):
    """An enzyme-like conversion with saturation, a C integer division and a
    square root, and a catalyst species that keeps the reactions alive."""
    laws = ['parameter_0 * species_0 / (parameter_1 + species_0)',
            'species_1 / 3 * parameter_2 + sqrt(species_2)', None]
    rate = [4000.0 * scale[0], 5000.0 * scale[1], 0.7 * scale[2]]
    pre = np.eye(3, dtype=np.int64)
    post = np.array([[0, 1, 0], [1, 0, 0], [0, 0, 1]])
    progs = [None if t is None else kinetic.compile_law(t, 3, rate)[:2]
             for t in laws]
    order = np.where([[t is None for t in laws]] * 3, pre, 0)
    times = np.linspace(0.0, t_end, samples).astype(np.float32)
    return Model(order, pre, post - pre, [0.0, 0.0, rate[2]],
                 [30000, 2000, 4], times, np.arange(3), laws=progs)


def prepare(case, seed):
    c = dict(case)
    kind = c['kind']
    rng = np.random.default_rng(seed)
    st = {'case': c, 'seed': int(seed)}
    if kind in ('tau', 'direct', 'grad'):
        # rate constants within 2% of the nominal ones
        m = networks.telegraph(t_end=c['t_end'], n_samples=c['samples']) \
            if kind == 'grad' else _net(c)
        m = m.with_rates(m.rate * np.exp(rng.uniform(-0.02, 0.02,
                                                     m.n_reactions)))
        st['model'] = m
        if kind == 'grad':
            st['log_rates'] = torch.tensor(
                np.log(m.rate), dtype=torch.float64, device='cuda',
                requires_grad=True)
            st['target'] = torch.from_numpy(rng.normal(
                size=(m.kappa, m.ita))).cuda()
        else:
            st['blob'] = device_blob(m, 'cuda')
    elif kind == 'laws':
        st['model'] = _law_model(c['t_end'], c['samples'],
                                 np.exp(rng.uniform(-0.02, 0.02, 3)))
        st['blob'] = device_blob(st['model'], 'cuda')
    elif kind == 'reduce':
        g = torch.Generator(device='cuda')
        g.manual_seed(int(seed))
        kf = c['kappa'] * c['samples']
        level = torch.linspace(50.0, 900.0, kf, device='cuda',
                               dtype=torch.float64)
        x = torch.randn((kf, c['n']), generator=g, device='cuda',
                        dtype=torch.float64)
        x = torch.clamp(torch.round(level[:, None] +
                                    x * torch.sqrt(level)[:, None]), min=0)
        st['samples'] = x.to(torch.int32).view(c['kappa'], c['samples'],
                                               c['n'])
        st['score'] = torch.randn((c['n'], c['reactions']), generator=g,
                                  device='cuda', dtype=torch.float64) * 8.0
        for k, s in (('gmean', 1.0), ('gvar', 0.03)):
            st[k] = s * torch.randn((c['kappa'], c['samples']), generator=g,
                                    device='cuda', dtype=torch.float64)
    elif kind == 'sweep':
        models, _ = networks.parameter_sweep(c['sets'], seed=int(seed),
                                             n_samples=c['samples'])
        st['batch'] = Batch(models, c['n'], method='tau', score=True,
                            stats=True, jacobian=True)
    elif kind == 'synthetic':
        # the same networks at every seed, their rates within 2%
        models = [m.with_rates(m.rate * np.exp(rng.uniform(-0.02, 0.02,
                                                           m.n_reactions)))
                  for m in networks.synthetic_networks(c['nets'], seed=0)]
        st['batch'] = Batch(models, c['n'], method=c['method'])
    else:
        scale = np.exp(rng.uniform(-0.02, 0.02, 4))
        p = networks.SCHLOGL_NOMINAL
        st['args'] = sim_maker.TLArgsList.make_list(
            sbml.read_sbml_string(sbml.schlogl_sbml()), [[250]],
            [[float(p[k] * s)] for k, s in zip(('c1', 'c2', 'c3', 'c4'),
                                               scale)] +
            [[p['A']], [p['B']]], [0], c['t_end'], c['samples'], c['n'],
            gillespie=c['gillespie'])[0]
    return st


def run(state):
    c, seed = state['case'], state['seed']
    kind = c['kind']
    if kind in ('tau', 'direct', 'laws'):
        r = simulate(state['model'], c['n'],
                     method=c['method'] if kind == 'laws' else kind,
                     seed=seed, d_blob=state['blob'])
        return {k: r[k] for k in ('samples', 'status', 'events')}
    if kind == 'grad':
        logk = state['log_rates']
        mean, var = sampled_moments(state['model'], logk, c['n'], seed=seed)
        loss = ((mean - state['target']) ** 2).sum() + var.sum()
        (g,) = torch.autograd.grad(loss, logk)
        return {'mean': mean.detach(), 'var': var.detach(), 'grad': g}
    if kind == 'reduce':
        ops = KernelOps()
        x = state['samples']
        mean, var = ops.moments(ops.sample_sums(x), c['n'], c['kappa'],
                                c['samples'])
        g = score_backward(x, state['score'], mean, var, state['gmean'],
                           state['gvar'])
        return {'mean': mean, 'var': var, 'grad': g}
    if kind in ('sweep', 'synthetic'):
        b = state['batch']
        b.run(seed=seed, step_budget=c['budget'])
        return b.out
    return {'samples': CuTauLeaping(seed=seed).run(state['args'])}


# per unit of simulated time and trajectory: direct-method steps, leaps
_STEPS = {('tau', 'schlogl'): (990.0, 113.0), ('tau', 'lv'): (63.0, 332.0),
          ('direct', 'schlogl'): (3700.0, 0.0),
          ('direct', 'lv'): (30000.0, 0.0),
          ('direct', 'telegraph'): (145.0, 0.0), ('laws', ''): (4000.0, 0.0)}
_REACTIONS = {'schlogl': 4, 'lv': 3, 'telegraph': 6, '': 3}


def _step_flops(reactions):
    # propensities, total, selection, logarithm, clock
    return 4.0 * reactions + 30.0


def work(case):
    c = dict(case)
    kind, n = c['kind'], float(c['n'])
    if kind == 'reduce':
        kf = c['kappa'] * c['samples']
        return {'bytes': n * (4.0 * kf + 8.0 * c['reactions']),
                'flops': n * (7.0 * kf + 2.0 * c['reactions'])}
    if kind in ('sweep', 'synthetic'):
        if kind == 'sweep':
            traj, rows, r, steps = n * c['sets'], 1.5 * c['samples'], 3.5, \
                min(c['budget'], 30000.0)
            score = 8.0 * r
        else:
            traj, rows, r, steps = n * c['nets'], 34.5 * 50, 132.0, \
                0.95 * c['budget']
            score = 0.0
        return {'bytes': traj * (4.0 * rows + 9.0 + score),
                'flops': traj * steps * _step_flops(r)}
    if kind == 'dropin':
        key = ('direct' if c['gillespie'] else 'tau', 'schlogl')
    elif kind == 'laws':
        key = ('laws', '')
    elif kind == 'grad':
        key = ('direct', 'telegraph')
    else:
        key = (kind, c['net'])
    r = _REACTIONS[key[1]]
    rows = c['samples'] * {'schlogl': 1, 'lv': 2, 'telegraph': 1,
                           '': 3}[key[1]]
    ssa, leaps = _STEPS[key]
    flops = n * c['t_end'] * (ssa * _step_flops(r) + leaps * 60.0 * r)
    out = 4.0 * rows + 9.0 + (8.0 * r if kind == 'grad' else 0.0)
    return {'bytes': n * out, 'flops': flops}


def exact(case, seed):
    if case['kind'] != 'reduce':
        return None
    st = prepare(case, seed)
    x = st['samples'].double()
    n = x.shape[2]
    mean = x.mean(dim=2)
    d = x - mean[..., None]
    var = (d * d).mean(dim=2)
    h = (st['gmean'][..., None] * d +
         st['gvar'][..., None] * (d * d - var[..., None])).sum(dim=(0, 1))
    return {'mean': mean, 'var': var, 'grad': h @ st['score'] / n}
