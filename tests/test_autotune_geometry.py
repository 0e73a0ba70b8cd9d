"""The geometry search's candidates, buckets and cache, with the timing
replaced by a fake (no GPU).  The library's own choice is a candidate, so a
tuned small run keeps the lane groups; a size bucket that the lane groups'
line crosses has an entry on each side; entries of other kernels are not
read."""

import json
import os

import pytest

from py_stoch_b200 import _lib, autotune, networks
from py_stoch_b200.simulator import run_kernel


@pytest.fixture
def tuner(tmp_path, monkeypatch):
    if not os.path.exists(_lib.LIB_PATH):
        pytest.skip('library not built')

    class Cuda(object):
        @staticmethod
        def get_device_name(device):
            return 'some GPU'

    class Torch(object):
        cuda = Cuda

        @staticmethod
        def device(name):
            return name

    monkeypatch.setattr(autotune, '_torch', lambda: Torch)

    def make(speed):
        t = autotune.Autotuner(path=str(tmp_path / 'c.json'))
        t.calls = []

        def fake(model, n, method, geometry):
            t.calls.append((n, dict(geometry)))
            return speed(n, geometry)
        t._time_single = fake
        return t
    return make


def test_small_runs_keep_the_lane_groups(tuner):
    m = networks.schlogl()
    # (the default dispatch is the fastest)
    t = tuner(lambda n, g: 2.0 if not any(g.values()) else 1.0)
    g = t.tune_geometry(m, 5000)
    assert g == autotune.DEFAULT_GEOMETRY
    assert run_kernel(m, 5000, 'tau', geometry=g)[0] == _lib.KERNEL_GROUP
    assert len(t.calls) == 1 + len(autotune.ROUNDS) * 2 * 2
    # same size bucket, the other side of the line: measured by itself
    t2 = tuner(lambda n, g: float(g['round_ssa'] == 40) + 1.0)
    assert t2.geometry(m, 5000) == g
    assert t2.geometry(m, 60000) is None
    h = t2.tune_geometry(m, 60000)
    assert h['round_ssa'] == 40 and t2.geometry(m, 60000) == h
    assert t2.geometry(m, 5000) == g
    assert run_kernel(m, 60000, 'tau', geometry=h)[0] == _lib.KERNEL_SORTED
    # from the cache, without timing
    t3 = tuner(None)
    assert t3.tune_geometry(m, 5000) == g and t3.tune_geometry(m, 60000) == h
    assert t3.calls == []


def test_entries_of_other_kernels_are_measured_again(tuner):
    m = networks.schlogl()
    t = tuner(lambda n, g: 1.0)
    with open(t.path, 'w') as f:
        json.dump({'some GPU': {'geom/1/R8/S16/N65536': {
            'geometry': {'round_ssa': 20, 'round_leap': 2, 'pool_slots': 1,
                         'sorted_block': 448}}}}, f)
    t = tuner(lambda n, g: 1.0)
    assert t.geometry(m, 60000) is None
    t.tune_geometry(m, 60000)
    assert t.calls
    with open(t.path) as f:
        data = json.load(f)
    assert len(data) == 2 and 'geom/1/R8/S16/N65536' in data['some GPU']
