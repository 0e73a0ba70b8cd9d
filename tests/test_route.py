"""The dispatch of single-model runs and the lanes of batched models, on the
CPU: which kernel a run takes, on both sides of every line.  Without a GPU
the lines are those of 148 SMs.
"""

import ctypes as C

import numpy as np
import pytest

from py_stoch_b200 import _lib, kinetic, networks
from py_stoch_b200.model import Model

SMS = 148


@pytest.fixture(scope='module')
def lib():
    import os
    if not os.path.exists(_lib.LIB_PATH):
        pytest.skip('library not built')
    import torch
    if torch.cuda.is_available():
        global SMS
        SMS = torch.cuda.get_device_properties(0).multi_processor_count
    return _lib.lib()


def route(lib, m, n, method, mapping=0, score=0, flags=0, **geo):
    r = _lib.RunDesc(n, 0, 0, method, mapping, 100, 63, 0, 0, flags,
                     geo.get('round_ssa', 0), geo.get('round_leap', 0),
                     geo.get('pool_slots', 0), geo.get('sorted_block', 0))
    k, lanes = C.c_int32(), C.c_int32()
    rc = lib.pyst_run_kernel(m.blob().ctypes.data, C.byref(r), score,
                             C.byref(k), C.byref(lanes))
    return rc if rc else (k.value, lanes.value)


def test_small_models(lib):
    m = networks.schlogl()
    for score in (0, 1):
        # most lanes first, then a thread per trajectory
        seen = [route(lib, m, n * SMS, 0, score=score)
                for n in range(1, 400)]
        assert seen[0] == (_lib.KERNEL_GROUP, 32)
        lanes = [x[1] for x in seen]
        assert lanes == sorted(lanes, reverse=True)
        assert seen[-1] == (_lib.KERNEL_THREAD, 1)
        assert {4, 8} <= set(lanes)
        seen = [route(lib, m, n * SMS, 1, score=score)
                for n in range(1, 400)]
        assert [x[1] for x in seen] == sorted([x[1] for x in seen],
                                              reverse=True)
        assert seen[-1] == (_lib.KERNEL_SORTED, 1)
    # an explicit geometry or the simple loop names the kernel
    for geo in ({'round_ssa': 40}, {'round_leap': 4}, {'pool_slots': 1},
                {'sorted_block': 448}):
        assert route(lib, m, 100, 1, **geo) == (_lib.KERNEL_SORTED, 1)
        assert route(lib, m, 100, 0, **geo)[0] == _lib.KERNEL_GROUP
    assert route(lib, m, 100, 1, flags=_lib.FLAG_UNSORTED) == (
        _lib.KERNEL_THREAD, 1)
    assert route(lib, m, 100, 1, mapping=_lib.MAP_WARP) == (
        _lib.KERNEL_WARP, 32)


def test_other_models(lib):
    # three changed species: not packable
    m = Model.mass_action([[1, 0], [1, 0], [0, 1]],
                          [[0, 1], [0, 0], [1, 0]], [1.0, 2.0], [9, 9, 9],
                          np.float32([0, 1]))
    assert lib.pyst_test_model_packable(m.blob().ctypes.data) == 0
    assert route(lib, m, 16 * SMS, 0) == (_lib.KERNEL_LOCKSTEP, 32)
    assert route(lib, m, 16 * SMS + 1, 0) == (_lib.KERNEL_THREAD, 1)
    assert route(lib, m, 16 * SMS, 0, score=1) == (_lib.KERNEL_THREAD, 1)
    assert route(lib, m, 10, 1) == (_lib.KERNEL_SORTED, 1)
    assert lib.pyst_batch_lanes(m.blob().ctypes.data) == 0
    big = networks.synthetic_networks(1, seed=3, r_range=(40, 40))[0]
    assert route(lib, big, 32 * SMS, 0) == (_lib.KERNEL_WARP, 32)
    assert route(lib, big, 32 * SMS + 1, 0) == (_lib.KERNEL_THREAD, 1)
    assert route(lib, big, 32 * SMS + 1, 0, score=1) == (_lib.KERNEL_WARP, 32)
    assert route(lib, big, 10, 0, mapping=_lib.MAP_THREAD, score=1) == 3
    rate = [2.0, 3.0]
    prog = kinetic.compile_law('parameter_0 * species_0 / (parameter_1 + '
                               'species_0)', 2, rate)[:2]
    laws = Model(np.zeros((2, 2), np.int64), np.eye(2, dtype=np.int64),
                 np.array([[-1, 1], [1, -1]]), [0.0, 3.0], [50, 50],
                 np.float32([0, 1]), np.arange(2), laws=[prog, None])
    assert route(lib, laws, 5000, 1) == (_lib.KERNEL_THREAD, 1)
    assert route(lib, laws, 100, 0) == (_lib.KERNEL_LOCKSTEP, 32)
    assert route(lib, laws, 100, 0, score=1) == 3
    assert lib.pyst_batch_lanes(laws.blob().ctypes.data) == 0


def test_batch_lanes(lib):
    assert lib.pyst_batch_lanes(networks.schlogl().blob().ctypes.data) == 4
    assert lib.pyst_batch_lanes(networks.telegraph().blob().ctypes.data) == 8
    four = Model.mass_action([[2], [2]], [[1], [3]], [1.0], [9, 9],
                             np.float32([0, 1]))
    assert lib.pyst_test_model_packable(four.blob().ctypes.data) == 1
    assert lib.pyst_batch_lanes(four.blob().ctypes.data) == 0
