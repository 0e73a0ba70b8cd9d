"""The gradient reduction on both sides of the line between score tiles in
shared memory and a thread per column, and past one block's threads, against
the NumPy restatement of the same operations: bit for bit.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('U', [1, 255, 257, 4097])
@pytest.mark.parametrize('R', [15, 31, 32, 33, 48, 256, 257, 600])
def test_columns(torch_cuda, built_lib, U, R):
    from py_stoch_b200.shard import KernelOps
    from test_shard_gloo import NumpyOps
    torch = torch_cuda
    rng = np.random.default_rng(U + R)
    kappa, ita = 2, 7
    smp = rng.integers(0, 3000, size=(kappa, ita, U)).astype(np.int32)
    score = rng.normal(size=(U, R))
    gm = rng.normal(size=(kappa, ita))
    gv = rng.normal(size=(kappa, ita)) / 30.0
    k, n = KernelOps(), NumpyOps()
    x = torch.from_numpy(smp).cuda()
    mean, var = k.moments(k.sample_sums(x), U, kappa, ita)
    nm, nv = n.moments(n.sample_sums(smp).numpy(), U, kappa, ita)
    part = k.score_partials(x, torch.from_numpy(score).cuda(), mean, var,
                            torch.from_numpy(gm).cuda(),
                            torch.from_numpy(gv).cuda())
    npart = n.score_partials(smp, score, nm, nv, gm, gv).numpy()
    np.testing.assert_array_equal(part.cpu().numpy(), npart)
    np.testing.assert_array_equal(k.score_combine(part, U).cpu().numpy(),
                                  n.score_combine(npart, U))
