"""The gradient reduction and the sample sums at the edges of their tiles
(256-trajectory chunks, 16-column score tiles, 64-row final tiles, 4096
sample chunks, rows aligned for 16-byte loads or not), against the NumPy
restatement of the same operations: bit for bit.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('U', [1, 255, 256, 257, 4096, 4097, 16640])
@pytest.mark.parametrize('kappa,ita,R', [(1, 1, 1), (1, 8, 16), (2, 5, 17),
                                         (1, 9, 33), (3, 3, 70)])
def test_reductions(torch_cuda, built_lib, U, kappa, ita, R):
    from py_stoch_b200.shard import KernelOps
    from test_shard_gloo import NumpyOps
    torch = torch_cuda
    rng = np.random.default_rng(U + R)
    smp = rng.integers(0, 2**31 - 1 if U < 300 else 3000,
                       size=(kappa, ita, U)).astype(np.int32)
    score = rng.normal(size=(U, R))
    gm = rng.normal(size=(kappa, ita))
    gv = rng.normal(size=(kappa, ita)) / 30.0
    k, n = KernelOps(), NumpyOps()
    # (the second copy starts off a 16-byte boundary)
    flat = torch.zeros(smp.size + 1, dtype=torch.int32, device='cuda')
    flat[1:] = torch.from_numpy(smp.ravel()).cuda()
    for x in (torch.from_numpy(smp).cuda(), flat[1:].view(kappa, ita, U)):
        sums = k.sample_sums(x)
        np.testing.assert_array_equal(sums.cpu().numpy(),
                                      n.sample_sums(smp).numpy())
    mean, var = k.moments(sums, U, kappa, ita)
    nm, nv = n.moments(sums.cpu().numpy(), U, kappa, ita)
    np.testing.assert_array_equal(mean.cpu().numpy(), nm)
    part = k.score_partials(x, torch.from_numpy(score).cuda(), mean, var,
                            torch.from_numpy(gm).cuda(),
                            torch.from_numpy(gv).cuda())
    npart = n.score_partials(smp, score, nm, nv, gm, gv).numpy()
    np.testing.assert_array_equal(part.cpu().numpy(), npart)
    np.testing.assert_array_equal(k.score_combine(part, U).cpu().numpy(),
                                  n.score_combine(npart, U))
