"""The Poisson sampler's FP32 decisions against the oracle's FP64 sampler, at
the means where a decision can go wrong: the smallest and the largest
inversion means, the switch to PTRS and its smallest counts (k < 4), means
whose counts leave the series' range (|k - lam| > (k + lam) / 2 is common
only for small means) and means up to the largest one supported.  Every draw
is equal: a decision that FP32 cannot take goes to FP64.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('lo,hi', [
    (1e-9, 1e-3), (1e-3, 1.0), (1.0, 9.999999), (9.9, 10.1), (10.0, 14.0),
    (14.0, 60.0), (60.0, 1e3), (1e3, 1e6), (1e6, 1e9)])
def test_sampler_decisions(torch_cuda, built_lib, oracle_mod, lo, hi):
    torch = torch_cuda
    rng = np.random.default_rng(int(hi * 7) % 1000)
    lam = np.exp(rng.uniform(np.log(lo), np.log(hi), 300000)).astype(
        np.float32)
    dl = torch.from_numpy(lam).cuda()
    dk = torch.empty(lam.size, dtype=torch.int32, device='cuda')
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for seed in (5, 6):
        assert built_lib.pyst_test_poisson(dl.data_ptr(), lam.size, seed,
                                           dk.data_ptr(), s) == 0
        np.testing.assert_array_equal(dk.cpu().numpy(),
                                      oracle_mod.poisson(lam, seed))
