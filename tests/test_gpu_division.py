"""The straight-line divisions and the uniforms against the correctly rounded
quotient and the integer conversion, bit for bit: over the ranges they are
used in, for significands next to 1 and 2, and for the quotients nearest to
the middle between two doubles that exist (for an odd divisor B one dividend
for each side, solved for with the inverse of 2^53 modulo B)."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(torch, lib, which, a, b):
    x = np.empty((a.size, 2))
    x[:, 0], x[:, 1] = a, b
    d = torch.from_numpy(x).cuda()
    out = torch.empty(a.size, dtype=torch.float64, device='cuda')
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.pyst_test_math(d.data_ptr(), a.size, which, out.data_ptr(),
                              s) == 0
    return out.cpu().numpy()


def same(got, want):
    np.testing.assert_array_equal(got.view(np.uint64), want.view(np.uint64))


def hard_pairs(divisors):
    """Dividends A in [2^52, 2^53) whose quotient by the odd B lies 1 / (2 B)
    from a midpoint: A 2^s - B (2 M + 1) = +-1 with s = 53 (A >= B) or 54."""
    out = []
    for B in divisors:
        for s in (53, 54):
            inv = pow(pow(2, s, B), -1, B)
            for k in (1, -1):
                A = inv * k % B
                for A in (A, A + B):
                    if not 2**52 <= A < 2**53 or (A >= B) != (s == 53):
                        continue
                    q = (A * 2**s - k) // B
                    if (A * 2**s - k) % B == 0 and q % 2 == 1:
                        out.append((A, B))
    return np.array(out, np.int64).reshape(-1, 2).astype(np.float64).T


def test_double_division(torch_cuda, built_lib):
    rng = np.random.default_rng(7)
    n = 1000000
    u = rng.integers(1, 2**53, n) * 2.0**-53
    e = -np.log(u)
    tot = np.exp(rng.uniform(np.log(2.0**-149), np.log(2.0**127), n))
    f = rng.uniform(np.sqrt(0.5), np.sqrt(2.0), n)
    near2 = 2.0 - rng.integers(1, 2**20, n) * 2.0**-52
    near1 = 1.0 + rng.integers(0, 2**20, n) * 2.0**-52
    m = 1.0 + rng.integers(0, 2**52, n) * 2.0**-52
    for a, b in ((e, tot), (f - 1.0, f + 1.0), (m, near2), (m, near1),
                 (near2, near2[::-1]), (near2, near1), (near1, near2),
                 (np.zeros(n), tot), (m[::-1], m),
                 (e, np.float32(tot).astype(np.float64) + 0.0)):
        ok = b > 0
        a, b = np.ascontiguousarray(a[ok]), np.ascontiguousarray(b[ok])
        want = a / b
        same(run(torch_cuda, built_lib, 5, a, b), want)
        same(run(torch_cuda, built_lib, 6, a, b), want)


def test_logarithm_next_to_one(torch_cuda, built_lib, oracle_mod):
    """Arguments whose division has the divisors next to 2."""
    import ctypes
    k = np.arange(-4000, 4000)
    x = np.concatenate([1.0 + np.where(k < 0, 2.0**-53, 2.0**-52) * k,
                        0.5 * (1.0 - np.arange(1, 4000) * 2.0**-53)])
    d = torch_cuda.from_numpy(x).cuda()
    out = torch_cuda.empty_like(d)
    s = ctypes.c_void_p(torch_cuda.cuda.current_stream().cuda_stream)
    assert built_lib.pyst_test_math(d.data_ptr(), x.size, 0, out.data_ptr(),
                                    s) == 0
    same(out.cpu().numpy(), oracle_mod.math(x, 0))


@pytest.mark.parametrize('where', ['next to 2', 'below 2', 'any', 'next to 1'])
def test_double_division_hard_cases(torch_cuda, built_lib, where):
    rng = np.random.default_rng(11)
    c = 20000
    B = {'next to 2': 2**53 - np.arange(1, 2 * c, 2),
         'below 2': 2**53 - np.unique(
             np.exp(rng.uniform(0, np.log(2.0**44), c)).astype(np.int64)) | 1,
         'any': rng.integers(2**52, 2**53, c) | 1,
         'next to 1': 2**52 + np.arange(1, 2 * c, 2)}[where]
    a, b = hard_pairs([int(x) for x in B if x < 2**53])
    assert a.size > c // 4
    bad = run(torch_cuda, built_lib, 5, a, b) != a / b
    assert not bad.any(), (int(bad.sum()), a[bad][:4], b[bad][:4])


def test_float_division(torch_cuda, built_lib):
    rng = np.random.default_rng(8)
    n = 2000000
    lam = np.exp(rng.uniform(np.log(10.0), np.log(1e9), n)).astype(np.float32)
    b = np.float32(0.931) + np.float32(2.53) * np.sqrt(lam)
    us = (rng.integers(1, 2**23, n) * 2.0**-24).astype(np.float32)
    two_a = np.float32(2) * (np.float32(-0.059) + np.float32(0.02483) * b)
    m1 = (1 + rng.integers(0, 2**23, n) * 2.0**-23).astype(np.float32)
    m2 = (2 - rng.integers(1, 2**12, n) * 2.0**-23).astype(np.float32)
    for p, q in ((np.full(n, np.float32(3.6224)), b - np.float32(2)),
                 (two_a, us), (m1, m2), (m1, m1[::-1]), (m2, m2[::-1])):
        p, q = np.ascontiguousarray(p), np.ascontiguousarray(q)
        want = (p / q).astype(np.float64)
        same(run(torch_cuda, built_lib, 7, p, q), want)
        same(run(torch_cuda, built_lib, 8, p, q), want)


@pytest.mark.parametrize('c', [1, 2, 3, 4])
def test_float_division_below_a_power_of_two(torch_cuda, built_lib, c):
    """Every dividend's significand for the divisors next to 2."""
    b = np.float32(2 - c * 2.0**-23)
    for lo in range(0, 2**23, 2**21):
        a = (1 + np.arange(lo, lo + 2**21) * 2.0**-23).astype(np.float32)
        b_all = np.full(a.size, b)
        same(run(torch_cuda, built_lib, 7, a, b_all),
             (a / b_all).astype(np.float64))


def test_uniforms(torch_cuda, built_lib):
    rng = np.random.default_rng(9)
    w = rng.integers(0, 2**32, (1000000, 2))
    ends = np.array([0, 1, 2047, 2048, 2**31, 2**32 - 2048, 2**32 - 2049,
                     2**32 - 1])
    w = np.concatenate([w, np.stack(np.meshgrid(ends, ends), -1).reshape(
        -1, 2)])
    hi, lo = w[:, 0].astype(np.float64), w[:, 1].astype(np.float64)
    want = ((w[:, 0] << 21 | w[:, 1] >> 11) + 1).astype(np.float64) * 2.0**-53
    same(run(torch_cuda, built_lib, 9, hi, lo), want)
