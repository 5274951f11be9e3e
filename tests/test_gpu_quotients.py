"""The square root, its reciprocal and the quotients that the factorisation forms
by correction steps (chol_tc.cuh) against CUDA's own, which are correctly
rounded: within a unit in the last place, 1 / sqrt within two (the reference is
a rounded root's rounded reciprocal, off by one itself); and the scaling of the
Gram (gram_tc.cuh) against long double."""
import ctypes as C

import numpy as np
import pytest

import native

pytestmark = pytest.mark.gpu

N = 1 << 20


@pytest.fixture(scope="module")
def lib(gpu_lib, tmp_path_factory):
    return C.CDLL(native.shared_object("kernel_hooks.cu", tmp_path_factory.mktemp("hooks")))


def _call(f, n, *arrays):
    f.restype = C.c_int
    f.argtypes = [C.c_int] + [C.c_void_p] * len(arrays)
    assert f(n, *(a.data_ptr() for a in arrays)) == 0


def _ulps(got, ref):
    """Places apart: the difference of the bit patterns of two numbers of one sign."""
    import torch
    assert torch.equal(torch.signbit(got), torch.signbit(ref))
    return int((got.view(torch.int64) - ref.view(torch.int64)).abs().max())


def _numbers(gen, n, lo, hi, edges=True):
    """Mantissas all over [1, 2), those next to its ends among them, exponents uniform in lo .. hi."""
    import torch
    m = 1.0 + torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)
    if edges:
        k = torch.arange(n // 8, device="cuda", dtype=torch.float64)
        m[: n // 8] = 1.0 + (k % 4096) * 2.0 ** -52
        m[n // 8: 2 * (n // 8)] = 2.0 - (1.0 + k % 4096) * 2.0 ** -52
    e = torch.randint(lo, hi + 1, (n,), device="cuda", generator=gen)
    return torch.ldexp(m, e)


@pytest.mark.parametrize("lo,hi", [(-2, 20), (-99, 98), (-300, -101), (101, 300)])
def test_root_reciprocal_and_quotient(lib, lo, hi):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(hi)
    b = _numbers(gen, N, lo, hi)
    a = _numbers(gen, N, -40, 40) * (1 - 2 * (torch.rand(N, device="cuda", generator=gen) < 0.5).double())
    root, inv, quot = (torch.empty(N, dtype=torch.float64, device="cuda") for _ in range(3))
    ref = torch.empty(3 * N, dtype=torch.float64, device="cuda")
    _call(lib.hook_quotients, N, a, b, root, inv, quot, ref)
    assert _ulps(root, ref[:N]) <= 1
    assert _ulps(inv, ref[N:2 * N]) <= 2
    assert _ulps(quot, ref[2 * N:]) <= 1


def test_gram_scaling(lib):
    """num / sqrt(pa qa pb qb) in long double: one rounding of a value that is known to a few 2^-100, so half a unit, and
    0 for a monomorphic SNP.  Frequencies of counts in up to 200,000 chromosomes, rare ones and near 1 among them, and
    pairs of the same SNP."""
    import torch
    n = 100000
    rng = np.random.default_rng(7)
    f = np.concatenate([rng.integers(1, 2000, 2 * n // 2) / 2000.0, rng.integers(1, 200000, n) / 200000.0])
    f[1::7] = 1.0 - 10.0 ** (-5.5 * rng.random(f[1::7].size))
    f[2::7] = 10.0 ** (-5.5 * rng.random(f[2::7].size))
    f[n:n + n // 4] = f[:n // 4]
    f[5], f[n + 6], f[7] = 0.0, 1.0, 1.0
    num = rng.standard_normal(n) * 10.0 ** rng.uniform(-3, 7, n)
    d = [torch.from_numpy(x).cuda() for x in (num, f, np.empty(n))]
    _call(lib.hook_gram_scaled, n, *d)
    got = d[2].cpu().numpy()
    assert got[5] == got[6] == got[7] == 0.0
    keep = np.ones(n, dtype=bool)
    keep[5:8] = False
    a, b = f[:n].astype(np.longdouble)[keep], f[n:].astype(np.longdouble)[keep]
    want = num[keep] / (np.sqrt(2 * a * (1 - a)) * np.sqrt(2 * b * (1 - b)))
    ulp = np.spacing(np.abs(got[keep]))
    assert np.max(np.abs((got[keep] - want) / ulp)) <= 0.51
