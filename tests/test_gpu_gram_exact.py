"""The genotype Gram's counts are exact up to the limits that its dispatch
states: FP32 sums of products 0, 1, 2 and 4 up to 2^24 on the tensor cores, for
up to 2^22 individuals, and integer sums beyond.

With every frequency 1/2 the scaled entry is (S - n) / sqrt(1/2)^2, so the
integer S comes back by rounding.  The codes are mostly 2 with odd numbers of
ones, which makes the sums large and their last bit matter; a zero here and
there makes them differ from SNP to SNP."""
import ctypes as C

import numpy as np
import pytest

import native

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hook(gpu_lib, tmp_path_factory):
    lib = C.CDLL(native.shared_object("kernel_hooks.cu", tmp_path_factory.mktemp("hooks")))
    f = lib.hook_gram
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.POINTER(C.c_int)]
    return f


def _codes(n, p, ones):
    """[p][ldx] int8 on the GPU: all 2, of which `ones[k]` of SNP k are 1 and k of it 0, at its own places."""
    import torch
    ldx = (n + 127) // 128 * 128
    g = torch.zeros((p, ldx), dtype=torch.int8, device="cuda")
    g[:, :n] = 2
    gen = torch.Generator().manual_seed(n + p)
    for k in range(p):
        at = torch.randperm(n, generator=gen)[:ones[k] + k].cuda()
        g[k, at[:ones[k]]] = 1
        g[k, at[ones[k]:]] = 0
    return g


def _counts(g, n):
    """S = sum_i g_ia g_ib in 64-bit integers, from counts of the codes."""
    import torch
    p = g.shape[0]
    s = torch.zeros((p, p), dtype=torch.int64)
    for a in range(p):
        s[a] = (g[a:a + 1, :n].to(torch.int16) * g[:, :n].to(torch.int16)).sum(dim=1, dtype=torch.int64).cpu()
    return s.numpy()


@pytest.mark.parametrize("n,p", [(1000, 130), (20000, 130), (50001, 9), (262145, 9), (1048577, 5), (2097153, 5),
                                 (4194303, 3), (4194304, 3), (4194305, 3)])
def test_counts_are_exact(hook, n, p):
    import torch
    g = _codes(n, p, [1 + 2 * ((7 * k) % 31) for k in range(p)])
    freq = torch.full((p,), 0.5, dtype=torch.float64, device="cuda")
    w = torch.zeros((p, p), dtype=torch.float64, device="cuda")
    err = C.c_int(-1)
    assert hook(g.data_ptr(), n, p, g.shape[1], freq.data_ptr(), w.data_ptr(), C.byref(err)) == 0
    assert err.value == 0
    # the square root of 1/2 squared and the quotient are each within an ulp
    got = n + w.cpu().numpy() / 2.0
    want = _counts(g, n)
    assert np.max(np.abs(got - np.rint(got))) <= 1e-8
    assert np.array_equal(np.rint(got).astype(np.int64), want)


@pytest.mark.parametrize("n", [20000, 4194304])
def test_counts_of_mixed_codes_are_exact(hook, n):
    import torch
    p, ldx = 6, (n + 127) // 128 * 128
    gen = torch.Generator(device="cuda").manual_seed(n)
    g = torch.zeros((p, ldx), dtype=torch.int8, device="cuda")
    for k, f in enumerate((0.02, 0.3, 0.5, 0.7, 0.95, 0.999)):
        g[k, :n] = (torch.rand((2, n), device="cuda", generator=gen) < f).sum(dim=0).to(torch.int8)
    freq = torch.full((p,), 0.5, dtype=torch.float64, device="cuda")
    w = torch.zeros((p, p), dtype=torch.float64, device="cuda")
    err = C.c_int(-1)
    assert hook(g.data_ptr(), n, p, ldx, freq.data_ptr(), w.data_ptr(), C.byref(err)) == 0 and err.value == 0
    assert np.array_equal(np.rint(n + w.cpu().numpy() / 2.0).astype(np.int64), _counts(g, n))
