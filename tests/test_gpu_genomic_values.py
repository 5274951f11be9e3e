"""Genomic values at the edges of the table kernel (dgv.cuh): one to five SNPs
left in the last group, chunks of 40 and sub-ranges of 960 SNPs, tiles of
1024, 2048 and 4096 individuals, every alignment of the caller's codes, .bed
records with a partial last byte; and the effects that its fixed-point sums
cannot hold (infinite, NaN, near the ends of the FP64 range), which take FP64
additions.

Reference: mu + X e in numpy FP64.  Tolerance: both sides add p terms and
round each at most a few times, so they agree to 4 (p + 16) eps times the sum
of the largest |x_k e_k| (Higham, Accuracy and Stability of Numerical
Algorithms, section 4.2); non-finite values must be the same."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (3, 4), (31, 5), (1021, 39), (1024, 41), (1025, 81), (2047, 959), (2049, 961), (8193, 171)]


def _inputs(n, p, seed):
    rng = np.random.default_rng(seed)
    codes = rng.binomial(2, rng.uniform(0.0, 1.0, p), size=(n, p)).astype(np.int8)
    freq = np.clip(codes.mean(axis=0) / 2.0 + rng.normal(0.0, 0.02, p), 0.0, 1.0)   # some are monomorphic
    eff = rng.standard_normal(p)
    eff[::7] = 0.0
    return np.asfortranarray(codes), freq, eff


def _values(codes, freq, eff, mu):
    sd = np.sqrt(2.0 * freq * (1.0 - freq))
    ok = (freq >= np.finfo(float).eps) & (1.0 - freq >= np.finfo(float).eps)
    x = np.where(ok, (codes - 2.0 * freq) / np.where(ok, sd, 1.0), 0.0)
    with np.errstate(invalid="ignore", over="ignore"):
        terms = np.where(eff == 0.0, 0.0, x * eff)
        big = np.max(np.abs(terms), axis=0).sum() if np.all(np.isfinite(terms)) else np.inf
        return mu + terms.sum(axis=1), 4.0 * (len(eff) + 16) * np.finfo(float).eps * (big + abs(mu))


def _same(got, want, tol):
    fin = np.isfinite(want)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[~fin & ~np.isnan(want)], want[~fin & ~np.isnan(want)])
    assert np.all(np.abs(got[fin] - want[fin]) <= tol)


def _bed(codes):
    n, p = codes.shape
    c = np.zeros((p, (n + 3) // 4 * 4), dtype=np.uint8)
    c[:, :n] = np.array([0, 2, 3], dtype=np.uint8)[codes.T]
    c = c.reshape(p, -1, 4)
    return c[..., 0] | c[..., 1] << 2 | c[..., 2] << 4 | c[..., 3] << 6


def _noalloc(lib, codes, freq, eff, mu, shift=0, pad=0):
    """The caller's buffer starts `shift` bytes into an allocation and has `pad` more rows than individuals."""
    import torch
    n, p = codes.shape
    ldg = n + pad
    host = np.full(shift + ldg * p, 9, dtype=np.int8)
    host[shift:].reshape(p, ldg)[:, :n] = codes.T
    d = torch.from_numpy(host).cuda()
    f, e = torch.from_numpy(freq).cuda(), torch.from_numpy(eff).cuda()
    out = torch.full((n,), np.nan, dtype=torch.float64, device="cuda")
    rc = lib.sodagpu_compute_dgv_noalloc(n, p, C.c_void_p(d.data_ptr() + shift), ldg, C.c_void_p(f.data_ptr()),
                                         float(mu), C.c_void_p(e.data_ptr()), C.c_void_p(out.data_ptr()), None)
    assert rc == 0
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("n,p", SIZES)
def test_every_entry_point_at_tile_edges(gpu_lib, n, p):
    import sodabayes_gb300 as sg
    codes, freq, eff = _inputs(n, p, 100 * n + p)
    want, tol = _values(codes, freq, eff, 1.5)
    _same(sg.predict(codes=codes, freq=freq, mu=1.5, effects=eff), want, tol)
    _same(sg.predict(bed=_bed(codes), nind=n, freq=freq, mu=1.5, effects=eff), want, tol)
    for shift in range(4):
        _same(_noalloc(gpu_lib, codes, freq, eff, 1.5, shift, pad=shift), want, tol)


@pytest.mark.parametrize("where", [0, 41, 970])
@pytest.mark.parametrize("value", [np.inf, np.nan, 1e290, 1e-300])
def test_effects_outside_the_fixed_point_range(gpu_lib, where, value):
    import sodabayes_gb300 as sg
    codes, _, eff = _inputs(70, 1000, 7)
    freq = np.full(1000, 0.25)
    if value == 1e-300:
        eff = eff * value
    eff[where] = value
    want, tol = _values(codes, freq, eff, 0.0)
    if not np.isfinite(tol):    # one term decides the non-finite values; the others stay within the finite terms' bound
        tol = 0.0
    _same(sg.predict(codes=codes, freq=freq, mu=0.0, effects=eff), want, tol)
    _same(sg.predict(bed=_bed(codes), nind=70, freq=freq, mu=0.0, effects=eff), want, tol)
    _same(_noalloc(gpu_lib, codes, freq, eff, 0.0), want, tol)
