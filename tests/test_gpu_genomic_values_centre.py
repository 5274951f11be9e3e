"""Genomic values where the centring matters (dgv.cuh): SNPs whose counted allele
is common, so that code - 2 f is near 0 for nearly everyone, and effects that
are not finite at SNPs that are monomorphic in the frequencies given, through
the three entry points that centre by frequencies and the one that has its own
table.

Reference: mu + sum x_k e_k in numpy FP64 with x = (code - 2 f) / sd.  Each side
rounds every x_k e_k a few times and adds p terms, so for each individual they
agree to 4 (p + 16) eps times the sum of its |x_k e_k| (Higham, Accuracy and
Stability of Numerical Algorithms, section 4.2), and the fixed-point weights
add 2^-60 of the sum of the |e_k / sd_k|."""
import ctypes as C

import numpy as np
import pytest

import sodabayes_gb300 as sg
from sodabayes_gb300 import JobOptions, SodaJob, make_config

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _bed(codes):
    n, p = codes.shape
    c = np.zeros((p, (n + 3) // 4 * 4), dtype=np.uint8)
    c[:, :n] = np.array([0, 2, 3], dtype=np.uint8)[codes.T]
    c = c.reshape(p, -1, 4)
    return c[..., 0] | c[..., 1] << 2 | c[..., 2] << 4 | c[..., 3] << 6


def _noalloc(lib, codes, freq, eff, mu):
    import torch
    n, p = codes.shape
    d = torch.from_numpy(np.ascontiguousarray(codes.T)).cuda()
    f, e = torch.from_numpy(freq).cuda(), torch.from_numpy(eff).cuda()
    out = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
    rc = lib.sodagpu_compute_dgv_noalloc(n, p, C.c_void_p(d.data_ptr()), n, C.c_void_p(f.data_ptr()), float(mu),
                                         C.c_void_p(e.data_ptr()), C.c_void_p(out.data_ptr()), None)
    assert rc == 0
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _all(lib, codes, freq, eff, mu):
    """The three entry points that centre by allele frequencies."""
    yield sg.predict(codes=codes, freq=freq, mu=mu, effects=eff)
    yield sg.predict(bed=_bed(codes), nind=codes.shape[0], freq=freq, mu=mu, effects=eff)
    yield _noalloc(lib, codes, freq, eff, mu)


def _job(codes):
    n, p = codes.shape
    job = SodaJob(make_config(n, p, JobOptions(method="BayesC", pi=0.9, blocksize=max(2, p // 3), seed=1)))
    job.load_genotypes(codes)
    job.build_z()
    return job


@pytest.mark.parametrize("n,p", [(300, 7), (1500, 41), (20000, 1000)])
def test_a_common_allele_does_not_cost_precision(gpu_lib, n, p):
    rng = np.random.default_rng(n + p)
    codes = np.full((n, p), 2, dtype=np.int8, order="F")
    for j in range(p):      # one to three other calls in n; every third SNP has the other allele common instead
        codes[rng.choice(n, size=1 + j % 3, replace=False), j] = 1
        if j % 3 == 2:
            codes[:, j] = 2 - codes[:, j]
    freq = codes.mean(axis=0) / 2.0
    eff = rng.standard_normal(p)
    sd = np.sqrt(2.0 * freq * (1.0 - freq))
    terms = (codes - 2.0 * freq) / sd * eff
    want = terms.sum(axis=1)
    tol = 4.0 * (p + 16) * EPS * np.abs(terms).sum(axis=1) + 2.0 ** -60 * np.abs(eff / sd).sum()
    for got in _all(gpu_lib, codes, freq, eff, 0.0):
        assert np.all(np.abs(got - want) <= tol)
    with _job(codes) as job:
        assert np.all(np.abs(job.compute_dgv(0.0, eff) - want) <= tol)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("f", [0.0, 1.0])
def test_non_finite_effect_of_a_monomorphic_snp(gpu_lib, value, f):
    """x = 0 there, and 0 times such an effect is not a number: everyone's value is NaN."""
    rng = np.random.default_rng(4)
    codes = np.asfortranarray(rng.binomial(2, 0.4, size=(50, 30)).astype(np.int8))
    codes[:, 11] = int(2 * f)
    freq = codes.mean(axis=0) / 2.0
    eff = rng.standard_normal(30)
    eff[11] = value
    for got in _all(gpu_lib, codes, freq, eff, 1.0):
        assert np.all(np.isnan(got))
    with _job(codes) as job:
        assert np.all(np.isnan(job.compute_dgv(1.0, eff)))
    eff[11] = 1e300     # a finite one adds nothing
    for got in _all(gpu_lib, codes, freq, eff, 1.0):
        assert np.all(np.isfinite(got))


@pytest.mark.parametrize("where", [0, 500, 959, 960, 1009])
@pytest.mark.parametrize("value", [1e290, np.inf])
def test_sub_ranges_of_both_kinds_in_one_split(gpu_lib, where, value):
    """More individuals than the scratch has room for two splits of: one split of a sub-range of 960 SNPs and one of 50,
    of which the one with the large effect is summed in FP64."""
    import torch
    n, p = 1100000, 1010
    gen = torch.Generator(device="cuda").manual_seed(3)
    g = torch.randint(0, 3, (p, n), dtype=torch.int8, device="cuda", generator=gen)
    freq = np.full(p, 0.45)
    eff = np.random.default_rng(6).standard_normal(p)
    eff[where] = value
    f, e = torch.from_numpy(freq).cuda(), torch.from_numpy(eff).cuda()
    out = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
    rc = gpu_lib.sodagpu_compute_dgv_noalloc(n, p, C.c_void_p(g.data_ptr()), n, C.c_void_p(f.data_ptr()), 0.0,
                                             C.c_void_p(e.data_ptr()), C.c_void_p(out.data_ptr()), None)
    assert rc == 0
    torch.cuda.synchronize()
    rows = np.concatenate([np.arange(0, 200), np.arange(4000, 4200), np.arange(n - 300, n)])
    codes = g[:, torch.from_numpy(rows).cuda()].cpu().numpy().T
    got = out.cpu().numpy()[rows]
    terms = (codes - 2.0 * freq) / np.sqrt(2.0 * freq * (1.0 - freq)) * eff
    want = terms.sum(axis=1)
    if np.isinf(value):
        assert np.array_equal(got, want)
    else:
        assert np.all(np.abs(got - want) <= 4.0 * (p + 16) * EPS * np.abs(terms).sum(axis=1))
