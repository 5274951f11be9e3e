"""Class statistics and accumulators of an iteration (models.f90:321-325,
526-548): the posterior means of class counts, of the sums of squared effects
per (group, class) and of every SNP's effect and classes, against the states
that gave them, with one to 24 cells, few and all effects non-zero, and at the
edges of a CTA's share of the SNPs (256, 16,384 and four times that, and more
SNPs than one pass of the accumulators' grid takes).

Reference: numpy in FP64.  A sum of m squares is off by at most (m + 2) eps of
itself (Higham, Accuracy and Stability of Numerical Algorithms, section 4.2),
on both sides; three kept samples add and divide once each.  Counts are equal."""
import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, make_config

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps
KEPT = 3
R4 = dict(nmix=4, mix=(0.0, 0.0001, 0.001, 0.01))


@pytest.mark.parametrize("method,groups,opts,n,p,bs,precision,chains", [
    ("BayesA", 1, {}, 60, 255, 50, "fp64", 1),
    ("BayesB", 1, {}, 60, 257, 50, "fp64", 2),
    ("BayesCpi", 1, {}, 40, 16385, 64, "fp64", 1),
    ("BayesRc", 6, R4, 60, 300, 100, "fp64", 1),
    ("BayesRc", 3, R4, 40, 4 * 16384 - 1, 128, "fp64", 1),     # the last size of the warps' sums
    ("BayesRc", 4, R4, 40, 4 * 16384, 128, "fp64", 1),         # the first of the threads' own, 16 cells
    ("BayesRc", 5, R4, 40, 4 * 16384, 128, "fp64", 1),         # 20 cells: the warps' sums again
    ("BayesR", 1, R4, 40, 4 * 16384 + 1, 128, "fp32", 1),
    ("BayesA", 1, {}, 40, 5 * 16384 + 33, 128, "fp32", 1),
    ("BayesCpi", 1, {}, 32, 160001, 128, "fp8", 4),
])
@pytest.mark.parametrize("dense", [False, True])
def test_statistics_and_means(gpu_lib, method, groups, opts, n, p, bs, precision, chains, dense):
    rng = np.random.default_rng(p + groups)
    codes = np.asfortranarray(rng.binomial(2, rng.uniform(0.2, 0.8, p), size=(n, p)).astype(np.int8))
    cfg = make_config(n, p, JobOptions(method=method, numit=50, burnin=0, thin=1, blocksize=bs, seed=3, scale_va=0.01,
                                       df_va=4.0, scale_ve=1.0, df_ve=4.0, precision=precision, chains=chains,
                                       ngroup=groups, **opts))
    grp = rng.integers(1, groups + 1, p).astype(np.int32)
    ng, nm = cfg.ngroup, cfg.nmix
    states = []
    with SodaJob(cfg) as job:
        job.load_genotypes(codes)
        job.load_pheno(10.0 + 3.0 * rng.standard_normal(n))
        if groups > 1:
            job.set_groups(grp)
        job.build_z()
        job.init_chains()
        if method not in ("BayesA", "BayesB"):
            first = 1e-9 if dense else 0.99
            pi = np.full((ng, nm), (1.0 - first) / (nm - 1))
            pi[:, 0] = first
            for c in range(chains):
                s = job.state(c)
                job.set_state(c, s["g"], s["cls"], s["vara_s"], s["yadj"], s["yaadj"], s["mu"], 1.0, 0.01, pi=pi)
        for _ in range(KEPT):
            job.run(1)
            states.append([job.state(c) for c in range(chains)])
        for c in range(chains):
            res = job.results(c)
            g = np.array([s[c]["g"] for s in states])
            cls = np.array([s[c]["cls"] for s in states])
            assert np.all(np.abs(res["gstore"] - g.mean(axis=0)) <= 8 * EPS * np.abs(g).sum(axis=0))
            if method == "BayesA":
                sq = np.array([[(g ** 2).sum() / KEPT]])
                assert np.abs(res["varstore"].sum() - sq[0, 0]) <= 2 * (p + 8) * EPS * sq[0, 0]
                continue
            for k in range(nm):
                assert np.array_equal(res["indiststore"][:, k], (cls == k + 1).sum(axis=0) / KEPT)
                for e in range(ng):
                    cell = (cls == k + 1) & (grp == e + 1)[None, :]
                    assert res["snpstore"][e, k] == cell.sum() / KEPT
                    want = (g ** 2)[cell].sum() / KEPT
                    assert np.abs(res["varstore"][e, k] - want) <= 2 * (p + 8) * EPS * want
        if method not in ("BayesA", "BayesB"):
            assert (np.mean(states[0][0]["g"] != 0) > 0.9) == dense
