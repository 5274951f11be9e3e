"""Residual recalibration (compute_residuals, utilities.f90:609-614): r becomes
y - mu - X g whatever it was before, at the edges of its 32 column splits and
of the 256 SNPs that are gathered at a time, with no, one, a few and all
effects non-zero, and for several chains.

Reference: numpy in FP64.  Both sides round every product and sum of at most p
terms and the sums of the splits: 4 (p + 34) eps times the sum of the terms'
magnitudes (Higham, Accuracy and Stability of Numerical Algorithms, section
4.2)."""
import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, make_config, synth

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("precision,chains", [("fp64", 1), ("fp32", 2), ("fp8", 4)])
@pytest.mark.parametrize("n,p,bs", [(70, 20, 10), (257, 1000, 250), (300, 32 * 256 + 33, 911), (1025, 32 * 512, 1024)])
def test_recalibrated_residual(gpu_lib, n, p, bs, precision, chains):
    rng = np.random.default_rng(n)
    codes = np.asfortranarray(rng.binomial(2, rng.uniform(0.1, 0.9, p), size=(n, p)).astype(np.int8))
    y = 20.0 + 3.0 * rng.standard_normal(n)
    cfg = make_config(n, p, JobOptions(method="BayesCpi", numit=50, burnin=0, blocksize=bs, seed=8, scale_va=0.01,
                                       df_va=4.0, scale_ve=1.0, df_ve=4.0, precision=precision, chains=chains,
                                       recal_every=2))
    x = synth.centred(codes)
    with SodaJob(cfg) as job:
        job.load_genotypes(codes)
        job.load_pheno(y)
        job.build_z()
        job.init_chains()
        pi = ((1 - 1e-12, 1e-12), (0.99, 0.01), (1e-12, 1 - 1e-12), (0.5, 0.5))
        for c in range(chains):    # residuals of nothing in particular, and from no effect to all of them
            job.set_state(c, np.zeros(p), np.ones(p, dtype=np.int32), np.full(p, 0.01), rng.standard_normal(n),
                          np.zeros(cfg.blocksize), 0.3, 5.0, 0.001, pi=np.array([pi[(c + (chains == 1)) % 4]]))
        job.run(1)
        before = [job.state(c) for c in range(chains)]
        job.run(1)
        for c in range(chains):
            s = job.state(c)
            want = y - s["mu"] - x @ s["g"]
            tol = 4.0 * (p + 34) * EPS * (np.abs(y) + abs(s["mu"]) + np.abs(x) @ np.abs(s["g"]))
            assert np.all(np.abs(s["yadj"] - want) <= tol)
            b = before[c]
            assert np.max(np.abs(b["yadj"] - (y - b["mu"] - x @ b["g"]))) > 1.0    # it was something else
