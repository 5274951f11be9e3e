"""d = lambda_max(X'X) + 0.001 is as good as FP64 sums make it, although an FP32
run turns the start vector.

Reference: the Rayleigh quotient, in long double, of numpy's eigenvector after
one correction step.  What d may be off by, in units of its own last place: the
bisection returns the upper end of an interval of one unit (0 to 1), and alpha_0
and the sum with 0.001 are each rounded to nearest (up to 1/2 each); the
rounding of the products with X'X is independent between rows and shrinks with
the square root of their number.  Uniform errors of these sizes have a root
mean square of sqrt(1/4 + 3/12) = 0.71; 0.9 leaves room for the sample of forty
subsets and for the products, and 3 bounds each one."""
import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, make_config, synth

pytestmark = pytest.mark.gpu


def _lambda_max(codes):
    n = codes.shape[0]
    c = codes.astype(float)
    f = codes.sum(axis=0, dtype=np.int64).astype(np.longdouble) / (2 * n)
    sd = np.sqrt(2 * f * (1 - f))
    gram = ((c.T @ c).astype(np.longdouble) - n * np.outer(2 * f, 2 * f)) / np.outer(sd, sd)
    w, v = np.linalg.eigh(gram.astype(float))
    x = v[:, -1].astype(np.longdouble)
    for _ in range(2):
        y = gram @ x
        lam = (x @ y) / (x @ x)
        coef = v.T @ (y - lam * x).astype(float)
        coef[:-1] /= w[:-1] - float(lam)
        coef[-1] = 0.0
        x = x - (v @ coef).astype(np.longdouble)
    return lam


def test_lambda_max_is_good_to_its_last_place(gpu_lib):
    err = []
    for bs, nb, n in ((96, 16, 300), (300, 16, 700), (600, 8, 1500)):
        codes, _, _ = synth.make(synth.SynthSpec(n=n, p=bs * nb, ld_block=50, rho=0.6, ncausal=5, h2=0.4, seed=bs))
        with SodaJob(make_config(n, bs * nb, JobOptions(method="BayesC", pi=0.9, blocksize=bs, seed=11))) as job:
            job.load_genotypes(codes)
            assert job.build_z() == 0
            d = job.z()[1]
        for b in range(nb):
            want = _lambda_max(codes[:, b * bs:(b + 1) * bs]) + np.longdouble(np.float32(0.001))
            err.append(float((np.longdouble(d[b]) - want) / np.longdouble(np.spacing(d[b]))))
    err = np.array(err)
    assert np.max(np.abs(err)) <= 3.0
    assert np.sqrt(np.mean(err ** 2)) <= 0.9
