"""The pivots of the Z build's factor, U_jj^2 = M_jj - sum_t U_tj^2, are off by few
roundings.

A pivot is rounded at the size of M_jj when M = d I - X'X is formed, when the
products of earlier panels are taken out (exactly summed), once for each step of
8 rows in its panel of 64 (0 to 7), for each row of its own step (0 to 7), and
twice over in the root; the Gram's entry, smaller than M_jj here, by its
numerator and itself.  Independent roundings of up to half a unit in the last
place of M_jj each, 0.29 rms, give sqrt((2 + 3.5 + 3.5 + 4 + 2) / 12) = 1.12
units; 1.35 leaves room for the sample.  (64 roundings of a panel's rows one by
one would be 1.9.)  Reference: long double."""
import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, make_config, synth

pytestmark = pytest.mark.gpu


def test_pivots_are_off_by_few_roundings(gpu_lib):
    err = []
    for n, bs, nb, rho in ((700, 300, 8, 0.6), (2000, 301, 4, 0.95), (1500, 600, 3, 0.6)):
        codes, _, _ = synth.make(synth.SynthSpec(n=n, p=bs * nb, ld_block=50, rho=rho, ncausal=5, h2=0.4, seed=bs))
        with SodaJob(make_config(n, bs * nb, JobOptions(method="BayesC", pi=0.9, blocksize=bs, seed=11))) as job:
            job.load_genotypes(codes)
            assert job.build_z() == 0
            xa, xxd, _ = job.z()
            f = job.freq().astype(np.longdouble)
        squares = (codes.astype(np.int64) ** 2).sum(axis=0).astype(np.longdouble)
        gram = (squares - n * (2 * f) ** 2) / (2 * f * (1 - f))
        m = np.repeat(xxd, bs).astype(np.longdouble) - gram
        u = xa[:bs].astype(np.longdouble)
        err.append((((u * u).sum(axis=0) - m) / np.spacing(m.astype(float))).astype(float))
    err = np.concatenate(err)
    assert np.sqrt(np.mean(err ** 2)) <= 1.35
    assert np.max(np.abs(err)) <= 7.5
