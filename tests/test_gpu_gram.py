"""The tensor-core Gram of the Z build at the edges of its tiles: subsets below,
at and above 128 SNPs, ragged last subsets, individuals below, at and above a
stage of 128, monomorphic SNPs, a permuted order and codes that are all 2
(the largest products).

d I - U'U is X'X, entry by entry: U and d come from the library, X from numpy
in FP64.  The counts of the Gram are exact, so what remains is rounding: the
factorisation's backward error, N eps d, and the scaling's, a few eps n."""
import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, make_config, synth

pytestmark = pytest.mark.gpu

SIZES = [(17, 7, 3), (127, 130, 65), (128, 256, 128), (129, 387, 129), (300, 513, 257), (1025, 700, 300)]


@pytest.mark.parametrize("n,p,bs", SIZES)
def test_z_factors_give_back_the_gram(gpu_lib, n, p, bs):
    rng = np.random.default_rng(n + p)
    codes = rng.binomial(2, rng.uniform(0.02, 0.98, p), size=(n, p)).astype(np.int8)
    codes[:, 5 % p] = 0
    codes[:, 6 % p] = 2
    codes[: n - 1, 3] = 2
    perm = rng.permutation(p)
    with SodaJob(make_config(n, p, JobOptions(method="BayesC", pi=0.9, blocksize=bs, seed=3))) as job:
        job.load_genotypes(np.asfortranarray(codes))
        nsk = job.build_z(perm.astype(np.int32) + 1)
        xa, xxd, skip = job.z()
    assert nsk == 0 and not skip.any()
    x = synth.centred(codes)[:, perm]
    for b, k in enumerate(range(0, p, bs)):
        u = xa[:, k:k + bs]
        gram = xxd[b] * np.eye(u.shape[1]) - u.T @ u
        want = x[:, k:k + bs].T @ x[:, k:k + bs]
        eps = np.finfo(float).eps
        assert np.max(np.abs(gram - want)) <= eps * (4 * u.shape[1] * xxd[b] + 32 * n)
