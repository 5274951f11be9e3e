"""d = lambda_max(X'X) + 0.001 of every subset where the Lanczos runs can go
wrong: fewer SNPs than the FP32 start's steps, one SNP short of and past a
cluster's eight slices, more SNPs than individuals (a rank-deficient matrix),
a subset of monomorphic SNPs (the zero matrix), identical columns (one non-zero
eigenvalue, so the recurrence breaks down at once), and two equal eigenvalues.

Reference: numpy's symmetric eigenvalues in FP64, which are good to a few eps
times the largest one; the Lanczos run stops when the eigenvalue no longer
moves by 1e-15 of it."""
import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, make_config, synth

pytestmark = pytest.mark.gpu


def _check(codes, bs):
    n, p = codes.shape
    with SodaJob(make_config(n, p, JobOptions(method="BayesC", pi=0.9, blocksize=bs, seed=11))) as job:
        job.load_genotypes(np.asfortranarray(codes.astype(np.int8)))
        job.build_z()
        _, xxd, _ = job.z()
    x = synth.centred(codes)
    for b, k in enumerate(range(0, p, bs)):
        xb = x[:, k:k + bs]
        lam = max(0.0, np.linalg.eigvalsh(xb.T @ xb)[-1])
        assert abs(xxd[b] - lam - np.float32(0.001)) <= 1e-13 * lam + 1e-15, b


@pytest.mark.parametrize("n,p,bs", [(50, 14, 7), (90, 18, 9), (400, 129, 65), (40, 300, 150), (700, 520, 260)])
def test_lambda_max_at_edge_sizes(gpu_lib, n, p, bs):
    rng = np.random.default_rng(n + p)
    _check(rng.binomial(2, rng.uniform(0.05, 0.95, p), size=(n, p)), bs)


def test_lambda_max_of_degenerate_subsets(gpu_lib):
    rng = np.random.default_rng(3)
    one = rng.binomial(2, 0.4, size=(200, 1))
    two = np.repeat(np.array([[0], [2]]), 100, axis=0)
    cross = np.tile(np.array([[0], [2]]), (100, 1))            # uncorrelated with `two`, the same frequency
    codes = np.concatenate([np.zeros((200, 20), dtype=int),     # the zero matrix
                            np.repeat(one, 20, axis=1),         # rank one
                            np.repeat(two, 10, axis=1), np.repeat(cross, 10, axis=1),   # two equal eigenvalues
                            2 - np.repeat(one, 20, axis=1)], axis=1)
    _check(codes, 20)
