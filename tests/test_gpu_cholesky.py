"""The digit Cholesky of the Z build at the edges of its panels (64 rows), tiles
(128 columns), digit groups (128 rows between drains) and subsets of uneven
size in one batch, and a batch in which one subset is not positive definite.

U'U + X'X = d I: the factorisation's backward error is at most N eps d (Higham,
Accuracy and Stability of Numerical Algorithms, theorem 10.3, gives (N + 1) eps
times the squares of the columns, which are d at most), and the Gram's scaling
adds a few eps n."""
import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, make_config, synth

pytestmark = pytest.mark.gpu


def _job(codes, bs, offset=0.0):
    n, p = codes.shape
    job = SodaJob(make_config(n, p, JobOptions(method="BayesC", pi=0.9, blocksize=bs, seed=5)))
    job.load_genotypes(np.asfortranarray(codes.astype(np.int8)))
    job.set_d_offset(offset)
    nsk = job.build_z()
    xa, xxd, skip = job.z()
    job.close()
    return nsk, xa, xxd, skip


@pytest.mark.parametrize("bs", [2, 63, 64, 65, 127, 128, 129, 191, 257, 320, 449])
def test_factor_at_panel_edges(gpu_lib, bs):
    n, p = 350, 2 * bs + max(2, bs // 2)
    rng = np.random.default_rng(bs)
    z = rng.standard_normal((n, p)) + 0.6 * rng.standard_normal((n, 1))      # correlated columns
    codes = (z > 0.4).astype(int) + (z > 1.1)
    nsk, xa, xxd, skip = _job(codes, bs)
    assert nsk == 0 and not skip.any()
    x = synth.centred(codes)
    eps = np.finfo(float).eps
    for b, k in enumerate(range(0, p, bs)):
        xb = x[:, k:k + bs]
        m = xb.shape[1]
        u = xa[:m, k:k + bs]
        assert np.array_equal(u, np.triu(u)) and np.all(np.diag(u) > 0)
        assert np.max(np.abs(u.T @ u + xb.T @ xb - xxd[b] * np.eye(m))) <= eps * (4 * m * xxd[b] + 32 * n)


def test_a_subset_that_is_not_positive_definite_leaves_the_others_alone(gpu_lib):
    """An offset below the gap between d and the largest eigenvalues of one subset only: that one takes the pivoted
    fallback (skipped SNPs), the others' factors are those of the shifted matrix."""
    rng = np.random.default_rng(9)
    n, bs = 400, 130
    codes = rng.binomial(2, 0.4, size=(n, 3 * bs))
    codes[:, bs:2 * bs] = np.repeat(rng.binomial(2, 0.4, size=(n, bs // 10)), 10, axis=1)   # rank 13
    x = synth.centred(codes)
    lam = [np.linalg.eigvalsh(x[:, k:k + bs].T @ x[:, k:k + bs]) for k in range(0, 3 * bs, bs)]
    shift = 0.5 * max(lam[0][-1], lam[2][-1])       # d - shift stays above no eigenvalue of subsets 0 and 2 either
    nsk, xa, xxd, skip = _job(codes, bs, offset=-shift)
    assert nsk == skip.sum() and skip[:bs].any() and skip[bs:2 * bs].any()
    nsk, xa, xxd, skip = _job(codes, bs)
    assert nsk == 0
