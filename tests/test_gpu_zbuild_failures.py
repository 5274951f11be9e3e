"""Subsets of the Z build that fail: a device wait that gives up in the pivoted
fallback is reported, and a subset that is not positive definite leaves the
others of its batch alone.  Both go through the C ABI with one call replaced
(zbuild_hooks.cu).  So does the memory that a build still holds at its end, which
decides how large a subset can be.

The factors of the other subsets do not depend on the failing one: they must be
those of the build in which none fails, bit for bit, and satisfy U'U + X'X =
d I within the factorisation's backward error (Higham, Accuracy and Stability
of Numerical Algorithms, theorem 10.3) and the Gram's scaling."""
import ctypes as C

import numpy as np
import pytest

import sodabayes_gb300 as sg
from sodabayes_gb300 import JobOptions, SodaGpuError, SodaJob, _abi, make_config, synth

import native

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hooks(gpu_lib, tmp_path_factory):
    so = native.shared_object("zbuild_hooks.cu", tmp_path_factory.mktemp("hooks"), ("zbuild.o", "sweep.o", "noalloc.o"))
    lib = _abi.bind(C.CDLL(so), _abi.PROTOTYPES)
    lib.zbuild_hooks.restype = None
    lib.zbuild_hooks.argtypes = [C.c_int, C.c_int, C.c_double]
    plain, sg._lib = sg._lib, lib
    lib.zbuild_free.restype = C.c_uint64
    lib.zbuild_free.argtypes = [C.c_int]
    lib.zbuild_hooks.free = lib.zbuild_free
    yield lib.zbuild_hooks
    sg._lib = plain


def _codes(n, p, seed):
    rng = np.random.default_rng(seed)
    z = rng.standard_normal((n, p)) + 0.5 * rng.standard_normal((n, 1))
    return (z > 0.3).astype(np.int8) + (z > 1.0).astype(np.int8)


def _build(codes, bs, offset=0.0):
    with SodaJob(make_config(*codes.shape, JobOptions(method="BayesC", pi=0.9, blocksize=bs, seed=5))) as job:
        job.load_genotypes(np.asfortranarray(codes))
        job.set_d_offset(offset)
        nsk = job.build_z()
        return (nsk,) + job.z()


def test_a_wait_that_gives_up_in_the_fallback_is_reported(hooks):
    codes = _codes(200, 80, 1)
    hooks(0, -1, 0.0)
    assert _build(codes, 40, offset=-5.0)[0] > 0      # every subset takes the fallback
    hooks(1, -1, 0.0)
    with pytest.raises(SodaGpuError) as e:
        _build(codes, 40, offset=-5.0)
    assert e.value.code == _abi.E_TIMEOUT
    assert _build(codes, 40)[0] == 0                  # no subset takes it
    hooks(0, -1, 0.0)


@pytest.mark.parametrize("bs", [65, 130, 300])
@pytest.mark.parametrize("late", [False, True])
def test_one_subset_that_is_not_positive_definite(hooks, bs, late):
    n = 400
    codes = _codes(n, 3 * bs + bs // 2, bs)
    x = synth.centred(codes)
    gram = x[:, bs:2 * bs].T @ x[:, bs:2 * bs]
    lam = np.linalg.eigvalsh(gram)
    # one eigenvalue of X'X above d (the last pivots fail), or d just above the largest diagonal entry (the first ones)
    shift = 0.001 + (0.3 * (lam[-1] - lam[-2]) if late else lam[-1] - 1.5 * gram.diagonal().max())
    hooks(0, -1, 0.0)
    nsk0, xa0, xxd0, skip0 = _build(codes, bs)
    assert nsk0 == 0 and not skip0.any()
    hooks(0, 1, shift)
    nsk, xa, xxd, skip = _build(codes, bs)
    hooks(0, -1, 0.0)
    inside = np.arange(codes.shape[1]) // bs == 1
    assert nsk == skip.sum() > 0 and not skip[~inside].any()
    assert np.array_equal(xxd[[0, 2, 3]], xxd0[[0, 2, 3]]) and xxd[1] == xxd0[1] - shift
    assert np.array_equal(xa[:, ~inside], xa0[:, ~inside])
    eps = np.finfo(float).eps
    for b, k in ((0, 0), (2, 2 * bs), (3, 3 * bs)):
        xb = x[:, k:min(k + bs, codes.shape[1])]
        m = xb.shape[1]
        u = xa[:m, k:k + m]
        assert np.max(np.abs(u.T @ u + xb.T @ xb - xxd[b] * np.eye(m))) <= eps * (4 * m * xxd[b] + 32 * n)


def test_memory_held_when_the_factors_are_packed(hooks):
    """W and U, 8 bytes an element each, besides the job's own arrays (here a few MB); 64 MB cover those and what the
    runtime keeps."""
    hooks(0, -1, 0.0)
    p = 4000
    codes = _codes(150, p, 2)
    _build(codes, p)                  # the kernels are loaded
    free = hooks.free(1)
    _build(codes, p)
    assert free - hooks.free(0) <= 2 * 8 * p * p + (64 << 20)
