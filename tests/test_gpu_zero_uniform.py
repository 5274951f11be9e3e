"""A class uniform of exactly 0, which an injected-draw tape can hold: the first
class with a probability above 0 is drawn, and the reference gives a class none
when another's log score lies more than 700 above its own (models.f90:232-236,
366-379), although exp of the difference is still a number there.  Scores that
are 704 apart come from a prior proportion of 1e-306; what the data and the
determinant add is a few units.  Both samplers, from classes 1 (SNPs drawn 32
at once in the regular one) and 2 (one by one)."""
import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, _abi, make_config

pytestmark = pytest.mark.gpu

N, P, BS, REPS = 60, 40, 20, 3


@pytest.mark.parametrize("soda", [True, False])
@pytest.mark.parametrize("start", [1, 2])
@pytest.mark.parametrize("method,pi,want", [("BayesB", (1.0, 1e-306), 1), ("BayesC", (1e-306, 1.0), 2),
                                            ("BayesR", (1e-306, 0.5, 0.5), 2)])
def test_class_of_a_zero_uniform(gpu_lib, method, pi, want, start, soda):
    rng = np.random.default_rng(3)
    codes = np.asfortranarray(rng.binomial(2, rng.uniform(0.2, 0.8, P), size=(N, P)).astype(np.int8))
    y = rng.standard_normal(N)
    kw = dict(nmix=3, mix=(0.0, 0.5, 1.0)) if method == "BayesR" else {}
    cfg = make_config(N, P, JobOptions(method=method, pi=0.9, numit=20, burnin=0, blocksize=BS, seed=3, scale_va=0.01,
                                       df_va=4.0, scale_ve=1.0, df_ve=4.0, precision="fp64", soda=soda, **kw))
    tape = rng.uniform(0.2, 0.8, size=(REPS, 3 + cfg.ngroup + cfg.blocksize + P, _abi.TAPE_W))
    tape[:, 3 + cfg.ngroup + cfg.blocksize:, 0] = 0.0
    with SodaJob(cfg) as job:
        job.load_genotypes(codes)
        job.load_pheno(y)
        job.build_z()
        job.set_tape(tape)
        job.init_chains()
        job.set_state(0, np.zeros(P), np.full(P, start), np.full(P, 0.01), y, np.zeros(cfg.blocksize), 0.0, 1.0, 0.01,
                      pi=np.array([pi]))
        job.run(1)
        assert np.all(job.state()["cls"] == want)
