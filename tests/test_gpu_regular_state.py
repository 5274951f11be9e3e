"""sodagpu_get_state and sodagpu_set_state touch blocksize entries of yaadj, also
in the regular sampler, whose own subset size is 8: a caller's array of fewer
entries (six SNPs), with guard entries behind it that must not change."""
import ctypes as C

import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, make_config, synth

pytestmark = pytest.mark.gpu


def test_small_regular_state_stays_in_the_callers_array(gpu_lib):
    n, p = 40, 6
    G, y, _ = synth.make(synth.SynthSpec(n=n, p=p, ncausal=2, h2=0.4, mean=5.0, seed=3))
    cfg = make_config(n, p, JobOptions(method="BayesC", pi=0.5, blocksize=1, numit=50, burnin=0, seed=4))
    assert cfg.blocksize < 8
    buf = np.full(64, 7.0)
    dp = C.POINTER(C.c_double)
    job = SodaJob(cfg)
    job.load_genotypes(G)
    job.load_pheno(y)
    job.build_z()
    job.init_chains()
    job.run(2)
    rc = job._lib.sodagpu_get_state(job._ctx, 0, None, None, None, None, buf.ctypes.data_as(dp), None)
    assert rc == 0
    assert np.all(buf[cfg.blocksize:] == 7.0)
    job.close()
