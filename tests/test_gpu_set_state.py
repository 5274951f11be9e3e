"""sodagpu_set_state through the C ABI: sodagpu_get_state gives back what was set,
and what lies behind the caller's yaadj (NaN) reaches no draw, also in the
regular sampler with fewer SNPs than its own subset size of 8."""
import ctypes as C

import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, make_config, synth

pytestmark = pytest.mark.gpu

DP, IP = C.POINTER(C.c_double), C.POINTER(C.c_int32)


def _d(a):
    return a.ctypes.data_as(DP)


@pytest.mark.parametrize("n,p,bs,soda", [(40, 6, 1, False), (40, 7, 7, False), (40, 9, 3, True), (130, 100, 50, True)])
@pytest.mark.parametrize("method", ["BayesA", "BayesC"])
def test_a_state_comes_back(gpu_lib, n, p, bs, soda, method):
    G, y, _ = synth.make(synth.SynthSpec(n=n, p=p, ncausal=2, h2=0.4, mean=5.0, seed=3))
    cfg = make_config(n, p, JobOptions(method=method, pi=0.5, blocksize=bs, numit=50, burnin=0, seed=4, soda=soda))
    rng = np.random.default_rng(n + p)
    g, vs, r = rng.standard_normal(p), rng.uniform(0.5, 1.5, p), rng.standard_normal(n)
    cls = (rng.integers(0, cfg.nmix, p) + 1).astype(np.int32)
    ra = np.concatenate([rng.standard_normal(cfg.blocksize), np.full(64, np.nan)])
    sc = np.array([4.5, 2.0, 0.25, 3.0])
    with SodaJob(cfg) as job:
        job.load_genotypes(G)
        job.load_pheno(y)
        job.build_z()
        job.init_chains()
        assert job._lib.sodagpu_set_state(job._ctx, 0, _d(g), cls.ctypes.data_as(IP), _d(vs), _d(r), _d(ra), _d(sc),
                                          None) == 0
        s = job.state()
        assert np.array_equal(s["g"], g) and np.array_equal(s["cls"], cls) and np.array_equal(s["vara_s"], vs)
        assert np.array_equal(s["yadj"], r)
        # rows without an augmenting matrix, all of them in the regular sampler, are 0
        assert np.array_equal(s["yaadj"], ra[:cfg.blocksize] if soda else np.zeros(cfg.blocksize))
        assert (s["mu"], s["vare"], s["vara"], s["included"]) == (4.5, 2.0, 0.25, 3)
        job.run(2)
        s = job.state()
        for k in ("g", "yadj", "yaadj", "vare"):
            assert np.all(np.isfinite(s[k])), k
