"""Single-site draws at the edges of their kernels: fewer and more SNPs than a
round of 32 drawn together, individuals that do not fill a word of four codes
or a warp's lanes, a residual too large for shared memory (more than 25,600
individuals), and a chain that is dense at first and sparse later, so that it
changes kernels.  Against the CPU oracle on the same counter-based draws, with
the bounds of the regular sampler's other tests: identical classes, effects and
residuals within 1e-9 relative after eight iterations."""
import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, make_config, synth

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.max(np.abs(a - b)) / max(1e-300, np.max(np.abs(b)))


@pytest.mark.parametrize("method", ["BayesB", "BayesCpi", "BayesR"])
@pytest.mark.parametrize("n,p", [(130, 31), (127, 33), (1001, 129), (515, 400), (25701, 9)])
def test_single_site_edges_against_oracle(gpu_lib, oracle_mod, n, p, method):
    G, y, _ = synth.make(synth.SynthSpec(n=n, p=p, ncausal=3, h2=0.4, mean=5.0, seed=n + p))
    o4 = method == "BayesR"
    cfg = make_config(n, p, JobOptions(method=method, pi=0.95, numit=50, burnin=0, seed=77, scale_va=0.02, df_va=4.0,
                                       scale_ve=0.5, df_ve=4.0, soda=False, chains=2, nmix=4 if o4 else 2,
                                       mix=(0.0, 1e-3, 1e-2, 1e-1) if o4 else (0.0, 1.0)))
    job, o = SodaJob(cfg), oracle_mod.Oracle(cfg)
    for s in (job, o):
        s.load_genotypes(G)
        s.load_pheno(y)
        s.build_z()
        s.init_chains()
        s.run(8)
    for c in range(2):
        sg, so = job.state(c), o.state(c)
        assert np.array_equal(sg["cls"], so["cls"])
        assert _rel(sg["g"], so["g"]) <= 1e-9 or np.all(so["g"] == 0)
        assert _rel(sg["yadj"], so["yadj"]) <= 1e-9
        assert sg["included"] == so["included"]
    job.close()
