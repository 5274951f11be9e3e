"""The CUDA-core residual update's list of changed SNPs at the edges of its
passes of 1,024 positions: subsets of 2 to 2,049 SNPs, every effect of which
changes (BayesA).  The residual is kept up by these updates alone (the first
recalibration comes after 1,000 iterations), so a SNP left out of the list or
listed twice parts it from y - mu - X g formed on the host from the chain's own
state, by about 1e-2 of its largest element.  Bounds: four iterations add at
most 4 x 2,052 rounded products to each element; at an effect of a tenth of the
residual each that is 1e-13 of it in FP64 and 5e-5 in FP32, were the roundings
all of one sign."""
import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, make_config, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,chains,bound",
                         [("fp64", 1, 1e-11), ("fp64", 4, 1e-11), ("fp32", 1, 1e-4), ("fp32", 4, 1e-4),
                          ("fp32", 8, 1e-4), ("fp8", 1, 1e-4)])
@pytest.mark.parametrize("s", [2, 1023, 1024, 1025, 2049])
def test_update_list_edges(gpu_lib, s, precision, chains, bound):
    n, p = 131, s + 3
    G, y, _ = synth.make(synth.SynthSpec(n=n, p=p, ncausal=3, h2=0.4, mean=5.0, seed=s))
    X = synth.centred(G)
    opts = JobOptions(method="BayesA", numit=50, burnin=0, seed=9 + s, scale_va=0.02, df_va=4.0, scale_ve=0.5, df_ve=4.0,
                      blocksize=s, precision=precision, chains=chains)
    with SodaJob(make_config(n, p, opts)) as job:
        job.load_genotypes(G)
        job.load_pheno(y)
        job.build_z()
        job.init_chains()
        job.run(4)
        for c in range(chains):
            st = job.state(c)
            assert np.count_nonzero(st["g"]) > 0.9 * p
            r = y - st["mu"] - X @ st["g"]
            assert np.max(np.abs(st["yadj"][:n] - r)) <= bound * np.max(np.abs(r)), c
