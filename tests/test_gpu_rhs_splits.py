"""The CUDA-core rhs at its largest numbers of K splits (18 for one tile of SNPs
with 9,001 individuals, 24 for 12,288 FP32 individuals).  FP64 against the CPU
oracle with the sweep's bounds; FP32 against FP64 on the same state.  A lane
adds at most 32 FP32 products of genotypes and the lanes' sums go through five
exchanges; each product and the two stored factors are rounded once: 40
roundings of 6e-8 against the sum of the absolute products, whose augmenting
part is at most sqrt(d) |ra| (U'U is at most d), and of d |g|."""
import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, make_config, synth

pytestmark = pytest.mark.gpu


def _cfg(n, p, s, precision, chains):
    return make_config(n, p, JobOptions(method="BayesCpi", pi=0.9, numit=50, burnin=0, seed=31, scale_va=0.02, df_va=4.0,
                                        scale_ve=0.5, df_ve=4.0, blocksize=s, precision=precision, chains=chains))


def test_splits_fp64_against_oracle(gpu_lib, oracle_mod):
    n, p, s = 9001, 41, 20
    G, y, _ = synth.make(synth.SynthSpec(n=n, p=p, ncausal=3, h2=0.4, mean=5.0, seed=1))
    cfg = _cfg(n, p, s, "fp64", 1)
    job, o = SodaJob(cfg), oracle_mod.Oracle(cfg)
    for x in (job, o):
        x.load_genotypes(G)
        x.load_pheno(y)
        x.build_z()
        x.init_chains()
        x.run(3)
    sg, so = job.state(0), o.state(0)
    assert np.array_equal(sg["cls"], so["cls"])
    for k in ("g", "yadj"):
        assert np.max(np.abs(sg[k] - so[k])) <= 1e-9 * np.max(np.abs(so[k])), k
    job.close()


@pytest.mark.parametrize("n,s,chains", [(9001, 20, 1), (9001, 65, 2), (12288, 64, 1), (12289, 64, 1)])
def test_splits_fp32_against_fp64(gpu_lib, n, s, chains):
    p = 2 * s + 1
    G, y, _ = synth.make(synth.SynthSpec(n=n, p=p, ncausal=3, h2=0.4, mean=5.0, seed=n))
    X = synth.centred(G)
    out, st, d = {}, None, None
    for precision in ("fp64", "fp32"):
        with SodaJob(_cfg(n, p, s, precision, chains)) as job:
            job.load_genotypes(G)
            job.load_pheno(y)
            job.build_z()
            job.init_chains()
            if st is None:
                job.run(2)
                st = [job.state(c) for c in range(chains)]
                d = np.max(job.z()[1])
            for c in range(chains):
                v = st[c]
                job.set_state(c, v["g"], v["cls"], v["vara_s"], v["yadj"], v["yaadj"], v["mu"], v["vare"], v["vara"],
                              v["included"])
            job.set_iteration(3)
            out[precision] = job.subset_rhs(0)
    for c in range(chains):
        size = np.abs(X[:, :s]).T @ np.abs(st[c]["yadj"][:n])
        size = size + np.sqrt(d) * np.linalg.norm(st[c]["yaadj"]) + d * np.abs(st[c]["g"][:s])
        err = np.abs(out["fp32"][c] - out["fp64"][c])
        assert np.all(err <= 40 * 2.0 ** -24 * size), (c, np.max(err / size))
