"""The pi draws on an injected-draw tape whose record is just long enough for
them one after another.  With ten classes, nine of them empty, the ten gamma
variates take 3, 5 (one candidate outside the support), 3, ... = 32 uniforms,
all of the record; read from the place that each would have if every one took
three, the last would be rejected and run past the record's end.  The GPU must
accept the tape and give the oracle's chain."""
import math

import numpy as np
import pytest

from sodabayes_gb300 import JobOptions, SodaJob, _abi, make_config, synth

pytestmark = pytest.mark.gpu

N, P, BS, REPS, NMIX = 60, 24, 8, 3, 10


def _accepts(shape, u):
    """Uniforms that rand_gamma (parallelrng.f90:294-333) takes from u, or None when u ends first."""
    d = shape - 1.0 / 3.0
    c = 1.0 / math.sqrt(9.0 * d)
    k = 0
    while True:
        v = -1.0
        while v <= 0.0:
            if k + 2 > len(u):
                return None
            x = math.sqrt(-2.0 * math.log(u[k])) * math.sin(2.0 * math.pi * u[k + 1])
            v = 1.0 + c * x
            k += 2
        if k + 1 > len(u):
            return None
        w = v * v * v
        k += 1
        if u[k - 1] < 1.0 - 0.0331 * x ** 4 or math.log(u[k - 1]) < 0.5 * x * x + d * (1.0 - w + math.log(w)):
            return k


def _tape(ngroup=1):
    sites = 3 + ngroup + BS + P
    rng = np.random.default_rng(1)
    t = rng.uniform(0.2, 0.8, size=(REPS, sites, _abi.TAPE_W))
    t[:, 3 + ngroup + BS:, 0] = 0.0          # every SNP's class uniform: the first class
    pi = t[:, 3]
    pi[:, 3:5] = 0.01, 0.75                  # the second variate's first candidate lies below the support
    pi[:, 26:31] = 0.5, math.exp(-1.125), 0.25, 0.9999, 0.1
    return t


def test_pi_draws_that_fill_their_record(gpu_lib, oracle_mod):
    tape = _tape()
    for u in tape[:, 3]:
        k, taken = 0, []
        for j in range(NMIX):
            taken.append(_accepts(1.0 + (P if j == 0 else 0), u[k:]))
            k += taken[-1]
        assert taken == [3, 5] + [3] * 8 and k == _abi.TAPE_W
        assert _accepts(1.0, u[27:]) is None
    G, y, _ = synth.make(synth.SynthSpec(n=N, p=P, ncausal=4, h2=0.4, mean=3.0, seed=2))
    cfg = make_config(N, P, JobOptions(method="BayesR", nmix=NMIX, mix=(0.0,) + tuple(1e-4 * 2 ** k for k in range(9)),
                                       numit=20, burnin=0, thin=1, blocksize=BS, seed=3, scale_va=0.02, df_va=4.0,
                                       scale_ve=0.5, df_ve=4.0, precision="fp64"))
    with SodaJob(cfg) as job:
        job.load_genotypes(G)
        job.load_pheno(y)
        job.build_z()
        job.set_tape(tape)
        job.init_chains()
        job.run(REPS - 1)
        got, z, acc = job.state(), job.z(), job.results()
    o = oracle_mod.Oracle(cfg)
    o.load_genotypes(G)
    o.load_pheno(y)
    o.set_z(z[0], z[1])
    o.play_tape(tape.ravel())
    o.init_chains()
    o.run(REPS - 1)
    want, oacc = o.state(), o.results()
    o.close()
    assert np.array_equal(got["cls"], want["cls"]) and np.all(got["cls"] == 1)
    for k in ("mu", "vare", "vara"):
        assert abs(got[k] - want[k]) <= 1e-9 * abs(want[k]), k
    assert np.allclose(acc["pstore"], oacc["pstore"], rtol=1e-9, atol=0.0)
