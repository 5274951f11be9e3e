"""The work this framework is measured on: passes through its public entry points (SodaJob, SodaBatch, predict and
the C ABI of include/sodagpu.h) at the shapes its users run, from one genomic prediction on device buffers to a whole
job of sixteen chains.

A case's "kind" says which path it takes:

  sweep    SodaJob.run of a few Gibbs iterations from a settled state, then every chain's state
  regular  the same with the regular sampler (-SODAOff)
  batch    SodaBatch.run of several analyses of uneven size, then every job's state
  rhs      SodaJob.subset_rhs of every subset: the conditional right-hand sides alone
  job      a whole short job: create, load, Z build, initialisation, iterations, every chain's state
  z        the set-up alone from host genotypes, in a permuted SNP order: frequencies and Z
  dgv      SodaJob.compute_dgv: genomic values of the training individuals
  predict  predict() from a PLINK .bed payload in host memory
  noalloc  sodagpu_compute_dgv_noalloc on the caller's device buffers

Genotypes are Binomial(2, maf) codes from thresholded AR(1) haplotypes (neighbouring SNPs in LD) or, where the values
do not matter to the path, independent SNPs.  A settled state has 1% of the SNPs in the model (all of them with BayesA), as
chains have after burn-in; it is loaded with set_state, so that it does not depend on an earlier sweep's rounding.
The FP32 and FP8 modes draw in single precision and widen the values on the way out: their floating outputs are
returned as float32, which holds every effect and right-hand side exactly.
"""
import ctypes

import numpy as np
import torch

from sodabayes_gb300 import BAYES_A, BAYES_B, JobOptions, SodaBatch, SodaJob, autotune_batch, library, make_config, predict

MIX4 = (0.0, 1e-4, 1e-3, 1e-2)
PI4 = (0.985, 0.009, 0.005, 0.001)
GROUPS = 3


def listed():
    return [
        # one genomic prediction inside a host's own loop, on its own device buffers: launches and latency
        dict(name="noalloc_small", kind="noalloc", n=1001, p=5003),
        # genomic values of the training set from posterior means, at the end of a job on a 50k chip
        dict(name="dgv_50k_chip", kind="dgv", n=20000, p=50000),
        # prediction mode: a .bed file of selection candidates (an odd number of individuals) and saved effects
        dict(name="predict_bed", kind="predict", n=4999, p=50000),
        # the default job of the command line: FP64, one chain, BayesR, at the size of the reference's examples
        dict(name="fp64_bayesr_example", kind="sweep", method="BayesR", precision="fp64", chains=1, n=2326, p=9346,
             blocksize=935, iters=20),
        # the same data with -SODAOff
        dict(name="regular_bayesr_example", kind="regular", method="BayesR", n=2326, p=9346, iters=1),
        # one FP32 chain at the 5,000 x 50,000 configuration
        dict(name="fp32_bayesr_5k_50k", kind="sweep", method="BayesR", precision="fp32", chains=1, n=5000, p=50000,
             blocksize=1000, iters=3),
        # sixteen FP8 chains at the subset shape of the 20,000 x 500,000 configuration (ten of its 250 subsets)
        dict(name="fp8_bayescpi_20k", kind="sweep", method="BayesCpi", precision="fp8", chains=16, n=20000, p=20000,
             blocksize=2000, iters=5),
        # sixteen FP8 chains at the subset shape of the 50,000 x 1,000,000 configuration, n and p ragged
        dict(name="fp8_bayesrc_50k_ragged", kind="sweep", method="BayesRc", precision="fp8", chains=16, n=49999,
             p=11987, blocksize=1000, iters=4),
        # several breeds or traits at once: analyses of uneven size in one launch per kernel
        dict(name="batch_bayesb_8", kind="batch", method="BayesB", precision="fp8", chains=1, jobs=8, n=5000,
             p=20000, iters=4),
        # conditional right-hand sides of a host that drives the sweep itself: eight chains, odd sizes
        dict(name="rhs_fp8_odd", kind="rhs", method="BayesB", precision="fp8", chains=8, n=3001, p=2331,
             blocksize=777),
        # set-up of a small job in a random SNP order (-rblocks), odd sizes
        dict(name="z_small_odd", kind="z", n=1501, p=3001, blocksize=301),
        # a whole short job at the 20,000-individual subset shape: Z build, packed codes, chains, one iteration
        dict(name="job_fp8_20k", kind="job", method="BayesCpi", precision="fp8", chains=16, n=20000, p=20000,
             blocksize=2000, iters=1),
    ]


def _logint(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "sweep", "sweep", "regular", "batch", "rhs", "job", "z", "dgv", "predict",
                       "noalloc"])
    method = rng.choice(["BayesA", "BayesB", "BayesC", "BayesCpi", "BayesR", "BayesRc"])
    if kind == "sweep":
        precision = rng.choice(["fp64", "fp32", "fp8", "fp8"])
        chains = rng.choice([4, 8, 16, 16]) if precision == "fp8" else rng.choice([1, 1, 2])
        n = _logint(rng, 500, {"fp64": 5000, "fp32": 10000, "fp8": 50000}[precision])
        p = _logint(rng, 2000, 20000)
        return dict(kind=kind, method=method, precision=precision, chains=chains, n=n, p=p,
                    blocksize=_logint(rng, 64, 2000), iters=rng.randint(1, 5))
    if kind == "regular":
        return dict(kind=kind, method=method, n=_logint(rng, 300, 5000), p=_logint(rng, 500, 9346), iters=1)
    if kind == "batch":
        return dict(kind=kind, method=method, precision=rng.choice(["fp64", "fp32", "fp8"]), chains=1,
                    jobs=rng.randint(2, 8), n=_logint(rng, 1000, 5000), p=_logint(rng, 4000, 20000),
                    iters=rng.randint(1, 4))
    if kind == "rhs":
        precision = rng.choice(["fp64", "fp32", "fp8", "fp8"])
        chains = rng.choice([4, 8, 16]) if precision == "fp8" else rng.choice([1, 2])
        bs = _logint(rng, 64, 2000)
        return dict(kind=kind, method=method, precision=precision, chains=chains, n=_logint(rng, 500, 20000),
                    p=bs * rng.randint(1, 3) + rng.randint(0, bs // 2), blocksize=bs)
    if kind == "job":
        precision = rng.choice(["fp64", "fp8"])
        return dict(kind=kind, method=method, precision=precision, chains=16 if precision == "fp8" else 1,
                    n=_logint(rng, 500, 20000), p=_logint(rng, 1000, 20000), blocksize=_logint(rng, 64, 2000), iters=1)
    if kind == "z":
        return dict(kind=kind, n=_logint(rng, 300, 5000), p=_logint(rng, 500, 6000), blocksize=_logint(rng, 30, 500))
    return dict(kind=kind, n=_logint(rng, 500, 20000), p=_logint(rng, 1000, 50000))


# ---- inputs -----------------------------------------------------------------------------------------------------

def _codes(n, p, seed, rho=0.7, block=50):
    """(p, n) int8 codes on the GPU: the column-major n x p matrix of the C ABI.  Blocks of 50 SNPs are AR(1)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    nb = -(-p // block)
    out = torch.zeros((nb, block, n), dtype=torch.int8, device="cuda")
    maf = torch.rand((nb, block), generator=gen, device="cuda") * 0.49 + 0.01
    thr = torch.special.ndtri(maf.double()).float()
    s = float(np.sqrt(1.0 - rho * rho))
    for _haplotype in range(2):
        z = torch.randn((nb, n), generator=gen, device="cuda")
        for t in range(block):
            if t:
                z = rho * z + s * torch.randn((nb, n), generator=gen, device="cuda")
            out[:, t] += z < thr[:, t, None]
    return out.view(nb * block, n)[:p].contiguous()


def _centring(codes):
    """(2 f, sd) of every SNP: the value of a code is (code - 2 f) / sd."""
    f = codes.sum(dim=1, dtype=torch.int64).double() / (2.0 * codes.shape[1])
    ok = (f > 1e-12) & (f < 1.0 - 1e-12)
    sd = torch.where(ok, torch.sqrt(2.0 * f * (1.0 - f)), torch.full_like(f, np.inf))
    return 2.0 * f, sd


def _values(codes, b, rows=4096):
    """X b in 64 bits: codes (p, n), b (p,)."""
    twof, sd = _centring(codes)
    out = torch.zeros(codes.shape[1], dtype=torch.float64, device=codes.device)
    for k in range(0, codes.shape[0], rows):
        c = codes[k:k + rows]
        w = b[k:k + rows] / sd[k:k + rows]
        out += c.double().T @ w - (twof[k:k + rows] * w).sum()
    return out


def _pheno(codes, seed):
    """y = X b + e with half of the variance genetic and variance 1 in all; host array."""
    p = codes.shape[0]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 1)
    pos = torch.randperm(p, generator=gen, device="cuda")[:max(8, p // 250)].sort().values
    v = _values(codes[pos].contiguous(), torch.randn(pos.numel(), generator=gen, device="cuda", dtype=torch.float64))
    e = torch.randn(codes.shape[1], generator=gen, device="cuda", dtype=torch.float64)
    return (v / v.std() * np.sqrt(0.5) + e * np.sqrt(0.5)).cpu().numpy()


def _options(case, seed, p):
    method = case.get("method", "BayesCpi")
    four = method in ("BayesR", "BayesRc")
    included = p if method == "BayesA" else max(1, p // 100)
    vara = 0.5 / included / (float(np.mean(MIX4[1:])) if four else 1.0)
    return JobOptions(method=method, pi=0.99, scale_va=vara, scale_ve=0.5, df_va=4.0, df_ve=4.0, numit=10000,
                      burnin=0, nmix=4 if four else 2, mix=MIX4 if four else (0.0, 1.0), seed=1000 + seed % 1000000,
                      blocksize=case.get("blocksize", 0), ngroup=GROUPS if method == "BayesRc" else 1,
                      precision=case.get("precision", "fp64"), chains=case.get("chains", 1),
                      soda=case["kind"] != "regular")


def _job(case, seed, codes, y, groups):
    opts = _options(case, seed, codes.shape[0])
    job = SodaJob(make_config(codes.shape[1], codes.shape[0], opts))
    job.load_genotypes(device_ptr=codes.data_ptr())
    job.load_pheno(y)
    if opts.method == "BayesRc":
        job.set_groups(groups)
    job.build_z()
    job.init_chains()
    return job


def _settle(job, codes, y, seed):
    """Loads every chain with a settled-looking state: effects of the included SNPs, r = y - mu - X g."""
    cfg, p = job.cfg, job.p
    vara = cfg.scale_va
    for c in range(job.chains):
        rng = np.random.default_rng([seed, c])
        g, cls, vs, pi = np.zeros(p), np.ones(p, dtype=np.int32), np.zeros(p), None
        if cfg.method == BAYES_A:
            nz = np.arange(p)
        else:
            nz = np.sort(rng.choice(p, size=max(1, p // 100), replace=False))
            cls[nz] = rng.integers(2, cfg.nmix + 1, size=nz.size)
        if cfg.method in (BAYES_A, BAYES_B):
            vs[:] = vara
            g[nz] = rng.standard_normal(nz.size) * np.sqrt(vara)
        else:
            g[nz] = rng.standard_normal(nz.size) * np.sqrt(np.array(cfg.mix[:cfg.nmix])[cls[nz] - 1] * vara)
            pi = np.tile(np.array(PI4 if cfg.nmix == 4 else (0.99, 0.01)), (cfg.ngroup, 1))
        at = torch.from_numpy(nz).cuda()
        mu = float(y.mean())
        r = y - mu - _values(codes[at].contiguous(), torch.from_numpy(g[nz]).cuda()).cpu().numpy()
        ra = rng.standard_normal(cfg.blocksize) * np.sqrt(0.5)
        job.set_state(c, g, cls, vs, r, ra, mu, 0.5, vara, nz.size, pi)


def _groups(p, seed):
    return np.random.default_rng([seed, 7]).integers(1, GROUPS + 1, size=p).astype(np.int32)


def _batch_sizes(case, seed):
    """Sizes of the jobs of a batch: the case's are the largest, the others spread down to a tenth."""
    rng = np.random.default_rng(case["n"] + case["jobs"])
    n = [max(200, int(case["n"] * 10.0 ** -u)) for u in [0.0] + list(rng.uniform(0.0, 1.0, case["jobs"] - 1))]
    p = [max(400, int(case["p"] * 10.0 ** -u)) for u in [0.0] + list(rng.uniform(0.0, 1.0, case["jobs"] - 1))]
    return n, p


def _prediction_inputs(case, seed):
    """Codes on the GPU, allele frequencies of the training set and effects, 2% of them zero."""
    n, p = case["n"], case["p"]
    codes = _codes(n, p, seed)
    rng = np.random.default_rng([seed, 3])
    twof, _ = _centring(codes)
    freq = np.clip(twof.cpu().numpy() / 2.0 + rng.normal(0.0, 0.01, p), 0.002, 0.998)
    eff = rng.standard_normal(p) / np.sqrt(p)
    eff[rng.random(p) < 0.02] = 0.0
    return codes, freq, eff, float(rng.normal())


def _bed(codes):
    """PLINK payload of (p, n) codes: two bits an individual, 0/1/2 stored as 00/10/11."""
    p, n = codes.shape
    c = torch.zeros((p, -(-n // 4) * 4), dtype=torch.uint8, device=codes.device)
    c[:, :n] = codes.to(torch.uint8) + (codes > 0).to(torch.uint8)
    c = c.view(p, -1, 4)
    return (c[..., 0] | c[..., 1] << 2 | c[..., 2] << 4 | c[..., 3] << 6).cpu().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("noalloc", "predict"):
        codes, freq, eff, mu = _prediction_inputs(case, seed)
        if kind == "predict":
            return dict(case=case, bed=_bed(codes), freq=freq, eff=eff, mu=mu)
        return dict(case=case, codes=codes, freq=torch.from_numpy(freq).cuda(), eff=torch.from_numpy(eff).cuda(), mu=mu,
                    pred=torch.empty(case["n"], dtype=torch.float64, device="cuda"), lib=library())
    if kind == "batch":
        ns, ps = _batch_sizes(case, seed)
        bs, _, _ = autotune_batch(ns, ps, 2000, 2000)
        jobs = []
        for j, (n, p, b) in enumerate(zip(ns, ps, bs)):
            codes = _codes(n, p, seed + 100 * j)
            y = _pheno(codes, seed + 100 * j)
            jobs.append(_job(dict(case, blocksize=max(2, int(b))), seed + j, codes, y, _groups(p, seed + j)))
            _settle(jobs[-1], codes, y, seed + 100 * j)
        return dict(case=case, jobs=jobs, batch=SodaBatch(jobs))
    codes = _codes(case["n"], case["p"], seed)
    torch.cuda.synchronize()   # jobs read the codes on streams of their own
    if kind == "z":
        rng = np.random.default_rng([seed, 5])
        return dict(case=case, cfg=make_config(case["n"], case["p"], _options(case, seed, case["p"])),
                    codes=codes.cpu().numpy().T, perm=rng.permutation(case["p"]).astype(np.int32) + 1)
    y = _pheno(codes, seed)
    groups = _groups(case["p"], seed)
    if kind == "job":
        return dict(case=case, codes=codes, y=y, groups=groups, seed=seed)
    if kind == "dgv":
        # genomic values need the genotypes in the context, whatever the subset size
        job = _job(dict(case, method="BayesCpi", blocksize=min(250, case["p"] // 2)), seed, codes, y, groups)
        rng = np.random.default_rng([seed, 3])
        eff = rng.standard_normal(case["p"]) / np.sqrt(case["p"])
        return dict(case=case, job=job, eff=eff, mu=float(rng.normal()))
    job = _job(case, seed, codes, y, groups)
    _settle(job, codes, y, seed)
    return dict(case=case, job=job)


# ---- one pass ---------------------------------------------------------------------------------------------------

def _state(job):
    """Every chain's state, in the precision of the mode."""
    one = np.float64 if job.cfg.precision == 0 else np.float32
    out = []
    for c in range(job.chains):
        s = job.state(c)
        out.append(dict(g=s["g"].astype(one, copy=False), cls=s["cls"], yadj=s["yadj"].astype(one, copy=False),
                        scalars=np.array([s["mu"], s["vare"], s["vara"]], dtype=one), included=s["included"]))
        if job.cfg.sampler == 0:   # the regular sampler has no augmented data
            out[-1]["yaadj"] = s["yaadj"].astype(one, copy=False)
        if job.cfg.method in (BAYES_A, BAYES_B):
            out[-1]["vara_s"] = s["vara_s"].astype(one, copy=False)
    return _whole(out)


def _whole(states):
    """The states of all chains of a job as one array for each quantity."""
    return {k: np.stack([s[k] for s in states]) for k in states[0]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "noalloc":
        n, p = case["n"], case["p"]
        rc = state["lib"].sodagpu_compute_dgv_noalloc(
            n, p, ctypes.c_void_p(state["codes"].data_ptr()), n, ctypes.c_void_p(state["freq"].data_ptr()), state["mu"],
            ctypes.c_void_p(state["eff"].data_ptr()), ctypes.c_void_p(state["pred"].data_ptr()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError("sodagpu_compute_dgv_noalloc: %d" % rc)
        return state["pred"]
    if kind == "predict":
        return predict(bed=state["bed"], nind=case["n"], freq=state["freq"], mu=state["mu"], effects=state["eff"])
    if kind == "dgv":
        return state["job"].compute_dgv(state["mu"], state["eff"])
    if kind == "rhs":
        job = state["job"]
        one = np.float64 if job.cfg.precision == 0 else np.float32
        return [job.subset_rhs(b).astype(one, copy=False) for b in range(job.cfg.nblocks)]
    if kind == "z":
        with SodaJob(state["cfg"]) as job:
            job.load_genotypes(state["codes"])
            job.build_z(state["perm"])
            xa, xxd, skip = job.z()
            return dict(freq=job.freq(), xa=xa, xxd=xxd, skip=skip)
    if kind == "batch":
        state["batch"].run(case["iters"])
        return [_state(job) for job in state["jobs"]]
    if kind == "job":
        with _job(case, state["seed"], state["codes"], state["y"], state["groups"]) as job:
            job.run(case["iters"])
            return dict(freq=job.freq(), chains=_state(job))
    state["job"].run(case["iters"])
    return _state(state["job"])


# ---- what a pass cannot do without ------------------------------------------------------------------------------

def work(case):
    kind, n, p = case["kind"], case["n"], case["p"]
    if kind in ("noalloc", "dgv"):
        return dict(bytes=n * p + 16.0 * p + 8.0 * n, flops=2.0 * n * p)
    if kind == "predict":
        return dict(bytes=n * p / 4.0 + 16.0 * p + 8.0 * n, flops=2.0 * n * p)
    if kind == "batch":
        parts = [_sweep_work(case, a, b, min(2000, max(2, b // 20))) for a, b in zip(*_batch_sizes(case, 0))]
        return dict(bytes=sum(w["bytes"] for w in parts), flops=sum(w["flops"] for w in parts))
    if kind in ("regular", "sweep"):
        return _sweep_work(case, n, p, case.get("blocksize", 0))
    bs = min(case["blocksize"], p)
    if kind == "rhs":
        w = _sweep_work(dict(case, iters=1), n, p, bs)
        return dict(bytes=w["bytes"] / 2.0, flops=w["flops"] / 2.0)
    # set-up: the codes once and the factor once; Gram (half of it) and Cholesky of every subset
    gram, chol = 1.0 * n * p * bs, p * bs * bs / 3.0
    set_up = dict(bytes=n * p + 8.0 * p * bs / 2.0, flops=gram + chol)
    if kind == "z":
        return set_up
    w = _sweep_work(case, n, p, bs)
    return dict(bytes=set_up["bytes"] + w["bytes"], flops=set_up["flops"] + w["flops"])


def _sweep_work(case, n, p, bs):
    """Iterations of every chain: two bits a genotype, the factor's triangle and the chains' state, each read once an
    iteration; x'r and r += x d of every SNP and chain."""
    chains, iters = case.get("chains", 1), case["iters"]
    wide = 8.0 if case.get("precision", "fp64") == "fp64" else 4.0
    state = chains * (p * 20.0 + n * 16.0)
    return dict(bytes=iters * (n * p / 4.0 + wide * p * bs / 2.0 + 2.0 * state),
                flops=iters * 4.0 * chains * p * (n + bs / 2.0))


# ---- the same in 64 bits ----------------------------------------------------------------------------------------

def exact(case, seed):
    """Genomic values, frequencies, Z and right-hand sides have a value that plain arithmetic gives.  The state after
    a sweep is a draw from the sampler's own random streams: it has none."""
    kind = case["kind"]
    if kind in ("noalloc", "predict"):
        codes, freq, eff, mu = _prediction_inputs(case, seed)
        f = torch.from_numpy(freq).cuda()
        return mu + _with(codes, 2.0 * f, torch.sqrt(2.0 * f * (1.0 - f)), torch.from_numpy(eff).cuda())
    if kind == "dgv":
        codes = _codes(case["n"], case["p"], seed)
        rng = np.random.default_rng([seed, 3])
        eff = rng.standard_normal(case["p"]) / np.sqrt(case["p"])
        return (float(rng.normal()) + _values(codes, torch.from_numpy(eff).cuda())).cpu().numpy()
    if kind == "z":
        codes = _codes(case["n"], case["p"], seed)
        perm = np.random.default_rng([seed, 5]).permutation(case["p"])
        bs, p = case["blocksize"], case["p"]
        xa, xxd = np.zeros((bs, p), order="F"), []
        for k in range(0, p, bs):
            u, d = _factor(codes[torch.from_numpy(perm[k:k + bs]).cuda()])
            xa[:u.shape[0], k:k + u.shape[1]] = u.cpu().numpy()
            xxd.append(d)
        return dict(freq=(_centring(codes)[0] / 2.0).cpu().numpy(), xa=xa, xxd=np.array(xxd),
                    skip=np.zeros(p, dtype=np.int32))
    if kind == "rhs":
        # the state that _settle loads, its effects and residuals taken from the same streams
        codes = _codes(case["n"], case["p"], seed)
        state = _Recorder(case, seed, codes)
        _settle(state, codes, _pheno(codes, seed), seed)
        bs, out = case["blocksize"], []
        for k in range(0, case["p"], bs):
            u, _ = _factor(codes[k:k + bs])
            x = _centred(codes[k:k + bs])
            out.append(np.stack([(x @ r + u.T @ ra[:u.shape[0]]).cpu().numpy() for r, ra in state.chains_loaded]))
        return out
    if kind == "job":
        codes = _codes(case["n"], case["p"], seed)
        return dict(freq=(_centring(codes)[0] / 2.0).cpu().numpy(), chains=None)
    return None


class _Recorder:
    """Stands in for a job in _settle: keeps the residuals that it is given."""

    def __init__(self, case, seed, codes):
        self.cfg = make_config(codes.shape[1], codes.shape[0], _options(case, seed, codes.shape[0]))
        self.p, self.chains, self.chains_loaded = codes.shape[0], case["chains"], []

    def set_state(self, c, g, cls, vs, r, ra, *rest):
        self.chains_loaded.append((torch.from_numpy(r).cuda(), torch.from_numpy(ra).cuda()))


def _with(codes, twof, sd, b, rows=4096):
    out = torch.zeros(codes.shape[1], dtype=torch.float64, device=codes.device)
    for k in range(0, codes.shape[0], rows):
        w = b[k:k + rows] / sd[k:k + rows]
        out += codes[k:k + rows].double().T @ w - (twof[k:k + rows] * w).sum()
    return out


def _centred(codes):
    twof, sd = _centring(codes)
    return (codes.double() - twof[:, None]) / sd[:, None]


def _factor(codes):
    """Upper factor of d I - X'X of one subset's codes, and d = its largest eigenvalue + 0.001 in single precision."""
    x = _centred(codes)
    a = x @ x.T
    d = float(torch.linalg.eigvalsh(a)[-1]) + float(np.float32(0.001))
    m = torch.eye(a.shape[0], dtype=a.dtype, device=a.device) * d - a
    return torch.linalg.cholesky(m).T, d
