"""Performance cases: what users of the engine run, through its public entry
points, on synthetic cohorts over the range of sizes the tests, the benchmark
workloads and the documentation use.

A case is one call (or one short sequence of calls) of a program that keeps
an engine and, except where it uploads itself, a resident genotype matrix:

    fit      slfmm_fit on resident genotypes: the whole LFMM2 fit with every
             per-SNP result written to the caller's page-locked arrays
    host     fit_lfmm2_host: payload in page-locked host memory -> results
    factors  estimate_factors: covariates + randomized SVD
    test     slfmm_test_associations with given factors
    many     fit_lfmm2_many: independent problems from host payloads
    traits   fit_lfmm2_traits: one model per trait on its own samples

Cohorts are admixed populations (Dirichlet proportions, drifted allele
frequencies, missing calls at random) drawn with torch from the seed.
"""
import ctypes
import math

import numpy as np
import torch

import schnellfmm_gb300 as sg

_PRECISION = {"fp8": sg.Precision.SPLIT_FP8, "bf16": sg.Precision.SPLIT_BF16, "fp32": sg.Precision.FP32}


def _case(kind, name=None, **kw):
    c = {"kind": kind, "precision": "fp8", "n": 0, "p": 0, "k": 5, "d": 1, "miss": 0.01, "n_pop": 4,
         "inbreeding": 0.0, "est_rate": 1.0, "nmf_k": 0, "nmf_iter": 0, "omega": False, "count": 0}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a first look at a small data set, one phenotype: the reference's
        # CPU-runnable size, where launches and synchronisations are the cost
        _case("fit", "fit-small", n=200, p=10_000, k=3, n_pop=2, omega=True),
        # a few hundred accessions and an odd SNP count in the split-BF16 mode
        _case("fit", "fit-bf16", precision="bf16", n=997, p=50_003, k=5, d=2, omega=True),
        # the plain FP32 mode, for users who want no operand splitting
        _case("fit", "fit-fp32", precision="fp32", n=2504, p=60_000, k=6, d=2, omega=True),
        # inbred plants (1135 accessions, 1.8 M SNPs), factors from 1 % of the SNPs
        _case("fit", "fit-plant", n=1135, p=1_800_000, k=12, miss=0.02, n_pop=8, inbreeding=0.9, est_rate=0.01),
        # a biobank: 50 traits jointly on 20 000 samples; the largest case
        _case("fit", "fit-biobank", n=20_000, p=1_000_000, k=20, d=50, miss=0.005, n_pop=10),
        # NMF imputation of a cohort with many missing calls
        _case("fit", "fit-nmf", n=3000, p=100_000, k=8, d=4, miss=0.07, n_pop=6, nmf_k=8, nmf_iter=10),
        # a one-shot run from host memory, ragged sample count
        _case("host", "host-cohort", n=12_001, p=250_000, k=10, d=10, miss=0.005, n_pop=6),
        # latent factors of a mid-size cohort, kept for several test runs
        _case("factors", "factors-cohort", n=5003, p=400_000, k=10, d=4, n_pop=6),
        # one phenotype tested on a biobank with factors estimated before
        _case("test", "test-trait", n=20_000, p=500_000, k=20, d=1, miss=0.005, n_pop=10),
        # many phenotypes jointly: a design of more than 128 columns
        _case("test", "test-wide", n=3000, p=100_000, k=30, d=100, n_pop=6),
        # a batch of unrelated data sets of uneven sizes
        _case("many", "many-sets", n=3000, p=200_000, k=16, d=8, count=12),
        # per-trait models on one cohort, each on the samples that have the trait
        _case("traits", "traits-masked", n=10_000, p=200_000, k=10, d=4, miss=0.005, n_pop=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit", "host", "factors", "test", "many", "traits"])
    n = _log(rng, 120, 20_000)
    k = rng.randint(2, 20)
    d = _log(rng, 1, 50)
    # at most the largest listed case's number of calls
    cells = {"fit": 2.0e10, "host": 3.0e9, "factors": 6.0e9, "test": 1.0e10, "many": 6.0e8, "traits": 2.0e9}[kind]
    p = _log(rng, 4_000, max(6_000, min(1_800_000, int(cells / n))))
    c = _case(kind, n=n, p=p, k=k, d=d, miss=round(rng.choice([0.0, 0.002, 0.005, 0.01, 0.03]), 4),
              n_pop=rng.randint(2, 10))
    if kind == "fit":
        form = rng.choice(["plain", "plain", "rate", "nmf", "bf16", "fp32"])
        if form == "rate":
            c.update(est_rate=rng.choice([0.01, 0.05, 0.1]), p=max(c["p"], 20_000))
        elif form == "nmf":
            c.update(nmf_k=rng.randint(2, 12), nmf_iter=rng.randint(3, 10), miss=rng.choice([0.02, 0.07]),
                     n=min(n, 5000), p=min(c["p"], 100_000), d=min(d, 8))
        elif form in ("bf16", "fp32"):
            c.update(precision=form, n=min(n, 6000), p=min(c["p"], 100_000), d=min(d, 8))
    elif kind == "test":
        c.update(d=min(_log(rng, 1, 100), n // 3))
    elif kind == "many":
        c.update(n=max(n, 400) if n <= 3000 else 3000, p=max(8_000, min(c["p"], 200_000)), k=min(k, 16),
                 d=min(d, 8), count=rng.randint(3, 12))
    elif kind == "traits":
        c.update(d=rng.randint(1, 4), n=max(n, 400))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _codes(case, n, p, seed):
    """SNP chunks (row 0, codes C x n) of the cohort: PLINK codes 0 (hom
    ref), 1 (missing), 2 (het), 3 (hom alt) as uint8 on the GPU, and the
    admixture proportions first."""
    rng = np.random.default_rng(seed)
    q = torch.from_numpy(rng.dirichlet(np.full(case["n_pop"], 0.5), size=n).astype(np.float32)).cuda()
    yield q
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 1)
    rows = max(1, min(p, (1 << 26) // n))

    def u(*shape):
        return torch.rand(shape, device="cuda", generator=gen)

    for r0 in range(0, p, rows):
        m = min(rows, p - r0)
        f = 0.02 + 0.48 * u(m, 1)
        drift = (0.05 * f * (1 - f)).sqrt() * torch.randn((m, case["n_pop"]), device="cuda", generator=gen)
        freq = (f + drift).clamp_(1e-3, 1 - 1e-3) @ q.T
        a = u(m, n) < freq
        b = u(m, n) < freq
        if case["inbreeding"] > 0:
            b = torch.where(u(m, n) < case["inbreeding"], a, b)
        g = a.to(torch.uint8) + b.to(torch.uint8)
        codes = g + (g > 0).to(torch.uint8)
        if case["miss"] > 0:
            codes.masked_fill_(u(m, n) < case["miss"], 1)
        yield r0, codes


def _payload(case, n, p, seed):
    """The cohort's SNP-major .bed payload (p x ceil(n / 4) bytes) in
    page-locked host memory, and its admixture proportions."""
    bps = (n + 3) // 4
    host = torch.empty((p, bps), dtype=torch.uint8, pin_memory=True)
    chunks = _codes(case, n, p, seed)
    q = next(chunks)
    for r0, codes in chunks:
        m = codes.shape[0]
        if n % 4:
            codes = torch.nn.functional.pad(codes, (0, 4 * bps - n))
        c4 = codes.view(m, bps, 4)
        packed = c4[..., 0] | (c4[..., 1] << 2) | (c4[..., 2] << 4) | (c4[..., 3] << 6)
        host[r0:r0 + m].copy_(packed, non_blocking=True)
    torch.cuda.synchronize()
    return host.numpy(), q.double().cpu().numpy()


def _covariates(q, d, seed):
    """Traits with a population term and noise."""
    rng = np.random.default_rng(seed)
    pop = q @ rng.normal(size=(q.shape[1], d))
    pop /= pop.std(axis=0) + 1e-12
    return np.ascontiguousarray(0.4 * pop + rng.normal(size=(q.shape[0], d)))


def _config(case, k=None):
    cfg = sg.Lfmm2Config(k=k or case["k"], norm=sg.SnpNorm.EIGENSTRAT)
    if case["nmf_k"]:
        cfg.impute = sg.ImputeStrategy.NMF
        cfg.nmf = sg.NmfConfig(k=case["nmf_k"], n_iter=case["nmf_iter"])
    return cfg


def _results(n, p, d, k, nmf_iter=0):
    """Page-locked result arrays, as a program that calls repeatedly keeps them."""
    out = {"u_hat": (n, k), "beta": (p, d), "tstat": (p, d), "pvalue": (p, d), "r2": (p, 3), "gif_per_trait": (d,)}
    if nmf_iter:
        out["nmf_cv"] = (nmf_iter,)
    return {name: torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy() for name, shape in out.items()}


def _inputs(case, seed):
    """What the fit kinds and exact() both start from: payload, covariates and,
    where the caller brings it, the sketch matrix."""
    packed, q = _payload(case, case["n"], case["p"], seed)
    x = _covariates(q, case["d"], seed + 2)
    omega = np.random.default_rng(seed + 3).normal(size=(case["n"], case["k"] + 10)) if case["omega"] else None
    return packed, q, x, omega


def _given_factors(case, q, seed):
    """Latent factors as an earlier run left them: the admixture axes and noise."""
    n, k = case["n"], case["k"]
    u = np.random.default_rng(seed + 4).normal(size=(n, k)) / math.sqrt(n)
    m = min(k, q.shape[1] - 1)
    u[:, :m] += (q[:, :m] - q[:, :m].mean(axis=0)) / math.sqrt(n)
    return np.ascontiguousarray(u)


def _sets(case):
    """The uneven problems of a batch: the first as large as the case says, the
    others spread over the range below it."""
    for i in range(case["count"]):
        a, b, c = ((i * g) % 1.0 for g in (0.6180339887, 0.7548776662, 0.5698402910))
        n = case["n"] - int(a * (case["n"] - 100))
        p = case["p"] - int(b * (case["p"] - case["p"] // 8))
        yield n, p, case["k"] - int(c * (case["k"] - 2)), case["d"] - int(a * (case["d"] - 1))


def prepare(case, seed):
    kind, n, p, k, d = case["kind"], case["n"], case["p"], case["k"], case["d"]
    eng = sg.Engine(precision=_PRECISION[case["precision"]])
    s = {"kind": kind, "eng": eng}
    if kind == "many":
        s["problems"], s["outs"] = [], []
        for i, (ni, pi, ki, di) in enumerate(_sets(case)):
            packed, q = _payload(case, ni, pi, seed + 101 * i)
            s["problems"].append((packed, ni, _covariates(q, di, seed + 101 * i + 2), _config(case, ki)))
            s["outs"].append(_results(ni, pi, di, ki))
        return s
    packed, q, x, omega = _inputs(case, seed)
    s["cfg"] = _config(case)
    s["omega"] = omega
    if kind == "host":
        s.update(packed=packed, n=n, x=x, out=_results(n, p, d, k))
        return s
    s["geno"] = s["est"] = eng.upload(packed, n)
    s["x"] = x
    if kind == "fit":
        if case["est_rate"] < 1.0:
            s["est"] = eng.upload(packed, n, snps=sg.SubsetSpec.from_rate(case["est_rate"]))
        s["out"] = _results(n, p, d, k, case["nmf_iter"])
    elif kind == "test":
        s["u_hat"] = _given_factors(case, q, seed)
        s["out"] = _results(n, p, d, k)
    elif kind == "traits":
        # up to 30 % of the samples lack a trait
        rng = np.random.default_rng(seed + 6)
        s["masks"] = np.ones((n, d), dtype=np.uint8)
        for t in range(d):
            s["masks"][rng.permutation(n)[:int(0.3 * n * (t + 1) / (d + 1))], t] = 0
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _c_results(out):
    def dp(name):
        return out[name].ctypes.data_as(ctypes.POINTER(ctypes.c_double)) if name in out else None
    return sg._Results(dp("u_hat"), dp("beta"), dp("tstat"), dp("pvalue"), dp("r2"), dp("gif_per_trait"), 0.0,
                       dp("nmf_cv"), 0.0, 0.0, 0.0, 0)


def _ptr(a):
    return None if a is None else a.ctypes.data_as(ctypes.c_void_p)


def _fields(r):
    v = {"u_hat": r.u_hat, "beta": r.beta, "tstat": r.tstat, "pvalue": r.pvalue, "r2": r.r2, "gif": r.gif,
         "gif_per_trait": r.gif_per_trait}
    return v


def run(state):
    s, eng = state, state["eng"]
    kind = s["kind"]
    if kind == "fit":
        res, cfg = _c_results(s["out"]), s["cfg"]._c()
        eng.check(eng.lib.slfmm_fit(eng.h, s["est"].h, s["geno"].h, _ptr(s["x"]), s["x"].shape[1],
                                    ctypes.byref(cfg), _ptr(s["omega"]), ctypes.byref(res)))
        v = dict(s["out"], gif=res.gif)
        if "nmf_cv" in v:
            v.update(nmf_cv_mean=res.nmf_cv_mean, nmf_gwas_cv_mae=res.nmf_gwas_cv_mae,
                     nmf_gwas_cv_mean_mae=res.nmf_gwas_cv_mean_mae, nmf_gwas_cv_count=int(res.nmf_gwas_cv_count))
        return v
    if kind == "test":
        res, cfg = _c_results({m: a for m, a in s["out"].items() if m != "u_hat"}), s["cfg"]._c()
        eng.check(eng.lib.slfmm_test_associations(eng.h, s["geno"].h, _ptr(s["x"]), s["x"].shape[1], _ptr(s["u_hat"]),
                                                  ctypes.byref(cfg), ctypes.byref(res)))
        return dict({m: a for m, a in s["out"].items() if m != "u_hat"}, gif=res.gif)
    if kind == "host":
        return _fields(sg.fit_lfmm2_host(s["packed"], s["n"], s["x"], s["cfg"], engine=eng, out=s["out"]))
    if kind == "factors":
        return sg.estimate_factors(s["geno"], sg.SubsetSpec.all(), s["x"], s["cfg"], engine=eng)
    if kind == "many":
        return [{m: v for m, v in _fields(r).items() if m not in ("gif", "gif_per_trait")}
                for r in sg.fit_lfmm2_many(s["problems"], engine=eng, outs=s["outs"])]
    return [_fields(r) for r in sg.fit_lfmm2_traits(s["geno"], s["x"], s["masks"], s["cfg"], engine=eng)]


def _fit_work(n, p, k, d, factors, test, p_est=None):
    """Bytes and operations of the two halves of a fit: the payload once, the
    results once; 2 q + 2 passes of width k + 10 over the estimation SNPs and
    one of width d + k over every SNP."""
    p_est = p if p_est is None else p_est
    bps = (n + 3) // 4
    byts = max(p if test else 0, p_est if factors else 0) * bps + 8 * n * (d + k)
    flops = 0.0
    if factors:
        flops += 6 * 2.0 * n * p_est * (k + 10)
    if test:
        byts += 8.0 * p * (3 * d + 3)
        flops += 2.0 * n * p * (d + k) + 4.0 * p * d * (d + k)
    return byts, flops


def work(case):
    kind, n, p, k, d = case["kind"], case["n"], case["p"], case["k"], case["d"]
    if kind == "many":
        sets = [_fit_work(*shape, True, True) for shape in _sets(case)]
        return {"bytes": sum(b for b, _ in sets), "flops": sum(f for _, f in sets)}
    if kind == "traits":
        b, f = _fit_work(int(0.85 * n), p, k, 1, True, True)
        return {"bytes": d * b, "flops": d * f}
    b, f = _fit_work(n, p, k, d, kind != "test", kind != "factors",
                     p if case["est_rate"] >= 1.0 else int(math.ceil(p / math.ceil(1.0 / case["est_rate"]))))
    if case["nmf_k"]:
        # two products per update, the initial ones, and the fills at the missing calls
        f += (2 * case["nmf_iter"] + 3) * 2.0 * n * p * case["nmf_k"] * (1 + 2 * case["miss"])
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def _standardised(case, seed):
    """Chunks (row 0, Y rows C x n FP64) of the Eigenstrat-standardised calls,
    missing calls at the mean, from the codes themselves."""
    chunks = _codes(case, case["n"], case["p"], seed)
    next(chunks)
    for r0, codes in chunks:
        for s0 in range(0, codes.shape[0], max(1, (1 << 25) // case["n"])):
            c = codes[s0:s0 + max(1, (1 << 25) // case["n"])]
            seen = c != 1
            g = (c.double() - (c > 0).double()) * seen
            nobs = seen.sum(1, keepdim=True).double()
            mean = g.sum(1, keepdim=True) / nobs.clamp(min=1.0)
            f = mean / 2
            var = 2 * f * (1 - f)
            scale = torch.where(var > 1e-10, var.clamp(min=1e-300).rsqrt(), torch.zeros_like(var))
            yield r0 + s0, (g - mean) * seen * scale


def _orth(a):
    return torch.linalg.qr(a)[0]


def _exact_factors(case, seed, x, omega):
    """The randomized SVD of the covariate-adjusted calls with this sketch."""
    n, p, k, lam = case["n"], case["p"], case["k"], 1e-5
    qd, sv, _ = torch.linalg.svd(x, full_matrices=False)
    dl = torch.sqrt(lam / (lam + sv * sv))
    proj = lambda a, w: a - qd @ ((1 - w)[:, None] * (qd.T @ a))  # noqa: E731
    w = proj(torch.from_numpy(omega).cuda(), dl)
    w = w - w.mean(0)

    def to_snps(a):
        out = torch.empty((p, a.shape[1]), dtype=torch.float64, device="cuda")
        for r0, y in _standardised(case, seed):
            out[r0:r0 + y.shape[0]] = y @ a
        return out

    def to_samples(z):
        out = torch.zeros((n, z.shape[1]), dtype=torch.float64, device="cuda")
        for r0, y in _standardised(case, seed):
            out += y.T @ z[r0:r0 + y.shape[0]]
        return out

    z = _orth(to_snps(w))
    for _ in range(2):
        s = proj(_orth(proj(to_samples(z), dl)), dl)
        z = _orth(to_snps(s - s.mean(0)))
    b = proj(to_samples(z), dl)
    u = torch.linalg.svd(b, full_matrices=False)[0][:, :k]
    return proj(u, 1 / dl)


def _exact_tests(case, seed, x, u):
    """Ordinary least squares t, ridge beta and sequential r2 of every SNP."""
    n, p, d, k = case["n"], case["p"], case["d"], case["k"]
    c = torch.cat([torch.ones((n, 1), dtype=torch.float64, device="cuda"), x, u], 1)
    inv = torch.linalg.inv(c.T @ c)
    ridge = torch.linalg.inv(x.T @ x + 1e-5 * torch.eye(d, dtype=torch.float64, device="cuda"))
    adj = x - u @ torch.linalg.solve(u.T @ u, u.T @ x)
    hat, bop, qx = (inv @ c.T).T, (ridge @ adj.T).T, _orth(x)
    qc = _orth(c)
    df = n - 1 - d - k
    beta, t = (torch.empty((p, d), dtype=torch.float64, device="cuda") for _ in range(2))
    r2 = torch.empty((p, 3), dtype=torch.float64, device="cuda")
    for r0, y in _standardised(case, seed):
        rows = slice(r0, r0 + y.shape[0])
        tss = (y * y).sum(1)
        rss = (tss - ((y @ qc) ** 2).sum(1)).clamp(min=0.0)
        live = tss > 1e-12
        safe = torch.where(live, tss, torch.ones_like(tss))
        ss = ((y @ qx) ** 2).sum(1)
        se = (rss / df).clamp(min=1e-300).sqrt()[:, None] * inv.diagonal()[1:d + 1].sqrt()
        t[rows] = (y @ hat[:, 1:d + 1]) / se * live[:, None]
        beta[rows] = y @ bop
        r2[rows] = torch.stack([ss / safe, (tss - rss - ss).clamp(min=0.0) / safe, rss / safe], 1) * live[:, None]
    med = []
    for j in range(d):  # median of t^2 over bins of 0.001
        v = ((t[:, j] ** 2) / 0.001).floor().clamp(max=99_999).sort().values
        mid = v[(p - 1) // 2] if p % 2 else (v[p // 2 - 1] + v[p // 2]) / 2
        med.append(float((mid + 0.5) * 0.001 / 0.4549))
    raw = torch.tensor(med, dtype=torch.float64, device="cuda")
    gif = raw.clamp(min=1.0)
    pv = torch.special.erfc(t.abs() / gif.sqrt() / math.sqrt(2.0))
    return {"beta": beta, "tstat": t, "pvalue": pv, "r2": r2, "gif_per_trait": gif, "gif": float(raw.mean())}


def exact(case, seed):
    """The tests' results (the factors' columns have no sign of their own, so
    they are compared through the tests)."""
    if case["nmf_k"] or case["n"] * case["p"] > 1.2e10:
        return None
    if not (case["kind"] == "test" or (case["kind"] == "fit" and case["omega"])):
        return None
    chunks = _codes(case, case["n"], case["p"], seed)
    q = next(chunks).double().cpu().numpy()
    chunks.close()
    x = _covariates(q, case["d"], seed + 2)
    xc = torch.from_numpy(x - x.mean(axis=0)).cuda()
    if case["kind"] == "test":
        u = torch.from_numpy(_given_factors(case, q, seed)).cuda()
    else:
        omega = np.random.default_rng(seed + 3).normal(size=(case["n"], case["k"] + 10))
        u = _exact_factors(case, seed, xc, omega)
    v = _exact_tests(case, seed, xc, u)
    if case["kind"] == "fit":
        v["u_hat"] = None
    return v
