"""The work that users of the framework have it do, as cases of a size each.

A case names a path (`path`), its sizes and its options:

  lmm_scan  trans / gw LMM scan with genotypes, eigenbasis and phenotypes resident:
            spectral rotation of every SNP, REML per gene, scan, FP64 refinement
  lmm_job   the whole LMM job from host buffers: .bed bytes and phenotypes in, decode,
            GRM, eigenbasis, rotation, REML, scan, results out
  lm_scan   trans / gw LM scan with genotypes and phenotypes resident, from .bed calls
            or from a VCF's FP32 dosages
  cis       one call of a cis scan (LM or LMM), phenotypes and covariates passed with it
  perm      gene-level permutations of a cis scan: permuted columns drawn on the device,
            then every column's own null fit and banded scan
  grm       `--make-grm`: .bed bytes in, GRM and its marker counts out
  glm       gw NB-GLM score scan of count phenotypes
  fission   `--pheno-norm int` and PEER factors of a phenotype table

Sizes are those of the benchmark configurations (`bench.py`, `eqtl_b200/config_bench.py`,
`eqtl_b200/perm_bench.py`) and generic ones below them. Inputs are drawn from the seed with
the distributions of `eqtl_b200/synth.py`: HWE or family genotypes at MAF ~ U(0.01, 0.5)
with random allele orientation and 1% missing calls, polygenic phenotypes with
h2 ~ U(0, 0.8), planted cis effects, N(0, 1) covariates that leak into Y,
negative-binomial counts.
"""
import math

import numpy as np
import torch

from eqtl_b200 import capi

PTHR = 1e-5
CHROM_LEN = 20_000_000
WINDOW = 1_000_000
DEV = "cuda"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the headline benchmark: trans/gw LMM over a genome-wide panel
        {"name": "lmm_gw_full", "path": "lmm_scan", "n": 2000, "m": 500_000, "genes": 10_000, "p": 1, "scope": "gw"},
        # a cohort-sized trans LMM scan: cis windows left out, one covariate, ragged sizes
        {"name": "lmm_trans_mid", "path": "lmm_scan", "n": 1201, "m": 60_011, "genes": 1_503, "p": 2, "scope": "trans"},
        # a first run of the program on a cohort with five covariates, from files in host memory
        {"name": "lmm_job", "path": "lmm_job", "n": 1000, "m": 100_000, "genes": 2_000, "p": 6},
        # the largest LM scan: 2e10 tests, ten covariates
        {"name": "lm_gw_full", "path": "lm_scan", "n": 1000, "m": 1_000_000, "genes": 20_000, "p": 11, "scope": "gw",
         "dosage": False},
        # imputed dosages from a VCF, trans scope, with stage-2 permutation candidates
        {"name": "lm_trans_dosage", "path": "lm_scan", "n": 670, "m": 60_000, "genes": 3_001, "p": 4, "scope": "trans",
         "dosage": True},
        # the small cis run of the test panel's size: latency of one call
        {"name": "cis_lm_small", "path": "cis", "model": "lm", "n": 200, "m": 20_000, "genes": 1_000, "p": 4},
        # cis LMM with PEER-like covariates, the observed scan
        {"name": "cis_lmm", "path": "cis", "model": "lmm", "n": 1000, "m": 45_000, "genes": 500, "p": 16},
        # one device batch of cis LMM permutations (each column has its own REML fit)
        {"name": "perm_cis_lmm", "path": "perm", "model": "lmm", "n": 1000, "m": 45_000, "genes": 16, "perms": 500,
         "p": 16},
        # one device batch of cis LM permutations
        {"name": "perm_cis_lm", "path": "perm", "model": "lm", "n": 1000, "m": 45_000, "genes": 32, "perms": 1000,
         "p": 16},
        # a relatedness matrix for a subset of a file's samples
        {"name": "grm_make", "path": "grm", "n": 1999, "n_file": 2100, "m": 200_000},
        # count phenotypes against every SNP
        {"name": "glm_gw", "path": "glm", "n": 1000, "m": 100_000, "genes": 2_000, "p": 3},
        # normalisation and hidden factors of a phenotype table
        {"name": "fission", "path": "fission", "n": 500, "genes": 20_000, "factors": 15},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["lmm_scan", "lmm_job", "lm_scan", "cis", "perm", "grm", "glm", "fission"])
    n = _log(rng, 120, 2000)
    if path == "lmm_scan":
        return {"path": path, "n": n, "m": _log(rng, 5_000, 300_000), "genes": _log(rng, 60, 6_000),
                "p": rng.randint(1, 8), "scope": rng.choice(["gw", "trans"])}
    if path == "lmm_job":
        return {"path": path, "n": n, "m": _log(rng, 5_000, 200_000), "genes": _log(rng, 60, 4_000),
                "p": rng.randint(1, 8)}
    if path == "lm_scan":
        dosage = rng.random() < 0.4
        return {"path": path, "n": min(n, 1000), "m": _log(rng, 5_000, 100_000 if dosage else 500_000),
                "genes": _log(rng, 60, 12_000), "p": rng.randint(1, 16), "scope": rng.choice(["gw", "trans"]),
                "dosage": dosage}
    if path == "cis":
        return {"path": path, "model": rng.choice(["lm", "lmm"]), "n": min(n, 1200), "m": _log(rng, 2_000, 60_000),
                "genes": _log(rng, 20, 3_000), "p": rng.randint(1, 20)}
    if path == "perm":
        genes = _log(rng, 2, 32)
        return {"path": path, "model": rng.choice(["lm", "lmm"]), "n": min(n, 1000), "m": _log(rng, 5_000, 45_000),
                "genes": genes, "perms": _log(rng, 100, 8000 // genes), "p": rng.randint(1, 16)}
    if path == "grm":
        return {"path": path, "n": n, "n_file": n + rng.choice([0, 1, 37, 150]), "m": _log(rng, 2_000, 250_000)}
    if path == "glm":
        return {"path": path, "n": min(n, 1000), "m": _log(rng, 5_000, 100_000), "genes": _log(rng, 30, 2_000),
                "p": rng.randint(1, 6)}
    return {"path": path, "n": min(n, 800), "genes": _log(rng, 300, 20_000), "factors": rng.randint(2, 25)}


# ------------------------------------------------------------------ the inputs
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _codes(gen, n, m, family):
    """int8 A1 counts [m, n] on the GPU, -1 = missing; `family` families of ten siblings lead the samples."""
    out = torch.empty(m, n, dtype=torch.int8, device=DEV)
    step = max(1, 60_000_000 // n)
    for s in range(0, m, step):
        k = min(step, m - s)
        af = 0.01 + 0.49 * torch.rand(k, 1, device=DEV, generator=gen)
        af = torch.where(torch.rand(k, 1, device=DEV, generator=gen) < 0.5, 1 - af, af)
        c = (torch.rand(k, n, device=DEV, generator=gen) < af).to(torch.int8)
        c += torch.rand(k, n, device=DEV, generator=gen) < af
        if family:
            hap = (torch.rand(k, family, 2, 2, device=DEV, generator=gen) < af[:, :, None, None]).to(torch.int8)
            pick = torch.rand(k, family, 10, 2, device=DEV, generator=gen) < 0.5
            sib = torch.where(pick, hap[:, :, None, :, 1], hap[:, :, None, :, 0]).sum(-1)
            c[:, : 10 * family] = sib.reshape(k, 10 * family).to(torch.int8)
        c[torch.rand(k, n, device=DEV, generator=gen) < 0.01] = -1
        out[s:s + k] = c
    return out


def _bed(codes):
    """Packed .bed rows [m, ceil(n / 4)] on the host."""
    m, n = codes.shape
    rows = np.empty((m, (n + 3) // 4), np.uint8)
    lut = torch.tensor([3, 2, 0, 1], dtype=torch.uint8, device=DEV)  # 0, 1, 2 A1 alleles, missing (-1)
    shift = torch.tensor([1, 4, 16, 64], dtype=torch.uint8, device=DEV)
    step = max(1, 100_000_000 // n)
    for s in range(0, m, step):
        c = codes[s:s + step]
        two = torch.zeros(c.shape[0], rows.shape[1] * 4, dtype=torch.uint8, device=DEV)
        two[:, :n] = lut[(c & 3).to(torch.int32)]
        rows[s:s + step] = (two.reshape(c.shape[0], -1, 4) * shift).sum(-1).to(torch.uint8).cpu().numpy()
    return rows


def _dosage(codes, gen):
    """FP32 ALT dosages of imputed calls (the call plus posterior spread, three decimals), NaN = missing."""
    d = codes.to(torch.float32)
    d = d + 0.15 * torch.randn(d.shape, device=DEV, generator=gen) * (torch.rand(d.shape, device=DEV, generator=gen) < 0.3)
    d = torch.round(d.clamp_(0, 2) * 1000) / 1000
    d[codes < 0] = float("nan")
    return d


def _imputed(d):
    """FP64 dosages with each row's missing calls at the mean of its others; [k, n] with NaN or -1 missing."""
    d = d.to(torch.float64)
    miss = torch.isnan(d) | (d < 0)
    d = torch.where(miss, torch.zeros_like(d), d)
    mu = d.sum(1, keepdim=True) / (~miss).sum(1, keepdim=True).clamp(min=1)
    return torch.where(miss, mu, d), mu


def _layout(case, gen):
    """SNP chromosomes and positions, and each gene's window, as host arrays."""
    m, genes = case["m"], case["genes"]
    nc = max(1, min(10, m // 1500))
    chrom = (torch.arange(m) * nc // m).to(torch.int32)
    pos = torch.randint(1, CHROM_LEN, (m,), device=DEV, generator=gen).cpu().to(torch.int64)
    pos = pos[torch.argsort(chrom.to(torch.int64) * CHROM_LEN + pos)]
    gc = torch.randint(0, nc, (genes,), device=DEV, generator=gen).cpu().to(torch.int32)
    tss = torch.randint(1, CHROM_LEN, (genes,), device=DEV, generator=gen).cpu().to(torch.int64)
    return [a.numpy() for a in (gc, (tss - WINDOW).clamp(min=1), tss + WINDOW, chrom, pos)]


def _polygenic(codes, genes, gen):
    sub = codes[:: max(1, codes.shape[0] // 2000)]
    d, mu = _imputed(sub)
    z = (d - mu) / (mu * (1 - mu / 2)).clamp(min=1e-12).sqrt()
    h2 = 0.8 * torch.rand(genes, device=DEV, generator=gen, dtype=torch.float64)
    u = z.T @ torch.randn(z.shape[0], genes, device=DEV, generator=gen, dtype=torch.float64) / math.sqrt(z.shape[0])
    e = torch.randn(z.shape[1], genes, device=DEV, generator=gen, dtype=torch.float64)
    return h2.sqrt() * u + (1 - h2).sqrt() * e


def _planted(codes, windows, Y, gen):
    """One to three cis effects per gene, beta ~ N(0, 0.3^2)."""
    gc, lo, hi, sc, sp = windows
    key, base = sc.astype(np.int64) * (4 * CHROM_LEN) + sp, gc.astype(np.int64) * (4 * CHROM_LEN)
    a, b = np.searchsorted(key, base + lo), np.searchsorted(key, base + hi, side="right")
    r = torch.rand(3, Y.shape[1], device=DEV, generator=gen).cpu().numpy()
    beta = 0.3 * torch.randn(3, Y.shape[1], device=DEV, generator=gen, dtype=torch.float64)
    for k in range(3):
        s = np.minimum(a + (r[k] * np.maximum(b - a, 1)).astype(np.int64), len(key) - 1)
        w = torch.from_numpy(((b > a) & (np.arange(len(gc)) % 3 >= k)).astype(np.float64)).to(DEV)
        d, _ = _imputed(codes[torch.from_numpy(s).to(DEV)])
        Y += (beta[k] * w) * d.T


def _counts(n, genes, C, gen):
    eta = 0.5 + 3.5 * torch.rand(genes, device=DEV, generator=gen, dtype=torch.float64) + 0.2 * C.sum(1, keepdim=True)
    phi = 0.05 + 0.95 * torch.rand(genes, device=DEV, generator=gen, dtype=torch.float64)
    state = torch.random.get_rng_state(), torch.cuda.get_rng_state()
    torch.manual_seed(int(torch.randint(1 << 30, (1,), device=DEV, generator=gen)))
    lam = torch.distributions.Gamma(1 / phi.expand(n, genes), 1 / (phi * eta.exp())).sample()
    Y = torch.poisson(lam)
    torch.random.set_rng_state(state[0])
    torch.cuda.set_rng_state(state[1])
    return Y


def _inputs(case, seed):
    """Everything that the case starts from: codes (and dosages) on the GPU, the rest as host arrays."""
    gen, path = _generator(seed), case["path"]
    n = case["n"]
    d = {}
    if path == "fission":
        Y = _counts(n, case["genes"], torch.zeros(n, 1, device=DEV, dtype=torch.float64), gen)
        k = case["factors"]
        X0 = torch.randn(n, k, device=DEV, generator=gen, dtype=torch.float64)
        W0 = torch.randn(case["genes"], k, device=DEV, generator=gen, dtype=torch.float64)
        return {"Y": _host(Y), "X0": _host(X0), "W0": _host(W0)}
    kin = path in ("lmm_scan", "lmm_job", "grm") or case.get("model") == "lmm"
    d["codes"] = codes = _codes(gen, case.get("n_file", n), case["m"], n // 40 if kin else 0)
    if case.get("dosage"):
        d["dosage"] = _dosage(codes, gen)
    if path == "grm":
        cols = torch.randperm(case["n_file"], device=DEV, generator=gen)[:n].sort().values
        d["cols"] = cols.to(torch.int32).cpu().numpy()
        return d
    C = torch.randn(n, case["p"] - 1, device=DEV, generator=gen, dtype=torch.float64)
    d["X"] = _host(torch.cat([torch.ones(n, 1, device=DEV, dtype=torch.float64), C], 1))
    d["windows"] = _layout(case, gen)
    if path == "glm":
        d["Y"] = _host(_counts(n, case["genes"], C, gen))
        return d
    if kin:
        Y = _polygenic(codes, case["genes"], gen)
    else:
        Y = torch.randn(n, case["genes"], device=DEV, generator=gen, dtype=torch.float64)
    Y += 0.5 * C.sum(1, keepdim=True)
    if path in ("cis", "perm"):
        _planted(codes, d["windows"], Y, gen)
    d["Y"] = _host(Y)
    return d


def _host(a):
    """Column-major host array of a GPU matrix, in page-locked memory as a program that cares for its copies has it."""
    t = torch.empty(a.shape[1], a.shape[0], dtype=a.dtype, pin_memory=True)
    t.copy_(a.T)
    return t.numpy().T


def _pinned(a):
    t = torch.empty(a.shape, dtype=getattr(torch, a.dtype.name), pin_memory=True)
    out = t.numpy()
    out[...] = a
    return out


def _windows(windows, scope):
    code = {"gw": 0, "trans": 1, "cis": 2}[scope]
    return None if code == 0 else (*windows, code)


def prepare(case, seed):
    d, path = _inputs(case, seed), case["path"]
    s = {"case": case, "ctx": capi.Context(0)}
    ctx, n = s["ctx"], case["n"]
    if path == "fission":
        return {**s, **d}
    codes = d.pop("codes")
    dosage = d.pop("dosage", None)
    s.update(d)
    if path in ("lmm_job", "grm"):
        s["rows"] = _pinned(_bed(codes))
        s["cols"] = d.get("cols", np.arange(n, dtype=np.int32))
        return s
    cols = np.arange(n, dtype=np.int32)
    if dosage is not None:
        ctx.load_dosage(dosage.cpu().numpy(), cols)
    else:
        ctx.load_bed(_bed(codes), n, cols)
    if path == "lmm_scan" or case.get("model") == "lmm":
        basis = ctx.lmm_basis(outputs=path == "perm")
    if path in ("lmm_scan", "lm_scan", "glm"):
        ctx.pheno_load(s["Y"], s["X"])
    if path == "perm":
        s.update(_null_fits(case, s, basis if case["model"] == "lmm" else None))
    return s


def _null_fits(case, s, basis):
    """The base vectors that a permutation run shuffles, from each gene's observed null fit."""
    Y, X = s.pop("Y"), s["X"]
    gc, lo, hi, sc, sp = s["windows"]
    B = case["perms"]
    out = {"keys": np.arange(1, case["genes"] + 1, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15),
           "windows": [np.repeat(a, B) for a in (gc, lo, hi)] + [sc, sp]}
    if basis is None:
        out["base"] = np.asfortranarray(Y - X @ np.linalg.lstsq(X, Y, rcond=None)[0])
        return out
    lam, Q = basis
    _, delta = s["ctx"].test_pairs("lmm", Y, X, np.zeros(1, np.int32), np.zeros(1, np.int64))
    Yt, Xt = Q.T @ Y, Q.T @ X
    dinv = 1.0 / (lam[:, None] * delta + 1.0)
    xb0 = np.empty_like(Yt)
    for g in range(Y.shape[1]):
        w = dinv[:, g:g + 1]
        xb0[:, g] = Xt @ np.linalg.solve(Xt.T @ (w * Xt), Xt.T @ (w[:, 0] * Yt[:, g]))
    out.update(base=np.asfortranarray((Yt - xb0) * np.sqrt(dinv)), xb0=np.asfortranarray(xb0),
               dinv=np.asfortranarray(dinv))
    return out


# -------------------------------------------------------------------- the call
def _perm_thr(case):
    """Stage-2 candidates of a trans LM scan: ten times the pair threshold."""
    return 10 * PTHR if case["path"] == "lm_scan" and case["scope"] == "trans" else 0.0


def run(s):
    case, ctx = s["case"], s["ctx"]
    path, n = case["path"], case["n"]
    if path == "lmm_scan":
        ctx.rotate()
        return _scan(case, ctx.scan_trans_lmm(None, None, PTHR, windows=_windows(s["windows"], case["scope"])))
    if path == "lmm_job":
        keep, af, miss = ctx.load_bed(s["rows"], n, s["cols"])
        ctx.pheno_load(s["Y"], s["X"])
        ctx.lmm_basis(outputs=False)
        return {**_scan(case, ctx.scan_trans_lmm(None, None, PTHR)), "keep": keep, "af": af, "miss": miss}
    if path == "lm_scan":
        thr = _perm_thr(case)
        return _scan(case, ctx.scan_trans_lm(None, None, PTHR, thr, _windows(s["windows"], case["scope"])), thr)
    if path == "cis":
        scan = ctx.scan_trans_lm if case["model"] == "lm" else ctx.scan_trans_lmm
        return _scan(case, scan(s["Y"], s["X"], PTHR, windows=_windows(s["windows"], "cis")))
    if path == "perm":
        ctx.pheno_permute(s["base"], s["X"], s["keys"], case["perms"], 1, s.get("xb0"), s.get("dinv"))
        windows = _windows(s["windows"], "cis")
        if case["model"] == "lm":
            return _scan(case, ctx.scan_trans_lm(None, None, 0.0, windows=windows))
        return _scan(case, ctx.scan_trans_lmm(None, None, 0.0, windows=windows, rotated=True))
    if path == "grm":
        keep, af, miss = ctx.load_bed(s["rows"], case["n_file"], s["cols"])
        K, N, used = ctx.grm()
        return {"K": K, "N": N, "used": used, "keep": keep, "af": af, "miss": miss}
    if path == "glm":
        genes, pairs, cands, phi, ok = ctx.scan_glm(None, None, PTHR)
        return {**_scan(case, (genes, pairs, cands)), "phi": phi, "ok": ok}
    Y = ctx.pheno_int(s["Y"])
    X, its = ctx.peer(Y, case["factors"], 1000, 1e-3, s["X0"], s["W0"])
    return {"Y": Y, "X": X, "iterations": its}


def _capacity(case):
    """Rows of the caller's pair buffer: twice the pairs expected by chance, and the planted ones."""
    return 1024 + 4 * case["genes"] + int(2 * PTHR * case["m"] * case["genes"])


def _pairs(case, pairs, thr):
    """The listed pairs in a buffer of a size that the caller chose beforehand, as a C program has it."""
    buf = np.zeros(_capacity(case) * int(round(thr / PTHR)), pairs.dtype)
    buf[:len(pairs)] = pairs
    return buf


def _scan(case, res, perm_thr=0.0):
    genes = res[0]
    out = {f: genes[f] for f in genes.dtype.names}
    for prefix, v, thr in (("pair_", res[1], PTHR), ("cand_", res[2], perm_thr)):
        if thr and case["path"] != "perm":  # permutations list no pairs
            v = _pairs(case, v, thr)
            out.update({prefix + f: v[f] for f in v.dtype.names if f != "reserved"})
    if len(res) > 3:
        out["delta"] = res[3]
    return out


# --------------------------------------------------------------- what it needs
def work(case):
    """Inputs read once, outputs written once, and the operations of the method itself: one contraction over the
    samples per statistic and test, n^2 per rotated SNP, n(n + 1) per GRM marker."""
    path, n, m, g = case["path"], case["n"], case.get("m", 0), case.get("genes", 0)
    p = case.get("p", 1)
    geno = m * n * 4 if case.get("dosage") else m * ((case.get("n_file", n) + 3) // 4)
    if path == "fission":
        k = case["factors"]
        return {"bytes": 8 * (4 * n * g + 2 * k * (n + g)), "flops": 2 * (6 * n * g * k + g * k ** 3 // 3)}
    if path == "grm":
        return {"bytes": geno + 8 * n * n + 2 * n * n + 13 * m, "flops": n * (n + 1) * m}
    tests = m * g
    cols = g
    if path in ("cis", "perm"):
        per = min(m, 2 * WINDOW * m // (max(1, min(10, m // 1500)) * CHROM_LEN))
        cols = g * case.get("perms", 1)
        tests = cols * per
    accs = {"lm_scan": 1, "glm": p + 2}.get(path, 1 if case.get("model") == "lm" else p + 2)
    flops = 2 * n * accs * tests
    if path in ("lmm_scan", "lmm_job"):
        flops += 2 * n * n * m
    if path == "lmm_job":
        flops += n * (n + 1) * m
    return {"bytes": geno + 8 * n * (g if path == "perm" else cols) + 56 * cols, "flops": flops}


# ------------------------------------------------------------ the 64-bit value
def exact(case, seed):
    """The same outputs in plain FP64. Left out: the ACAT sums (they hinge on how the t tail is quantised near
    t = 0, which the reference's own arithmetic defines), REML's delta (the optimum is flat: the statistics at it
    are what has a value), the NB-GLM (its null fits are defined by their stopping rule) and the drawn
    permutations."""
    path = case["path"]
    if path in ("glm", "perm"):
        return None
    d = _inputs(case, seed)
    if path == "fission":
        return _exact_fission(case, d)
    if path == "grm":
        return {"K": _exact_grm(d["codes"], torch.from_numpy(d["cols"]).to(DEV).long())[0].cpu().numpy(), "N": None,
                "used": None, "keep": None, "af": None, "miss": None}
    rows = d["dosage"] if case.get("dosage") else d["codes"]
    mixed = path in ("lmm_scan", "lmm_job") or case.get("model") == "lmm"
    scope = case.get("scope", "cis" if path == "cis" else "gw")
    out = _exact_scan(rows, d["Y"], d["X"], d["windows"], scope, mixed, _perm_thr(case))
    for f, v in out.items():
        if v is not None and f.startswith(("pair_", "cand_")):
            thr = PTHR if f.startswith("pair_") else _perm_thr(case)
            out[f] = _pairs(case, v, thr)
    return out


def _exact_grm(codes, cols):
    n = cols.numel()
    A = torch.zeros(n, n, device=DEV, dtype=torch.float64)
    J = torch.zeros_like(A)
    used = 0
    for s in range(0, codes.shape[0], 16384):
        c = codes[s:s + 16384][:, cols]
        d, mu = _imputed(c)
        ok = ((mu > 2e-8) & (mu < 2 - 2e-8))[:, 0]
        c, d, mu = c[ok], d[ok], mu[ok]
        z = (d - mu) / (mu * (1 - mu / 2)).sqrt()
        A += z.T @ z
        miss = (c < 0).to(torch.float64)
        J += miss.T @ miss
        used += int(ok.sum())
    miss = J.diagonal().clone()
    N = used - miss[:, None] - miss[None, :] + J
    return A / N, N


def _weights(delta, lam):
    return 1.0 / (lam[:, None] * delta + 1.0).clamp(min=1e-12)


def _negll(delta, Yt, Xt, lam):
    """-loglik of every column at its own delta, A = X'WX and b = X'Wy."""
    n, p = Xt.shape
    W = _weights(delta, lam)
    A = torch.einsum("ia,ib,ig->gab", Xt, Xt, W) if p < 3 else ((Xt[:, :, None] * Xt[:, None, :]).reshape(n, p * p).T @ W).T.reshape(-1, p, p)
    b = (Xt.T @ (W * Yt)).T
    L = torch.linalg.cholesky(A)
    z = torch.linalg.solve_triangular(L, b[:, :, None], upper=False)[:, :, 0]
    q = ((W * Yt * Yt).sum(0) - (z * z).sum(1)).clamp(min=1e-12)
    ld = 2 * L.diagonal(dim1=1, dim2=2).log().sum(1)
    return 0.5 * ((n - p) * torch.log(q / (n - p)) - W.log().sum(0) + ld), A, b, q


def _reml(Yt, Xt, lam):
    """Each column's REML delta: the grid, then golden section (log-spaced refinement is not the point here)."""
    f = lambda d: _negll(d, Yt, Xt, lam)[0]  # noqa: E731
    grid = [1.0] + [1e-5 * 2.0 ** k for k in range(34)]
    vals = torch.stack([f(torch.full((Yt.shape[1],), g, device=DEV, dtype=torch.float64)) for g in grid])
    best = torch.tensor(grid, device=DEV, dtype=torch.float64)[vals.argmin(0)]
    lo, hi = (best / 4).clamp(min=1e-8), (best * 4).clamp(max=1e6)
    phi = (1 + math.sqrt(5)) / 2
    for _ in range(40):
        a, b = hi - (hi - lo) / phi, lo + (hi - lo) / phi
        left = f(a) < f(b)
        lo, hi = torch.where(left, lo, a), torch.where(left, b, hi)
    return 0.5 * (lo + hi)


def _t_p(t, df):
    """Two-sided Student-t p of a FP64 tensor: the regularised incomplete beta function by Lentz's continued fraction."""
    x = df / (df + t * t)
    a, b = torch.full_like(x, 0.5 * df), torch.full_like(x, 0.5)
    swap = ~(x < (a + 1) / (a + b + 2))
    a, b, x = torch.where(swap, b, a), torch.where(swap, a, b), torch.where(swap, t * t / (df + t * t), x)
    front = torch.exp(a * x.log() + b * torch.log1p(-x) - torch.lgamma(a) - torch.lgamma(b) + torch.lgamma(a + b)) / a
    c, d = torch.ones_like(x), 1 / (1 - (a + b) * x / (a + 1))
    h = d.clone()
    for k in range(1, 400):
        for aa in (k * (b - k) * x / ((a - 1 + 2 * k) * (a + 2 * k)),
                   -(a + k) * (a + b + k) * x / ((a + 2 * k) * (a + 1 + 2 * k))):
            d, c = 1 / (1 + aa * d), 1 + aa / c
            h = h * d * c
    return torch.where(swap, 1 - front * h, front * h).clamp(0, 1)


def _t_critical(p, df):
    lo, hi = 0.0, 1e3
    for _ in range(100):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if float(_t_p(torch.tensor([mid], dtype=torch.float64), df)) > p else (lo, mid)
    return hi


def _exact_scan(rows, Y, X, windows, scope, mixed, cand_thr):
    Y, X = torch.from_numpy(np.array(Y)).to(DEV), torch.from_numpy(np.array(X)).to(DEV)
    (n, G), p, m = Y.shape, X.shape[1], rows.shape[0]
    df = n - p - 1
    if mixed:
        lam, Q = torch.linalg.eigh(_exact_grm(rows, torch.arange(n, device=DEV))[0])
        lam = lam.clamp(min=0)
        Yt, Xt = Q.T @ Y, Q.T @ X
        delta = torch.cat([_reml(Yt[:, g:g + 2000], Xt, lam) for g in range(0, G, 2000)])
        _, A, b, rss = _negll(delta, Yt, Xt, lam)
        W = _weights(delta, lam)
        R = W * (Yt - Xt @ torch.linalg.solve(A, b[:, :, None])[:, :, 0].T)
        U = torch.linalg.cholesky(torch.linalg.inv(A))  # a'A^-1 a = |U'a|^2
    else:
        P = torch.linalg.inv(X.T @ X) @ X.T
        R = Y - X @ (P @ Y)
        rss = (R * R).sum(0)
    gc, lo, hi, sc, sp = [torch.from_numpy(a).to(DEV) for a in windows]
    best = {k: torch.zeros(G, device=DEV, dtype=torch.float64) for k in ("beta", "s", "t2")}
    best["t2"] -= 1
    best_snp = torch.full((G,), -1, device=DEV)
    t_min = _t_critical(max(PTHR, cand_thr), df)
    found = []
    step = max(256, min(16384, 300_000_000 // (8 * G)))
    for s in range(0, m, step):
        d, mu = _imputed(rows[s:s + step])
        g = d - mu
        if mixed:
            g = g @ Q
            num = g @ R
            S = (g * g) @ W
            for k in range(p):
                S -= (g @ (W * (Xt @ U[:, :, k].T))).square()
        else:
            num = g @ R
            S = ((g * g).sum(1) - ((g @ X) * (g @ P.T)).sum(1))[:, None].expand(-1, G)
        r = num * num / (S * rss)
        t2 = df * r / (1 - r)
        if scope != "gw":
            k = slice(s, s + step)
            near = (sc[k, None] == gc) & (sp[k, None] >= lo) & (sp[k, None] <= hi)
            t2 = torch.where(near == (scope == "cis"), t2, torch.full_like(t2, -1.0))
        top, at = t2.max(0)
        better = top > best["t2"]
        col = torch.arange(G, device=DEV)
        for key, v in (("beta", (num / S)[at, col]), ("s", S[at, col]), ("t2", top)):
            best[key] = torch.where(better, v, best[key])
        best_snp = torch.where(better, at + s, best_snp)
        i, j = torch.nonzero(t2 >= t_min * t_min, as_tuple=True)
        found.append(torch.stack([(i + s).double(), j.double(), (num / S)[i, j], S[i, j], t2[i, j]]))
    snp, gene, beta, _, t2 = torch.cat(found, 1)

    def fields(beta, t2, prefix, order):
        t = t2.clamp(min=0).sqrt() * beta.sign()
        v = {"beta": beta, "se": beta.abs() / t.abs(), "t": t, "p": _t_p(t, df), "r2": t2 / (t2 + df)}
        return {prefix + k: x[order].cpu().numpy() for k, x in v.items()}

    none = {"n_tested": None, "acat_used": None, "acat_tan_sum": None, "best_snp": None, "delta": None}
    tested = torch.nonzero(best["t2"] >= 0)[:, 0]
    out = {**none, **(fields(best["beta"], best["t2"], "best_", tested) if tested.numel() == G else {})}
    p_of = _t_p(t2.sqrt(), df)
    keep = torch.nonzero(p_of <= PTHR)[:, 0]
    out.update(fields(beta, t2, "pair_", keep[torch.argsort(snp[keep] * G + gene[keep])]))
    if cand_thr:
        keep = torch.nonzero(p_of < cand_thr)[:, 0]
        order = np.lexsort((snp[keep].cpu().numpy(), p_of[keep].cpu().numpy(), gene[keep].cpu().numpy()))
        out.update(fields(beta, t2, "cand_", keep[torch.from_numpy(order).to(DEV)]))
    return out


def _exact_fission(case, d):
    Y = torch.from_numpy(np.array(d["Y"])).to(DEV)
    n, G = Y.shape
    srt = Y.T.contiguous().sort(1).values
    at = Y.T.contiguous()
    rank = 0.5 * (torch.searchsorted(srt, at, right=False) + 1 + torch.searchsorted(srt, at, right=True)).double()
    Z = torch.special.ndtri((rank - 0.5) / n).T
    # PEER: W, Alpha, X and Eps updates until the mean squared residual rests
    k = case["factors"]
    X, W = (torch.from_numpy(np.array(d[v])).to(DEV) for v in ("X0", "W0"))
    Yc = Z - Z.mean(0)
    eye = torch.eye(k, device=DEV, dtype=torch.float64)
    eps = torch.full((G,), 0.01, device=DEV, dtype=torch.float64)
    XE, alpha = n * eye + X.T @ X, torch.full((k,), (0.001 + 0.5 * G) / 0.1, device=DEV, dtype=torch.float64)
    b1, last = (Yc * Yc + 0.01).sum(0), math.inf
    for _ in range(1000):
        XtY = X.T @ Yc
        cov = torch.linalg.inv(torch.diag(alpha) + eps[:, None, None] * XE)
        W = eps[:, None] * (cov @ XtY.T[:, :, None])[:, :, 0]
        E2 = cov + W[:, :, None] * W[:, None, :]
        alpha = (0.001 + 0.5 * G) / (0.1 + 0.5 * E2.sum(0).diagonal())
        Xcov = torch.linalg.inv((eps[:, None, None] * E2).sum(0) + eye)
        X = Yc @ (W * eps[:, None]) @ Xcov
        XE = n * Xcov + X.T @ X
        b = 10 + 0.5 * (b1 - 2 * (XtY.T * W).sum(1) + (XE * E2).sum((1, 2)))
        eps = (0.1 + 0.5 * n) / b.clamp(min=1e-10)
        res = float(((Yc - X @ W.T) ** 2).mean())
        if abs(last - res) < 1e-3:
            break
        last = res
    return {"Y": Z.cpu().numpy(), "X": X.cpu().numpy(), "iterations": None}
