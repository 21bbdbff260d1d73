"""GPU parity of the LM scan's 16-pair screen at the sizes and values where its
chunk form hands over to the general one: SNP counts around 16 and 256, a SNP
that fails the subset gate inside a chunk, equal SNPs (ties for the best), a
phenotype without variance, a deferred p, a perfect fit and a NaN."""
import numpy as np
import pytest

import oracle_scan
import restate as R
from gpu_util import check_scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 15, 16, 17, 255, 256, 257, 515])
def test_lm_screen_chunk_edges(m):
    from eqtl_b200 import capi, synth
    n, G = 120, 131
    rng = np.random.default_rng(m)
    codes = rng.binomial(2, rng.uniform(0.1, 0.9, (m, 1)), (m, n)).astype(np.int8)
    codes[:, 0] = 1  # no SNP is monomorphic
    codes[:, 1] = 2
    if m > 12:
        codes[9] = codes[5]                    # a tie inside a chunk
        codes[m - 1] = codes[5]                # and one across chunks
    flat, perfect, missing = 2, 3, 4
    X = np.column_stack([np.ones(n), rng.standard_normal(n)])
    Y = rng.standard_normal((n, G))
    Y[:, 1] += 6.0 * codes[min(5, m - 1)]      # p < 1e-14: its term is left to the host
    Y[:, flat] = 3.0                           # no variance left
    Y[:, perfect] = codes[min(7, m - 1)] + X @ [0.5, -1.0]
    Y[5, missing] = np.nan
    rows = synth.pack_bed_rows(codes)
    with capi.Context(0) as c:
        c.load_bed(rows, n, np.arange(n))
        genes, pairs, cands = c.scan_trans_lm(Y, X, pthr=1e-2)
    dec = R.decode_bed_rows(rows, n, np.arange(n), "impute", 0.8, 0.0)
    assert dec.keep.all()
    # every SNP is tested; a NaN phenotype enters no p. What is left of a flat or
    # perfectly fitted phenotype is rounding noise: its p has no value to compare
    assert np.all(genes["n_tested"] == m) and genes["acat_used"][missing] == 0
    rest = np.setdiff1d(np.arange(G), [flat, perfect, missing])
    ora, ref = oracle_scan.trans_lm(dec.dosage, Y[:, rest], X, 1e-2)
    at = {int(g): j for j, g in enumerate(rest)}
    pairs = pairs[np.isin(pairs["gene"], rest)].copy()
    pairs["gene"] = [at[int(g)] for g in pairs["gene"]]
    check_scan((genes[rest], pairs, cands), ora, ref, 1e-2, n - 3)


@pytest.mark.parametrize("gated", [0, 7, 15, 16, 40])
def test_lm_screen_gate_in_chunk(gated):
    """On a sample view one SNP loses its variance: it is not tested, the other
    SNPs of its chunk are."""
    from eqtl_b200 import capi, synth
    n, m, G = 90, 41, 20
    rng = np.random.default_rng(gated)
    codes = rng.binomial(2, 0.4, (m, n)).astype(np.int8)
    codes[:, :2] = [0, 2]
    sub = np.arange(10, 90)
    codes[gated, 10:] = 0
    codes[gated, :10] = rng.integers(0, 3, 10)
    codes[gated, :2] = [0, 2]
    Y = rng.standard_normal((n, G))
    X = np.ones((n, 1))
    rows = synth.pack_bed_rows(codes)
    with capi.Context(0) as c:
        c.load_bed(rows, n, np.arange(n))
        c.geno_subset(sub)
        res = c.scan_trans_lm(Y[sub], X[sub], pthr=1e-2)
    dec = R.decode_bed_rows(rows, n, np.arange(n), "impute", 0.8, 0.0)
    ora, ref = oracle_scan.trans_lm(dec.dosage[:, sub], Y[sub], X[sub], 1e-2)
    assert np.all(res[0]["n_tested"] == m - 1)
    check_scan(res, ora, ref, 1e-2, len(sub) - 2)


@pytest.mark.parametrize("scope", [1, 2])
@pytest.mark.parametrize("model,p", [("lm", 2), ("lmm", 1), ("lmm", 2), ("lmm", 4)])
def test_screen_window_blocks(model, p, scope):
    """Blocks of 16 SNPs inside every gene's window, clear of all of them, and
    mixed (window edges and a chromosome's end inside a block), for genes with a
    window over the whole chromosome, a part of it, one SNP, nothing, and no
    location."""
    from eqtl_b200 import capi, synth
    n, G = 75, 70
    rng = np.random.default_rng(7 + p)
    per = [150, 89, 40]                      # chromosomes that end inside blocks
    m = sum(per)
    schrom = np.repeat(np.arange(3), per).astype(np.int32)
    spos = np.concatenate([np.sort(rng.choice(np.arange(1, 4000), k, replace=False)) for k in per])
    codes = rng.binomial(2, rng.uniform(0.15, 0.85, (m, 1)), (m, n)).astype(np.int8)
    codes[:, :3] = [0, 1, 2]
    gchrom = rng.integers(-1, 3, G).astype(np.int32)
    lo = rng.integers(1, 4000, G)
    hi = lo + rng.integers(0, 2500, G)
    gchrom[:34], lo[:34], hi[:34] = 0, 1, 4000          # a warp whose genes share a window
    hi[40] = lo[40] = spos[200]
    gchrom[40] = schrom[200]
    gchrom[41], lo[41], hi[41] = 1, 3990, 100
    X = np.column_stack([np.ones(n), rng.standard_normal((n, p - 1))])
    Y = rng.standard_normal((n, G))
    win = (gchrom, lo, hi, schrom, spos, scope)
    mask = oracle_scan.windows_mask(schrom, spos, gchrom, lo, hi)
    excl = mask if scope == 1 else ~mask
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        if model == "lm":
            res = c.scan_trans_lm(Y, X, pthr=1e-2, windows=win)
            ora, ref = oracle_scan.trans_lm(codes.astype(float), Y, X, 1e-2, excl=excl)
        else:
            Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
            lam = np.sort(rng.gamma(0.5, 2.0, n))
            c.set_basis(Q, lam)
            res = c.scan_trans_lmm(Y, X, pthr=1e-2, windows=win)
            ora, ref = oracle_scan.trans_lmm(codes.astype(float), Y, X, Q, lam, 1e-2, excl=excl, deltas=res[3])
    check_scan(res[:3], ora, ref, 1e-2, n - p - 1, rel=1e-9 if model == "lm" else 1e-6)
