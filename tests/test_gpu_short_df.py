"""GPU: scans with few residual degrees of freedom (below about 29), whose long tails
the epilogues screen from the node tables instead of the per-interval cubics: SNP
counts around the chunk of 16 and the tile, every epilogue, with and without windows.
The screen's FP32 r = t^2 / (t^2 + df) is good to about 6e-7 of 1 - r; at r <= 0.9 and
df <= 28 (t <= 16) that is up to 16 / 0.2 * 6e-7 = 5e-5 of t."""
import numpy as np
import pytest

import oracle_scan
from gpu_util import check_scan

pytestmark = pytest.mark.gpu
T_ERR_SHORT = 5e-5


@pytest.mark.parametrize("model,p", [("lm", 1), ("lm", 3), ("lmm", 1), ("lmm", 2), ("lmm", 3)])
@pytest.mark.parametrize("df", [8, 28])
@pytest.mark.parametrize("m,G", [(15, 3), (257, 130), (700, 300)])
@pytest.mark.parametrize("scope", [0, 1, 2])
def test_short_df(model, p, df, m, G, scope):
    from eqtl_b200 import capi, synth
    n = df + p + 1
    rng = np.random.default_rng(1000 * df + 10 * m + p)
    codes = rng.binomial(2, rng.uniform(0.2, 0.8, (m, 1)), (m, n)).astype(np.int8)
    codes[:, :6] = [0, 1, 2, 0, 1, 2]
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    lam = np.sort(rng.gamma(0.5, 2.0, n))
    X = np.column_stack([np.ones(n), rng.standard_normal((n, p - 1))])
    Y = rng.standard_normal((n, G))
    pos = np.sort(rng.integers(1, 1_000_000, m))
    lo = rng.integers(1, 900_000, G)
    w = (rng.integers(0, 2, G).astype(np.int32), lo, lo + 150_000, np.zeros(m, np.int32), pos)
    windows = w + (scope,) if scope else None
    inside = oracle_scan.windows_mask(w[3], w[4], *w[:3])
    excl = None if scope == 0 else inside if scope == 1 else ~inside
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        if model == "lm":
            res = c.scan_trans_lm(Y, X, pthr=1e-3, windows=windows)
            ora, ref = oracle_scan.trans_lm(codes.astype(float), Y, X, 1e-3, excl=excl)
            check_scan(res, ora, ref, 1e-3, df, t_err=T_ERR_SHORT, rel=1e-8)
        else:
            c.set_basis(Q, lam)
            res = c.scan_trans_lmm(Y, X, pthr=1e-3, windows=windows)
            ora, ref = oracle_scan.trans_lmm(codes.astype(float), Y, X, Q, lam, 1e-3, deltas=res[3], excl=excl)
            check_scan(res[:3], ora, ref, 1e-3, df, t_err=T_ERR_SHORT, rel=1e-6)
