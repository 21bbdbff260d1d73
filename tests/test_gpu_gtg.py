"""GPU parity of the LM's per-SNP residual sums of squares and gate
(snp_gtg_kernel) at the edges of its blocks (128 SNPs, 32 samples) and of its
covariate instances, from 2-bit rows with a shuffled sample map and from FP32
dosages."""
import numpy as np
import pytest

import restate as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [1, 2, 3, 12, 13, 25, 32])
@pytest.mark.parametrize("n,m", [(40, 1), (64, 127), (65, 129), (97, 300)])
@pytest.mark.parametrize("dense", [False, True])
def test_lm_denominators(p, n, m, dense):
    """beta = gty / gtg and t of every SNP against the oracle within 1e-9, the
    LM's stated FP64 tolerance."""
    from eqtl_b200 import capi, synth
    rng = np.random.default_rng(1000 * p + n)
    n_file = n + 5
    codes = rng.binomial(2, rng.uniform(0.15, 0.85, (m, 1)), (m, n_file)).astype(np.int8)
    codes[rng.random((m, n_file)) < 0.05] = -1
    codes[:, :8] = [0, 1, 2, 0, 1, 2, 0, 2]
    cols = rng.permutation(n_file)[:n].astype(np.int32)
    cols[:8] = np.arange(8)
    cols = np.unique(cols)
    cols = np.concatenate([cols, np.setdiff1d(np.arange(n_file), cols)[:n - cols.size]]).astype(np.int32)
    rng.shuffle(cols)
    X = np.column_stack([np.ones(n), rng.standard_normal((n, p - 1))])
    Y = rng.standard_normal((n, 1)) + 0.5 * X.sum(1, keepdims=True)
    snps = np.arange(m, dtype=np.int64)
    with capi.Context(0) as c:
        if dense:
            ds = codes.astype(np.float32) * 0.75
            ds[codes < 0] = np.nan
            c.load_dosage(ds, cols)
            dos = R.decode_dosage_rows(ds, cols, "impute", 0.8, 0.0).dosage
        else:
            rows = synth.pack_bed_rows(codes)
            c.load_bed(rows, n_file, cols)
            dos = R.decode_bed_rows(rows, n_file, cols, "impute", 0.8, 0.0).dosage
        assert c.n_kept == m
        out, _ = c.test_pairs("lm", Y, X, np.zeros(m, np.int32), snps)
    st = R.test_lm_many(R.prep_lm(Y[:, 0], X), dos)
    np.testing.assert_allclose(out["beta"], st["beta"], rtol=1e-9, atol=1e-13)
    np.testing.assert_allclose(out["se"], st["se"], rtol=1e-9)
    np.testing.assert_allclose(out["t"], st["stat"], rtol=1e-8, atol=1e-10)
