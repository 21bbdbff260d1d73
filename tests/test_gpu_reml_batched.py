"""GPU parity of the batched REML (p > 3 covariate columns): the group sizes of
its factorisation kernels (8, 16 and 32 lanes) at their edges, with one column,
a part of a block, and several blocks of columns."""
import numpy as np
import pytest

import restate as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [4, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("G", [1, 3, 37])
def test_batched_reml_matches_oracle(p, G):
    """Each column's delta is an optimum of the oracle's objective (-loglik
    within 1e-6 relative of the oracle's own search; the optimum is flat), and
    the pair statistics that use the caches (chi0, the factor of A00, rss)
    match the oracle's at that delta within 1e-6."""
    from eqtl_b200 import capi, synth
    n, m = 131, 12
    rng = np.random.default_rng(100 * p + G)
    g = synth.make_genotypes(5, n=n, m=m, n_chrom=1, chrom_len=1_000_000, miss_rate=0.0, maf_lo=0.1)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    lam = np.sort(np.concatenate([np.zeros(1), rng.gamma(0.5, 2.0, n - 1)]))
    X = np.column_stack([np.ones(n), rng.standard_normal((n, p - 1))])
    Y = (Q * np.sqrt(rng.uniform(0, 2, G)[:, None, None] * lam + 1.0)) @ rng.standard_normal((n, 1))
    Y = Y[:, :, 0].T + 0.3 * X.sum(1, keepdims=True)
    cols = np.repeat(np.arange(G, dtype=np.int32), 2)
    snps = np.tile(np.array([0, m - 1], np.int64), G)
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(g.codes), n, np.arange(n))
        c.set_basis(Q, lam)
        out, delta = c.test_pairs("lmm", Y, X, cols, snps)
    Xt, df = Q.T @ X, n - p
    for j in range(G):
        yt = Q.T @ Y[:, j]
        best = R.reml_negll(R.optimize_delta(yt, Xt, lam), yt, Xt, lam, df)
        assert abs(R.reml_negll(delta[j], yt, Xt, lam, df) - best) <= 1e-6 * abs(best), (j, delta[j])
        st = R.test_lmm_many(R.prep_lmm(Y[:, j], X, Q, lam, delta=delta[j]), g.codes[[0, m - 1]].astype(float))
        for f, k in (("beta", "beta"), ("se", "se"), ("t", "stat")):
            np.testing.assert_allclose(out[f][2 * j:2 * j + 2], st[k], rtol=1e-6, atol=1e-12)
