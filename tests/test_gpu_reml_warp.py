"""GPU parity of the REML of up to 3 covariate columns (one warp per column): few
samples, a ragged last pass over them, an idle second warp, more than one block."""
import numpy as np
import pytest

import restate as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [1, 2, 3])
@pytest.mark.parametrize("n,G", [(12, 1), (32, 2), (65, 37)])
def test_warp_reml_matches_oracle(n, p, G):
    """-loglik at each column's delta within 1e-6 relative of the oracle's own
    search (the optimum is flat), pair statistics at that delta within 1e-6."""
    from eqtl_b200 import capi, synth
    rng = np.random.default_rng(1000 * n + 10 * p + G)
    codes = rng.binomial(2, 0.4, (3, n)).astype(np.int8)
    codes[:, :3] = [0, 1, 2]
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    lam = np.sort(np.concatenate([np.zeros(1), rng.gamma(0.5, 2.0, n - 1)]))
    X = np.column_stack([np.ones(n), rng.standard_normal((n, p - 1))])
    Y = (Q * np.sqrt(rng.uniform(0, 2, G)[:, None, None] * lam + 1.0)) @ rng.standard_normal((n, 1))
    Y = Y[:, :, 0].T + 0.3 * X.sum(1, keepdims=True)
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        c.set_basis(Q, lam)
        out, delta = c.test_pairs("lmm", Y, X, np.arange(G, dtype=np.int32), np.full(G, 2, np.int64))
    Xt, df = Q.T @ X, n - p
    for j in range(G):
        yt = Q.T @ Y[:, j]
        best = R.reml_negll(R.optimize_delta(yt, Xt, lam), yt, Xt, lam, df)
        assert abs(R.reml_negll(delta[j], yt, Xt, lam, df) - best) <= 1e-6 * abs(best), (j, delta[j])
        st = R.test_lmm_many(R.prep_lmm(Y[:, j], X, Q, lam, delta=delta[j]), codes[2:3].astype(float))
        for f, k in (("beta", "beta"), ("se", "se"), ("t", "stat")):
            np.testing.assert_allclose(out[f][j], st[k][0], rtol=1e-6, atol=1e-12)
