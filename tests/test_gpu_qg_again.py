"""GPU: pairs whose S = gg - a'A00^-1 a cancels (genes with delta at the top of the
search) in a refinement whose Q'g is exact. They are done again by DGEMM, some or
all pairs of the list, so that they agree with the same pairs tested alone."""
import numpy as np
import pytest

import restate as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("high", [0, 1, 3])
def test_cancelling_pairs(high):
    from eqtl_b200 import capi, synth
    n, m, G = 1201, 7700, 3
    rng = np.random.default_rng(high)
    codes = rng.binomial(2, rng.uniform(0.1, 0.9, (m, 1)), (m, n)).astype(np.int8)
    codes[:, :3] = [0, 1, 2]
    assert n * n * m >= 10 << 30
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    lam = np.sort(np.concatenate([np.zeros(1), rng.gamma(0.5, 2.0, n - 1)]))
    X = np.ones((n, 1))
    h = np.where(np.arange(G) < high, 1e8, 1.0)
    Y = np.column_stack([(Q * np.sqrt(v * lam + 1.0)) @ rng.standard_normal(n) for v in h])
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        c.set_basis(Q, lam)
        cols, snps = np.repeat(np.arange(G, dtype=np.int32), m), np.tile(np.arange(m), G)
        out, delta = c.test_pairs("lmm", Y, X, cols, snps)
        few = rng.permutation(G * m)[:200]
        alone, _ = c.test_pairs("lmm", Y, X, cols[few], snps[few])
    assert (delta[:high] > 1e4).all() and (delta[high:] < 1e4).all()
    # S keeps at least 1e-8 of gg here: 1e-16 sqrt(n) / 1e-8 of rounding is below 1e-6
    for f in ("beta", "t"):
        np.testing.assert_allclose(out[f][few], alone[f], rtol=1e-6, atol=1e-6 * np.abs(alone[f]).mean())
    for j in range(G):
        st = R.test_lmm_many(R.prep_lmm(Y[:, j], X, Q, lam, delta=delta[j]), codes.astype(float))
        np.testing.assert_allclose(out["t"][j * m:(j + 1) * m], st["stat"], rtol=1e-6, atol=1e-6)
