"""GPU: the rounding error of the LM's per-SNP residual sums of squares against 80-bit
sums. beta and se of a pair give gtg back, 1 / (se^2 (t^2 + df)) = gtg / yty, with
some four roundings; the sums of squares themselves carry at most 8 units of u = 2^-53
(chains of four, four of them, a compensated total), where one chain over the samples
carries n / 2 of them when its addends repeat, as a SNP's few dosages do."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = np.longdouble


def _inverse(a):
    p = len(a)
    b = np.concatenate([a, np.eye(p, dtype=L)], 1)
    for i in range(p):
        b[i] /= b[i, i]
        for r in range(p):
            if r != i:
                b[r] -= b[r, i] * b[i]
    return b[:, p:]


@pytest.mark.parametrize("n", [63, 320, 1000, 2000])
@pytest.mark.parametrize("p", [1, 11, 24, 32])
def test_gtg_rounding(n, p):
    from eqtl_b200 import capi, synth
    rng = np.random.default_rng(n + p)
    m = 300
    codes = rng.binomial(2, rng.uniform(0.05, 0.95, (m, 1)), (m, n)).astype(np.int8)
    codes[:, :3] = [0, 1, 2]
    codes[rng.random((m, n)) < 0.01] = -1
    X = np.column_stack([np.ones(n), rng.standard_normal((n, p - 1))])
    Y = rng.standard_normal((n, 1))
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        assert c.n_kept == m
        out, _ = c.test_pairs("lm", Y, X, np.zeros(m, np.int32), np.arange(m))
    t, se = out["t"].astype(L), out["se"].astype(L)
    d = codes.astype(float)
    mu = np.array([x[x >= 0].mean() for x in d])[:, None]
    g, xl = np.where(d < 0, 0.0, d - mu).astype(L), X.astype(L)
    v = g @ xl
    gtg = (g * g).sum(1) - np.einsum("ia,ab,ib->i", v, _inverse(xl.T @ xl), v)
    err = (1 / (se * se * (t * t + (n - p - 1)) * gtg)).astype(L)
    err = (err / np.median(err) - 1).astype(float)  # yty, the same for all SNPs, and its error drop out
    assert np.sqrt((err ** 2).mean()) < 8 * 2.0 ** -53
