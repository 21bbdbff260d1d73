"""GPU parity of the grouped scans (p > 2) on 128-SNP tiles: gene counts around
the 128-row tile, the pair of tiles and the rule that picks pairs, SNP counts
around the tile and the 16-SNP chunk, odd and even accumulator counts (a last
group of one or of two), dense and with window lists."""
import numpy as np
import pytest

import oracle_scan
from gpu_util import T_ERR, check_scan

pytestmark = pytest.mark.gpu


def _codes(rng, m, n):
    c = rng.binomial(2, rng.uniform(0.1, 0.9, (m, 1)), (m, n)).astype(np.int8)
    c[:, :3] = [0, 1, 2]
    return c


def _windows(rng, m, G):
    pos = np.sort(rng.integers(1, 1_000_000, m))
    lo = rng.integers(1, 900_000, G)
    return rng.integers(0, 2, G).astype(np.int32), lo, lo + 150_000, np.zeros(m, np.int32), pos


@pytest.mark.parametrize("G,m", [(1, 15), (127, 128), (129, 129), (256, 385), (257, 112), (897, 257)])
@pytest.mark.parametrize("p", [3, 4])
@pytest.mark.parametrize("windows", [False, True])
def test_grouped_lmm(G, m, p, windows):
    from eqtl_b200 import capi, synth
    n = 66
    rng = np.random.default_rng(G + m + p)
    codes = _codes(rng, m, n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    lam = np.sort(rng.gamma(0.5, 2.0, n))
    X = np.column_stack([np.ones(n), rng.standard_normal((n, p - 1))])
    Y = (Q * np.sqrt(lam + 1.0)) @ rng.standard_normal((n, G))
    Y[:, G - 1] += 2.0 * codes[m - 1]
    w = _windows(rng, m, G) if windows else None
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        c.set_basis(Q, lam)
        res = c.scan_trans_lmm(Y, X, pthr=1e-3, **({"windows": w + (True,)} if windows else {}))
    excl = oracle_scan.windows_mask(w[3], w[4], *w[:3]) if windows else None
    ora, ref = oracle_scan.trans_lmm(codes.astype(float), Y, X, Q, lam, 1e-3, deltas=res[3], excl=excl)
    check_scan(res[:3], ora, ref, 1e-3, n - p - 1, rel=1e-6)


@pytest.mark.parametrize("G,m", [(1, 15), (129, 129), (256, 257)])
@pytest.mark.parametrize("p", [3, 4])
def test_grouped_glm(G, m, p):
    from eqtl_b200 import capi, synth
    n = 90
    rng = np.random.default_rng(G + m + p)
    codes = _codes(rng, m, n)
    X = np.column_stack([np.ones(n), rng.standard_normal((n, p - 1))])
    mu = np.exp(2.0 + 0.2 * X[:, 1:].sum(1, keepdims=True) + rng.normal(0, 0.2, (1, G)))
    Y = rng.poisson(mu * rng.gamma(4.0, 0.25, (n, G))).astype(float)
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        genes, pairs, cands, phi, conv = c.scan_glm(Y, X, pthr=1e-3)
    ora, ref = oracle_scan.glm(codes.astype(float), Y, X, 1e-3)
    assert np.array_equal(conv, ora["converged"])
    check_scan((genes, pairs, cands), ora, ref, 1e-3, None, t_err=T_ERR, rel=1e-6)
