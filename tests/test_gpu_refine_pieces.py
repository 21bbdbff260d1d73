"""GPU: lists so long that the refinement takes them in pieces (32 MB of sums a piece:
123,000 pairs with 32 covariates, 175,000 of the NB-GLM with 20) and the results leave
the device in pieces of 2^20 pairs. Every pair is listed with pthr = 1, or nearly so with
0.999 (the LMM lists no pair whose |t| is rounding). The device memory that such a
scan takes does not grow with the covariates."""
import numpy as np
import pytest

import oracle_scan

pytestmark = pytest.mark.gpu


def _codes(rng, m, n):
    codes = rng.binomial(2, rng.uniform(0.2, 0.8, (m, 1)), (m, n)).astype(np.int8)
    codes[:, :3] = [0, 1, 2]
    return codes


def _check(pairs, cands, st, pthr, perm_thr, rtol):
    m, G = st["p"].shape
    listed = (st["p"] <= pthr).ravel()
    got = np.zeros(m * G, bool)
    key = pairs["snp"] * G + pairs["gene"]
    assert (np.diff(key) > 0).all()
    got[key] = True
    edge = np.abs(st["p"].ravel() - pthr) < (1e-6 if pthr < 1 else 0)  # either side of the threshold
    assert np.array_equal(got | edge, listed | edge) and got.mean() > 0.99
    for f, k in (("beta", "beta"), ("t", "stat")):
        ref = st[k].ravel()[key]
        np.testing.assert_allclose(pairs[f], ref, rtol=rtol, atol=rtol * np.abs(ref).mean())
    want = pairs[pairs["p"] < perm_thr]
    assert np.array_equal(cands, want[np.lexsort((want["snp"], want["p"], want["gene"]))])


def test_lmm_pieces():
    from eqtl_b200 import capi, synth
    n, m, G, p = 80, 1100, 300, 32
    rng = np.random.default_rng(1)
    codes = _codes(rng, m, n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    lam = np.sort(rng.gamma(0.5, 2.0, n))
    X = np.column_stack([np.ones(n), rng.standard_normal((n, p - 1))])
    Y = (Q * np.sqrt(lam + 1.0)) @ rng.standard_normal((n, G))
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        c.set_basis(Q, lam)
        genes, pairs, cands, delta = c.scan_trans_lmm(Y, X, pthr=0.999, perm_thr=0.3)
    ora, _ = oracle_scan.trans_lmm(codes.astype(float), Y, X, Q, lam, 0.0, deltas=delta)
    _check(pairs, cands, ora["stats"], 0.999, 0.3, 1e-6)


def test_glm_pieces():
    from eqtl_b200 import capi, synth
    n, m, G, p = 150, 1900, 100, 20
    rng = np.random.default_rng(2)
    codes = _codes(rng, m, n)
    X = np.column_stack([np.ones(n), 0.2 * rng.standard_normal((n, p - 1))])
    Y = rng.poisson(np.exp(2.0 + 0.3 * X[:, 1:4].sum(1, keepdims=True)) * rng.gamma(4.0, 0.25, (n, G))).astype(float)
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        genes, pairs, cands, phi, conv = c.scan_glm(Y, X, pthr=0.999, perm_thr=0.3)
    ora, _ = oracle_scan.glm(codes.astype(float), Y, X, 0.0)
    assert conv.all()
    _check(pairs, cands, ora["stats"], 0.999, 0.3, 1e-6)


def test_result_pieces():
    from eqtl_b200 import capi, synth
    n, m, G = 40, 1200, 900  # 1,080,000 pairs and as many candidates
    rng = np.random.default_rng(3)
    codes, X, Y = _codes(rng, m, n), np.ones((n, 1)), rng.standard_normal((n, G))
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        genes, pairs, cands = c.scan_trans_lm(Y, X, pthr=1.0, perm_thr=2.0)
    ora, _ = oracle_scan.trans_lm(codes.astype(float), Y, X, 0.0)
    _check(pairs, cands, ora["stats"], 1.0, 2.0, 1e-9)


def test_memory_of_a_long_list():
    import torch
    from eqtl_b200 import capi, synth
    n, m, G, p = 64, 4000, 500, 32
    rng = np.random.default_rng(4)
    codes, Y = _codes(rng, m, n), rng.standard_normal((n, G))
    X = np.column_stack([np.ones(n), rng.standard_normal((n, p - 1))])
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        c.set_basis(Q, np.linspace(0.0, 2.0, n))
        c.scan_trans_lmm(Y, X, pthr=1e-3)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        _, pairs, _, _ = c.scan_trans_lmm(Y, X, pthr=0.999)
        used = before - torch.cuda.mem_get_info()[0]
    k = m * G
    assert len(pairs) > 0.99 * k
    # 56 bytes refined, 60 of candidates, keys and lists; two pieces; 34 sums would be 272 more
    assert used < 160 * k + (96 << 20)
