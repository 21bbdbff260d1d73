"""GPU: a scan's result lists at the sizes where their making changes: one block's
sort (up to 4096 keys), the radix sort, several of its blocks, a gene with more
candidates than are ranked on the device. With pthr = 1 every
tested pair is a candidate, so the lists have exactly genes x SNPs entries."""
import numpy as np
import pytest

import oracle_scan
from gpu_util import check_scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,m", [(1, 3), (8, 511), (8, 512), (17, 241), (40, 700), (300, 301), (2, 9000)])
def test_result_lists(G, m):
    from eqtl_b200 import capi, synth
    n = 40
    rng = np.random.default_rng(G + m)
    codes = rng.binomial(2, rng.uniform(0.1, 0.9, (m, 1)), (m, n)).astype(np.int8)
    codes[:, :3] = [0, 1, 2]
    codes[m // 2] = codes[0]  # equal p in every gene: the best is the lower SNP
    X, Y = np.ones((n, 1)), rng.standard_normal((n, G))
    Y[:, 0] += 3.0 * codes[0]
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        genes, pairs, cands = c.scan_trans_lm(Y, X, pthr=1.0, perm_thr=0.25)
    ora, ref = oracle_scan.trans_lm(codes.astype(float), Y, X, 1.0)
    check_scan((genes, pairs, cands), ora, ref, 1.0, n - 2)
    assert len(pairs) == G * m
    order = pairs["snp"] * G + pairs["gene"]
    assert (np.diff(order) > 0).all()
    for g in (0, G - 1):
        q = pairs[pairs["gene"] == g]
        b = np.lexsort((q["snp"], q["p"]))[0]
        assert genes["best_snp"][g] == q["snp"][b] and genes["best_p"][g] == q["p"][b]
    want = pairs[pairs["p"] < 0.25]
    want = want[np.lexsort((want["snp"], want["p"], want["gene"]))]
    assert np.array_equal(cands, want)
