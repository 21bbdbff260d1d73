"""GPU: scans of a panel whose SNPs are all filtered out, in a context that has
scanned another panel and in a new one: no gene tests anything, and nothing of the
earlier scan comes back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, M, G = 60, 700, 300


def _scans(c, Y, counts, X, windows):
    q, _ = np.linalg.qr(np.random.default_rng(5).standard_normal((N, N)))
    c.set_basis(q, np.linspace(0.0, 2.0, N))
    for w in (None, windows):
        for p in (1, 3):
            yield c.scan_trans_lm(Y, X[:, :p], pthr=0.5, perm_thr=0.5, windows=w)
            yield c.scan_trans_lmm(Y, X[:, :p], pthr=0.5, perm_thr=0.5, windows=w)[:3]
            yield c.scan_glm(counts, X[:, :p], pthr=0.5, perm_thr=0.5, windows=w)[:3]


@pytest.mark.parametrize("used", [False, True])
def test_every_snp_filtered_out(used):
    from eqtl_b200 import capi, synth
    rng = np.random.default_rng(3)
    codes = rng.binomial(2, rng.uniform(0.1, 0.9, (M, 1)), (M, N)).astype(np.int8)
    rows = synth.pack_bed_rows(codes)
    X = np.column_stack([np.ones(N), rng.standard_normal((N, 2))])
    Y = rng.standard_normal((N, G))
    counts = rng.negative_binomial(5, 0.1, (N, G)).astype(float)
    gene = [rng.integers(0, 2, G).astype(np.int32), np.zeros(G, np.int64), np.full(G, 1 << 30, np.int64)]
    with capi.Context(0) as c:
        if used:
            c.load_bed(rows, N, np.arange(N))
            snp = [np.sort(rng.integers(0, 2, M)).astype(np.int32), np.arange(M, dtype=np.int64)]
            for genes, pairs, cands in _scans(c, Y, counts, X, (*gene, *snp, 2)):
                assert genes["n_tested"].any() and len(pairs) and len(cands)
        c.load_bed(rows, N, np.arange(N), maf_min=0.6)  # no allele is that common
        assert c.n_kept == 0
        snp = [np.zeros(0, np.int32), np.zeros(0, np.int64)]
        for genes, pairs, cands in _scans(c, Y, counts, X, (*gene, *snp, 2)):
            assert (genes["n_tested"] == 0).all() and (genes["acat_used"] == 0).all()
            assert (genes["acat_tan_sum"] == 0).all()
            assert (genes["best_snp"] == -1).all() and (genes["best_p"] == 2).all()
            assert len(pairs) == 0 and len(cands) == 0
