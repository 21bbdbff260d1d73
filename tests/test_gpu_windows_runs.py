"""GPU: the tile list of a cis scan over many chromosome runs (a draft assembly), around
the 1024 threads that enter them in their table and beyond 16,384: one SNP to a run and
several, chromosome numbers far apart, the SNPs' -1, a chromosome in two runs."""
import numpy as np
import pytest

import oracle_scan
from gpu_util import check_scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("runs,m", [(1, 40), (1023, 1023), (1024, 3000), (1025, 1025), (1500, 4000), (20_000, 20_000),
                                    (17_000, 25_000)])
@pytest.mark.parametrize("kind", ["grouped", "split"])
def test_many_runs(runs, m, kind):
    from eqtl_b200 import capi, synth
    n, G = 40, 60
    rng = np.random.default_rng(runs + m)
    codes = rng.binomial(2, rng.uniform(0.1, 0.9, (m, 1)), (m, n)).astype(np.int8)
    codes[:, :3] = [0, 1, 2]
    number = np.concatenate([[-1], rng.choice(2 ** 31 - 1, runs, replace=False)])[:runs]
    rng.shuffle(number)
    chrom = number[np.sort(np.concatenate([np.arange(runs), rng.integers(0, runs, m - runs)]))].astype(np.int32)
    if kind == "split" and runs > 2:
        chrom[-1] = chrom[0]
    pos = np.empty(m, np.int64)
    edge = np.concatenate([[0], np.nonzero(np.diff(chrom))[0] + 1, [m]])
    for a, b in zip(edge[:-1], edge[1:]):
        pos[a:b] = np.sort(rng.integers(1, 1000, b - a))
    gchrom = rng.choice(np.concatenate([number, [-1, 5, 2 ** 31 - 1]]), G).astype(np.int32)
    lo = rng.integers(1, 600, G)
    hi = lo + 500
    lo[:4], hi[:4] = 0, 2000
    X, Y = np.ones((n, 1)), rng.standard_normal((n, G))
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        res = c.scan_trans_lm(Y, X, pthr=1e-1, windows=(gchrom, lo, hi, chrom, pos, 2))
    excl = ~oracle_scan.windows_mask(chrom, pos, gchrom, lo, hi)
    assert runs == 1 or (~excl).any()  # one run: chromosome -1, which no gene's window is on
    ora, ref = oracle_scan.trans_lm(codes.astype(float), Y, X, 1e-1, excl=excl)
    check_scan(res, ora, ref, 1e-1, n - 2)
