"""GPU: a cis scan's tile list and block bounds made on the device: SNP counts
around the block and the tile, SNPs in genome order, a chromosome in two runs,
positions that decrease, genes without a location, on an absent chromosome, with
an empty window or a window past the ends."""
import numpy as np
import pytest

import oracle_scan
from gpu_util import check_scan

pytestmark = pytest.mark.gpu


def _layout(kind, m, rng):
    chrom = np.sort(rng.integers(0, 5, m)).astype(np.int32)
    pos = rng.integers(1, 100_000, m)
    pos = pos[np.lexsort((pos, chrom))]
    if kind == "split" and m > 2:
        chrom[-1] = chrom[0]
    if kind == "decreasing" and m > 2:
        chrom[:] = 1
        pos = np.sort(pos)[::-1].copy()
    return chrom, pos


@pytest.mark.parametrize("m,G", [(1, 1), (16, 3), (255, 130), (257, 129), (1500, 260)])
@pytest.mark.parametrize("kind", ["sorted", "split", "decreasing"])
def test_cis_tiles(m, G, kind):
    from eqtl_b200 import capi, synth
    n = 40
    rng = np.random.default_rng(m + G)
    codes = rng.binomial(2, rng.uniform(0.1, 0.9, (m, 1)), (m, n)).astype(np.int8)
    codes[:, :3] = [0, 1, 2]
    chrom, pos = _layout(kind, m, rng)
    gchrom = rng.integers(-1, 6, G).astype(np.int32)
    lo = rng.integers(-20_000, 100_000, G)
    hi = lo + rng.integers(-10, 30_000, G)
    gchrom[0], lo[0], hi[0] = chrom[0], -(1 << 40), 1 << 40
    X, Y = np.ones((n, 1)), rng.standard_normal((n, G))
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        res = c.scan_trans_lm(Y, X, pthr=1e-1, windows=(gchrom, lo, hi, chrom, pos, 2))
    excl = ~oracle_scan.windows_mask(chrom, pos, gchrom, lo, hi)
    ora, ref = oracle_scan.trans_lm(codes.astype(float), Y, X, 1e-1, excl=excl)
    check_scan(res, ora, ref, 1e-1, n - 2)
