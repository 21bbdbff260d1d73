"""GPU parity of scans and rotations whose 128-row tiles run in pairs on two
SMs: gene and sample counts around the tile, the pair and the rule that picks
them, with a last pair whose second half is partly or wholly past the rows."""
import numpy as np
import pytest

import oracle_scan
import restate as R
from gpu_util import check_scan

pytestmark = pytest.mark.gpu


def _codes(rng, m, n):
    c = rng.binomial(2, rng.uniform(0.1, 0.9, (m, 1)), (m, n)).astype(np.int8)
    c[:, :3] = [0, 1, 2]
    return c


@pytest.mark.parametrize("G", [127, 128, 129, 255, 256, 257, 385, 769, 897])
@pytest.mark.parametrize("m,dense", [(255, False), (513, True)])
def test_lm_gene_tiles(G, m, dense):
    from eqtl_b200 import capi, synth
    n = 70
    rng = np.random.default_rng(G + m)
    codes = _codes(rng, m, n)
    Y, X = rng.standard_normal((n, G)), np.column_stack([np.ones(n), rng.standard_normal(n)])
    Y[:, G - 1] += 2.0 * codes[m - 1]
    with capi.Context(0) as c:
        if dense:
            c.load_dosage(codes.astype(np.float32), np.arange(n))
        else:
            c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        res = c.scan_trans_lm(Y, X, pthr=1e-3)
    ora, ref = oracle_scan.trans_lm(codes.astype(float), Y, X, 1e-3)
    check_scan(res, ora, ref, 1e-3, n - 3)


@pytest.mark.parametrize("n", [130, 200, 257, 300])
def test_rotation_sample_tiles(n):
    """The LMM's statistics screen on the rotated operands: two, two (ragged),
    three and three row tiles of eigenvectors."""
    from eqtl_b200 import capi, synth
    m, G = 140, 9
    rng = np.random.default_rng(n)
    codes = _codes(rng, m, n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    lam = np.sort(rng.gamma(0.5, 2.0, n))
    X = np.ones((n, 1))
    Y = (Q * np.sqrt(lam + 1.0)) @ rng.standard_normal((n, G))
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        c.set_basis(Q, lam)
        res = c.scan_trans_lmm(Y, X, pthr=1e-2)
    ora, ref = oracle_scan.trans_lmm(codes.astype(float), Y, X, Q, lam, 1e-2, deltas=res[3])
    check_scan(res[:3], ora, ref, 1e-2, n - 2, rel=1e-6)
