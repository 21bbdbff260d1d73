"""GPU parity of the grouped LMM scan's gene operands: covariate counts around the
register blocks of their kernel (4, 8, 16, 32), odd and even sample counts."""
import numpy as np
import pytest

import oracle_scan
from gpu_util import check_scan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [5, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("n", [97, 600])
def test_gene_operands(p, n):
    from eqtl_b200 import capi, synth
    m, G = 150, 5
    rng = np.random.default_rng(100 * p + n)
    codes = rng.binomial(2, rng.uniform(0.1, 0.9, (m, 1)), (m, n)).astype(np.int8)
    codes[:, :3] = [0, 1, 2]
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    lam = np.sort(rng.gamma(0.5, 2.0, n))
    X = np.column_stack([np.ones(n), rng.standard_normal((n, p - 1))])
    Y = (Q * np.sqrt(lam + 1.0)) @ rng.standard_normal((n, G))
    with capi.Context(0) as c:
        c.load_bed(synth.pack_bed_rows(codes), n, np.arange(n))
        c.set_basis(Q, lam)
        res = c.scan_trans_lmm(Y, X, pthr=1e-2)
    ora, ref = oracle_scan.trans_lmm(codes.astype(float), Y, X, Q, lam, 1e-2, deltas=res[3])
    check_scan(res[:3], ora, ref, 1e-2, n - p - 1, rel=1e-6)
