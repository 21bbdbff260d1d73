"""GPU parity of the refinement's Q'g: exact on the tensor cores from 10 * 2^30
n^2 u on, at sample counts around its digit rows (three eigenvectors to 16 rows,
256 rows to a tile), with and without missing calls, for two bases in turn and on
a sample view; by DGEMM below that and for FP32 dosages."""
import numpy as np
import pytest

import restate as R

pytestmark = pytest.mark.gpu


def _check(c, n, dos, Q, lam, seed):
    """beta and t of every SNP against the oracle at the device's delta. The sums
    are exact up to FP64 rounding; 1e-10 leaves room for the cancellation in
    S = gg - a'A00^-1 a."""
    rng = np.random.default_rng(seed)
    X = np.column_stack([np.ones(n), rng.standard_normal(n)])
    Y = rng.standard_normal((n, 1))
    m = dos.shape[0]
    out, delta = c.test_pairs("lmm", Y, X, np.zeros(m, np.int32), np.arange(m))
    st = R.test_lmm_many(R.prep_lmm(Y[:, 0], X, Q, lam, delta=delta[0]), dos)
    np.testing.assert_allclose(out["beta"], st["beta"], rtol=1e-10, atol=1e-10 * np.abs(st["beta"]).mean())
    np.testing.assert_allclose(out["t"], st["stat"], rtol=1e-10, atol=1e-10)


def _basis(rng, n):
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    Q[np.abs(Q) < 1e-3] *= 1e-9  # entries far below their eigenvector's largest
    Q, _ = np.linalg.qr(Q)
    return Q, np.sort(rng.gamma(0.5, 2.0, n))


@pytest.mark.parametrize("n,m", [(40, 1), (97, 513), (1199, 7520), (1200, 7681), (1201, 7700)])
@pytest.mark.parametrize("miss", [0.0, 0.02])
def test_qg(n, m, miss):
    from eqtl_b200 import capi, synth
    rng = np.random.default_rng(n + m)
    n_file = n + 3
    codes = rng.binomial(2, rng.uniform(0.1, 0.9, (m, 1)), (m, n_file)).astype(np.int8)
    codes[rng.random((m, n_file)) < miss] = -1
    codes[:, :6] = [0, 1, 2, 0, 1, 2]
    cols = np.concatenate([rng.permutation(6), 6 + rng.permutation(n_file - 6)])[:n].astype(np.int32)
    Q, lam = _basis(rng, n)
    rows = synth.pack_bed_rows(codes)
    with capi.Context(0) as c:
        c.load_bed(rows, n_file, cols)
        assert c.n_kept == m
        c.set_basis(Q, lam)
        _check(c, n, R.decode_bed_rows(rows, n_file, cols, "impute", 0.8, 0.0).dosage, Q, lam, n)
        # another basis, then a view of the samples: nothing of the first is kept
        Q2, lam2 = _basis(rng, n)
        c.set_basis(Q2, lam2)
        dos = R.decode_bed_rows(rows, n_file, cols, "impute", 0.8, 0.0).dosage
        _check(c, n, dos, Q2, lam2, n + 1)
        keep = np.sort(np.concatenate([np.arange(6), 6 + rng.permutation(n - 6)[:n - 9]])).astype(np.int32)
        assert n < 1000 or (n - 3) ** 2 * m >= 10 << 30
        c.geno_subset(keep)
        Q3, lam3 = _basis(rng, keep.size)
        c.set_basis(Q3, lam3)
        _check(c, keep.size, dos[:, keep], Q3, lam3, n + 2)


def test_dosage_rows_keep_the_dgemm():
    from eqtl_b200 import capi
    rng = np.random.default_rng(3)
    n, m = 70, 40
    ds = np.round(rng.uniform(0, 2, (m, n)), 3).astype(np.float32)
    Q, lam = _basis(rng, n)
    with capi.Context(0) as c:
        c.load_dosage(ds, np.arange(n))
        c.set_basis(Q, lam)
        _check(c, n, ds.astype(np.float64), Q, lam, 5)
