"""GPU parity of the kernels that sort a column per block (permutation draws and
the rank transform): column lengths at the edges of the block sizes, and past
4096, where the segmented sort takes over."""
import os
import sys

import numpy as np
import pytest

import driver

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import philox  # noqa: E402

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 127, 128, 129, 256, 257, 512, 513, 1024, 1025, 2048, 2049, 4095, 4096, 4097]


@pytest.fixture(scope="module")
def ctx():
    from eqtl_b200 import capi
    with capi.Context(0) as c:
        yield c


@pytest.mark.parametrize("n", SIZES)
def test_permuted_columns(ctx, n):
    rng = np.random.default_rng(n)
    base, keys = rng.normal(size=(n, 2)), [philox.fnv1a64("A"), philox.fnv1a64("B")]
    got = ctx.pheno_permute(base, np.ones((n, 1)), np.array(keys, np.uint64), 3, 11, out=True)
    np.testing.assert_array_equal(got, philox.permuted_columns(base, [int(k) for k in keys], 3, 11, None, None))


@pytest.mark.parametrize("n", [1] + SIZES)
def test_rank_transform(ctx, n):
    rng = np.random.default_rng(n)
    Y = np.column_stack([rng.standard_normal(n), rng.poisson(2.0, n), rng.standard_normal(n),
                         np.where(rng.random(n) < 0.5, -0.0, 0.0), np.full(n, -1e300),
                         rng.choice([-1.5, 5e-324, -5e-324, 1e308], n)]).astype(np.float64)
    Y[rng.random(n) < 0.2, 2] = np.nan
    Y[0, 2], Y[n - 1, 2] = np.inf, -np.inf
    got = ctx.pheno_int(Y)
    for j in range(Y.shape[1]):
        fin = np.isfinite(Y[:, j])
        ref = driver.inverse_normal_transform(Y[:, j])
        np.testing.assert_array_equal(got[~fin, j], Y[~fin, j])
        np.testing.assert_allclose(got[fin, j], ref[fin], rtol=1e-13, atol=1e-15)
