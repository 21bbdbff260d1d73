"""GPU: the device memory of table preparations (rank transform, PEER) is given back to
the calls that follow, and above 1 GiB, or after a failed call, at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLACK = 64 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _prepare(c, n, G, K):
    rng = np.random.default_rng(1)
    Y = c.pheno_int(rng.standard_normal((n, G)))
    c.peer(Y, K, 1, 1e-3, rng.standard_normal((n, K)), rng.standard_normal((G, K)))


def test_given_back():
    from eqtl_b200 import capi
    with capi.Context(0) as c:
        _prepare(c, 60, 100, 2)  # the libraries' own memory
        c.pheno_load(np.ones((10, 2)), np.ones((10, 1)))
        before = _free()
        _prepare(c, 60, 20_000, 40)  # 256 MB of second moments
        c.launch_count()  # a query does not touch them
        _prepare(c, 60, 20_000, 40)
        c.pheno_load(np.ones((10, 2)), np.ones((10, 1)))
        assert _free() > before - SLACK
        _prepare(c, 97, 16_000, 96)  # 1.2 GB
        assert _free() > before - SLACK


def test_given_back_after_an_error():
    from eqtl_b200 import capi
    with capi.Context(0) as c:
        _prepare(c, 60, 100, 2)
        c.pheno_load(np.ones((10, 2)), np.ones((10, 1)))
        before = _free()
        _prepare(c, 60, 20_000, 40)
        with pytest.raises(capi.EqtlError):
            _prepare(c, 60, 200, 60)  # as many factors as samples
        assert _free() > before - SLACK
