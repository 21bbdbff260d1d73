"""CPU checks of the binding's result lists, on a stand-in for the library's scan that
reports a number of pairs: how much room it offers, what its results keep."""
import numpy as np
import pytest

from eqtl_b200 import capi

N, M, G = 20, 200_000, 5_000


class Scan:
    """Finds `found` pairs of G genes; keeps the room that it was offered."""

    def __init__(self, found):
        self.found, self.offered = found, []

    def __call__(self, h, prm, Y, X, genes, pairs, cap_p, n_pairs, cands, cap_c, n_cands):
        self.offered.append((cap_p, cap_c))
        n_pairs._obj.value, n_cands._obj.value = self.found, 0
        return -7 if self.found > cap_p else 0


def _context():
    c = object.__new__(capi.Context)
    c.lib, c.h, c.n_kept, c.n = None, None, M, N
    return c


def _run(scan, thr, windows=None, perm_thr=0.0):
    X = np.ones((N, 1))
    return _context()._scan(scan, np.zeros((N, G)), X, thr, perm_thr, windows)


def _held(a):
    return (a if a.base is None else a.base).nbytes


@pytest.mark.parametrize("found", [0, 3, 70_000])
def test_results_hold_their_entries(found):
    genes, pairs, cands = _run(Scan(found), 1e-3, perm_thr=1e-3)
    assert len(genes) == G and len(pairs) == found and len(cands) == 0
    assert pairs.dtype == capi.PAIR_DTYPE
    assert _held(pairs) == pairs.nbytes and _held(cands) == 0


def test_room_offered():
    scan = Scan(0)
    for thr in (0.0, 1e-6, 0.05, 2.0):
        _run(scan, thr, perm_thr=thr / 2)
    room = [(1 << 16) + min(int(3 * M * G * t), 1 << 24) for t in (0.0, 5e-7, 1e-6, 0.025, 0.05, 1.0)]
    assert scan.offered == [(room[0], room[0]), (room[2], room[1]), (room[4], room[3]), (room[5], room[5])]


def test_limited_address_space(monkeypatch):
    empty = np.empty

    def limited(shape, *a, **k):
        if np.prod(shape) > 1 << 22:
            raise MemoryError
        return empty(shape, *a, **k)

    scan = Scan(100_000)
    monkeypatch.setattr(capi.np, "empty", limited)
    _, pairs, _ = _run(scan, 0.05)
    assert len(pairs) == 100_000 and scan.offered == [(1 << 16, 1 << 16), (100_000, 1 << 16)]
    scan.found = 1 << 23
    with pytest.raises(MemoryError):
        _run(scan, 0.05)


def test_nan_threshold():
    """Nothing is below it; it is the library's to accept."""
    scan = Scan(0)
    genes, pairs, cands = _run(scan, float("nan"), perm_thr=float("nan"))
    assert len(genes) == G and len(pairs) == 0 and scan.offered == [(1 << 16, 1 << 16)]
