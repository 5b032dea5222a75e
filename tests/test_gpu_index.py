"""The cell index at the sizes where its sort and scans change form (one block up
to 8,192 particles, several tiles, many) and with refinement tables several
levels deep: Morton order, the cell table, and every table entry against numpy on
the keys."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BITS = 21


def _check(pos, **kw):
    from meshoid_gb300 import Meshoid

    n = len(pos)
    M = Meshoid(pos, kernel_radius=np.full(n, 0.1), des_ngb=4, **kw)
    keys = M._keys.cpu().numpy().astype(np.uint64)
    order, rank = M._order.cpu().numpy(), M._rank.cpu().numpy()
    assert np.array_equal(np.sort(order), np.arange(n)) and np.array_equal(rank[order], np.arange(n))
    low = 9  # bits the sort leaves alone
    assert np.all(np.diff((keys >> np.uint64(low)).astype(np.int64)) >= 0)
    same = (keys[1:] >> np.uint64(low)) == (keys[:-1] >> np.uint64(low))
    assert np.all(order[1:][same] > order[:-1][same])  # stable
    L = M._cells.grid_level
    start = M._cell_start.cpu().numpy().astype(np.int64)
    cell = (keys >> np.uint64(3 * (BITS - L))).astype(np.int64)
    assert np.array_equal(start, np.searchsorted(cell, np.arange(8 ** L + 1)))
    if M._brick_of is None:
        return 0
    T = M._cells.brick_threshold
    bricks = M._bricks.cpu().numpy().view(np.uint32).astype(np.int64)
    of = M._brick_of.cpu().numpy()
    assert np.array_equal(of >= 0, np.diff(start) > T)
    todo, seen = [(int(of[c]), L, int(start[c]), int(start[c + 1])) for c in np.nonzero(of >= 0)[0]], set()
    while todo:
        b, level, a, e = todo.pop()
        assert b not in seen
        seen.add(b)
        t = bricks[b]
        assert (t[1025], t[1026]) == (a, e)
        sub = (keys[a:e] >> np.uint64(3 * (BITS - level - 3))).astype(np.int64) & 511
        assert np.array_equal(t[:513], a + np.searchsorted(sub, np.arange(513)))
        big = (np.diff(t[:513]) > T) & (level + 6 <= 18)
        child = t[513:1025]
        assert np.array_equal(child != 0xffffffff, big)
        todo += [(int(child[s]), level + 3, int(t[s]), int(t[s + 1])) for s in np.nonzero(big)[0]]
    return len(seen)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1024, 1025, 8191, 8192, 8193, 40000, 300001])
def test_sorted_cells(n):
    rng = np.random.default_rng(n)
    _check(rng.random((n, 3))) if n >= 4 else _check(np.concatenate([rng.random((n, 3))] * 4)[: max(n, 4)])


@pytest.mark.parametrize("n,kw", [(5000, {}), (60000, {}), (200000, {"brick_threshold": 100}),
                                  (60000, {"grid_level": 2}), (60000, {"brick_threshold": 0}),
                                  (60000, {"boxsize": 1.0})])
def test_refinement_tables(n, kw):
    rng = np.random.default_rng(n)
    pos = np.concatenate([rng.random((n // 4, 3)), 0.5 + 1e-3 * rng.standard_normal((n // 2, 3)),
                          0.2 + 1e-5 * rng.standard_normal((n // 4, 3))])
    got = _check(pos[rng.permutation(len(pos))], **kw)
    assert got > 0 or kw.get("brick_threshold") == 0
