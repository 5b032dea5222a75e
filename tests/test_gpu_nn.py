"""Nearest particle of arbitrary points (the query behind Reconstruct and
Slice) against all pairs in FP64, ties by particle index: inside and far outside
the particles, on particles, beside a dense clump, in boxes and in 1 to 3
dimensions, and with fewer particles than a warp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _brute(pos, t, box):
    out = np.empty(len(t), np.int64)
    for a in range(0, len(t), 256):
        d = pos[None] - t[a:a + 256, None]
        if box:
            d = np.where(np.abs(d) > 0.5 * box, -np.copysign(box - np.abs(d), d), d)
        d2 = np.zeros(d.shape[:2])
        for c in range(pos.shape[1]):
            d2 = d2 + d[..., c] * d[..., c]
        out[a:a + 256] = np.argmin(d2, axis=1)  # the first of equals
    return out


@pytest.mark.parametrize("n,dim,box,kind", [
    (20, 3, 0, "uniform"), (2000, 3, 0, "uniform"), (6000, 3, 0, "clump"), (6000, 3, 1.0, "clump"),
    (40, 3, 1.0, "uniform"), (1500, 2, 0, "clump"), (700, 2, 1.0, "uniform"), (300, 1, 0, "uniform"),
    (50, 1, 1.0, "uniform"), (512, 3, 0, "lattice"), (512, 3, 1.0, "lattice"), (64, 3, 0, "same")])
def test_nearest_particle_equals_all_pairs(n, dim, box, kind):
    from meshoid_gb300 import Meshoid

    rng = np.random.default_rng(n + dim)
    pos = rng.random((n, dim))
    if kind == "clump":  # nine tenths of the particles in a clump 1e-3 across
        pos[n // 10:] = 0.3 + 1e-3 * rng.random((n - n // 10, dim))
    elif kind == "lattice":
        g = np.arange(8) / 8.0
        pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[rng.permutation(512)]
    elif kind == "same":
        pos = np.full((n, dim), 0.25)
    t = [rng.random((400, dim)), pos[rng.integers(0, n, 100)], 0.3 + 2e-3 * rng.random((100, dim))]
    if kind == "lattice":
        t.append((np.floor(8 * rng.random((200, 3))) + 0.5) / 8.0)  # eight nearest, all equal
    if not box:
        t.append(rng.normal(size=(100, dim)) * 50.0)
    t = np.concatenate(t)
    # h given: only the cell index is built
    M = Meshoid(pos, kernel_radius=np.full(n, 0.1), des_ngb=4, boxsize=box or None)
    got = M._nn(t).cpu().numpy()
    assert np.array_equal(got, _brute(pos, t, box))
