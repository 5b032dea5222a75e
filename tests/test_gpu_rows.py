"""Sorted neighbour rows (mg_neighbor_lists): each row ordered by FP64 distance
with ties by particle index, for every row length that changes the sorting
network (one, two or four elements per lane) and its padding, full and masked."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2, 16, 31, 32, 33, 63, 64, 65, 100, 128])
@pytest.mark.parametrize("masked", [False, True])
def test_rows_sorted_by_distance_then_index(k, masked):
    from meshoid_gb300 import Meshoid

    # lattice points: most distances tie, so the order within a row is decided
    # by the particle index
    g = np.arange(8) / 8.0
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    pos = pos[np.random.default_rng(k).permutation(len(pos))]
    mask = np.zeros(len(pos), bool)
    mask[::7] = True
    rows = np.nonzero(mask)[0] if masked else np.arange(len(pos))
    M = Meshoid(pos, des_ngb=k, particle_mask=mask if masked else None)
    ngb, dist = M.ngb.cpu().numpy(), M.ngbdist.cpu().numpy()
    d = pos[None, :, :] - pos[rows][:, None, :]
    d2 = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]
    ref = np.lexsort((np.broadcast_to(np.arange(len(pos)), d2.shape), d2), axis=1)[:, :k]
    assert np.array_equal(ngb, ref)
    assert np.array_equal(dist, np.sqrt(np.take_along_axis(d2, ref, 1)))
    assert torch.equal(M.NearestNeighbors(), M.ngb)
