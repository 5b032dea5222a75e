"""The thread-per-query first pass against the warp path alone (mg_knn_set_group_pass):
the same neighbour sets and distances, and h to the solver's noise, in open and
periodic sets of 1 to 3 dimensions, for row lengths up to the pass's limit, query
counts that leave a warp partly filled, scattered query lists (boxes over far
too many particles), clumps at a box edge, and points that coincide."""
import numpy as np
import pytest

from gpu_util import as_np, sets_equal_rows, summary

pytestmark = pytest.mark.gpu

H_RTOL = 1e-9  # both solve h in float-float; the rows' order differs


def _points(kind, n, dim, rng):
    p = rng.random((n, dim))
    if kind == "edge":  # half the points in a clump that straddles the box's corner
        p[n // 2:] = np.mod(1e-2 * rng.standard_normal((n - n // 2, dim)), 1.0)
        p[p >= 1.0] = 0.0
    elif kind == "lattice":
        m = int(round(n ** (1.0 / dim)))
        g = np.arange(m) / m
        p = np.stack(np.meshgrid(*[g] * dim, indexing="ij"), -1).reshape(-1, dim)
    return p


@pytest.mark.parametrize("kind,n,dim,box,k", [
    ("uniform", 33, 3, None, 32), ("uniform", 1000, 3, 1.0, 32), ("uniform", 5001, 3, 1.0, 32),
    ("uniform", 40000, 3, 1.0, 31), ("edge", 20001, 3, 1.0, 32), ("edge", 20001, 3, None, 32),
    ("lattice", 13824, 3, 1.0, 32), ("lattice", 13824, 3, None, 13), ("uniform", 9999, 2, 1.0, 20),
    ("edge", 9999, 2, 1.0, 20), ("uniform", 3001, 1, 1.0, 4), ("uniform", 3001, 1, None, 3),
    ("uniform", 20000, 3, None, 11), ("uniform", 100, 3, 1.0, 16)])
@pytest.mark.parametrize("masked", [False, True])
def test_first_pass_equals_warp_path(kind, n, dim, box, k, masked):
    from meshoid_gb300 import Meshoid, _native

    rng = np.random.default_rng(n + dim)
    p = _points(kind, n, dim, rng)
    mask = rng.random(len(p)) < 0.05 if masked else None
    lib = _native.load()
    prev = lib.mg_knn_set_group_pass(1)
    try:
        A = Meshoid(p, des_ngb=k, boxsize=box, particle_mask=mask)
        lib.mg_knn_set_group_pass(0)
        B = Meshoid(p, des_ngb=k, boxsize=box, particle_mask=mask)
    finally:
        lib.mg_knn_set_group_pass(prev)
    assert sets_equal_rows(as_np(A.ngb), as_np(B.ngb)) == 0
    np.testing.assert_array_equal(as_np(A.ngbdist), as_np(B.ngbdist))
    e = np.abs(as_np(A.kernel_radius) / as_np(B.kernel_radius) - 1)
    assert e.max() <= H_RTOL, summary(e)


def test_coincident_points():
    """More coincident points than neighbours are wanted have no smoothing length;
    few of them do, and both searches find the same sets."""
    from meshoid_gb300 import Meshoid, _native

    rng = np.random.default_rng(5)
    p = rng.random((4000, 3))
    p[1::4] = p[::4]  # pairs of coincident points
    lib = _native.load()
    prev = lib.mg_knn_set_group_pass(1)
    try:
        A = Meshoid(p)
        lib.mg_knn_set_group_pass(0)
        B = Meshoid(p)
    finally:
        lib.mg_knn_set_group_pass(prev)
    assert sets_equal_rows(as_np(A.ngb), as_np(B.ngb)) == 0
    np.testing.assert_array_equal(as_np(A.ngbdist), as_np(B.ngbdist))
