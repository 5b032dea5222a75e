"""The order-1 derivative sweep at the shapes where its split of components and
neighbours over a query's four lanes changes: 1 to 21 components (one, two, and
four groups of four at a time, with a partial last group), neighbour counts that
are and are not multiples of 4 and 16, query counts that leave a block partly
filled, 1 to 3 dimensions and a box, against the oracle.

Tolerance: 1e-5 of the row norm, the contract of the first derivatives, on the
rows that have a reproducible answer: with small k some rows hold fewer particles
inside the kernel than the dim + 1 of a fit, where the reference raises and the
GPU returns the minimum-norm solution, and others are so nearly singular that the
FP64 answer itself moves by more than a quarter of the tolerance when h is scaled
by 1 + 1e-12."""
import numpy as np
import pytest

from gpu_util import as_np, row_rel_err, summary

pytestmark = pytest.mark.gpu


def _field(p, nf, seed):
    rng = np.random.default_rng(seed)
    k = rng.normal(size=(p.shape[1], nf))
    return np.sin(p @ k + rng.uniform(0, 6, nf)) + 0.1 * (p @ rng.normal(size=(p.shape[1], nf)))


def _reference(p, k, box, f):
    """The oracle's D, and the rows that have a reproducible answer."""
    from oracle import oracle as O

    R = O.OracleMeshoid(p, des_ngb=k, boxsize=box)
    ref = R.D(f)
    full = (R.ngbdist < R.kernel_radius[:, None]).sum(1) > p.shape[1]
    R.kernel_radius = R.kernel_radius * (1 + 1e-12)
    R.reset_dweights()
    return ref, full & (row_rel_err(R.D(f), ref) <= 2.5e-6)


@pytest.mark.parametrize("nf", [1, 3, 4, 5, 8, 9, 12, 13, 16, 17, 19, 20, 21])
def test_components(nf):
    from meshoid_gb300 import Meshoid
    from oracle import oracle as O

    p = np.random.default_rng(nf).random((1003, 3))
    f = _field(p, nf, nf)
    got, ref = as_np(Meshoid(p).D(f)), O.OracleMeshoid(p).D(f)
    for c in range(nf):
        e = row_rel_err(got[:, c], ref[:, c])
        assert e.max() <= 1e-5, (c, summary(e))


@pytest.mark.parametrize("n,dim,k,box,nf", [
    (33, 3, 32, None, 5), (95, 3, 30, None, 17), (400, 3, 17, None, 3), (400, 3, 12, 1.0, 8), (700, 3, 100, None, 6),
    (500, 3, 128, 1.0, 4), (300, 2, 20, None, 7), (300, 2, 21, 1.0, 16), (120, 1, 6, None, 5), (64, 1, 8, 1.0, 2)])
def test_shapes(n, dim, k, box, nf):
    from meshoid_gb300 import Meshoid

    p = np.random.default_rng(n).random((n, dim))
    if box:
        f = np.stack([np.sin(2 * np.pi * p[:, c % dim] + c) for c in range(nf)], 1)
    else:
        f = _field(p, nf, n)
    ref, sure = _reference(p, k, box, f)
    assert sure.mean() > 0.2
    e = row_rel_err(as_np(Meshoid(p, des_ngb=k, boxsize=box).D(f)), ref)[sure]
    assert e.max() <= 1e-5, summary(e)
    mask = np.arange(n) % 3 == 0  # a query list
    e = row_rel_err(as_np(Meshoid(p, des_ngb=k, boxsize=box, particle_mask=mask).D(f)), ref[mask])[sure[mask]]
    assert e.max() <= 1e-5, summary(e)
