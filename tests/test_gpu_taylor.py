"""Reconstruct at order 1 against its definition in FP64 on the derivatives that D
returns: scalar, vector and tensor fields, 1 to 3 dimensions, open and periodic, one
target and several blocks of them, and the path that stays for differentiated
inputs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,box,shape,nt", [(3, None, (), 1), (3, None, (3,), 1000), (3, 1.0, (), 257),
                                              (3, 1.0, (2, 2), 300), (2, None, (5,), 256), (1, None, (), 77)])
def test_reconstruct_order1(dim, box, shape, nt):
    from meshoid_gb300 import Meshoid

    rng = np.random.default_rng(nt)
    pos = rng.random((4000, dim))
    f = rng.random((4000,) + shape)
    x = rng.random((nt, dim))
    M = Meshoid(pos, boxsize=box)
    got = M.Reconstruct(f, x, order=1).cpu().numpy()
    ft = torch.as_tensor(f, device=M.device).requires_grad_(True)
    other = M.Reconstruct(ft, x, order=1).detach().cpu().numpy()
    mask = M.particle_mask.cpu().numpy()
    D = M.D(f).cpu().numpy().astype(np.float64)
    nn = M._nn(x).cpu().numpy()
    d = x - pos[nn]
    if box:
        d -= box * np.round(d / box)
    ref = f[nn] + np.einsum("ij,i...j->i...", d, D[np.searchsorted(mask, nn)])
    # three products and sums in FP64
    tol = 8 * 2.0 ** -53 * (np.abs(ref).max() + np.abs(D).max())
    assert got.shape == (nt,) + shape
    assert np.max(np.abs(got - ref)) <= tol and np.max(np.abs(other - ref)) <= tol
