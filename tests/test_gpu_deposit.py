"""GridDensity where its tile pass changes form: one cube over whole tiles, fewer
overlaps than warps, warps with a partial set of overlaps, cubes of a few nodes, and
tiles with more overlaps than one work item takes, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,res,hdx,spread,box", [
    (1, 8, 20.0, 1.0, False), (3, 9, 3.0, 1.0, False), (33, 17, 2.0, 1.0, False), (300, 16, 6.0, 1.0, False),
    (2000, 40, 1.1, 1.0, False), (9001, 12, 1.3, 0.3, False), (9001, 12, 1.3, 0.3, True), (300, 16, 3.0, 1.0, True),
])
def test_tiles(n, res, hdx, spread, box):
    from meshoid_gb300 import grid_deposition as GD
    from oracle import oracle as O

    rng = np.random.default_rng(n + res)
    dx = 1.0 / (res - 1)
    p = 0.5 + spread * (rng.random((n, 3)) - 0.5)
    h = hdx * dx * (1.0 + rng.random(n))
    f = 0.5 + rng.random(n)
    c = np.full(3, 0.5)
    b = 1.0 if box else -1.0
    ref = O.grid_density(f, p, h, c, 1.0, res, b)
    got = GD.GridDensity(f, p, h, c, 1.0, res=res, box_size=b)
    got = got.cpu().numpy() if hasattr(got, "cpu") else np.asarray(got)
    # an item adds up to 4096 values in FP32; 64 roundings for a weight and its sum
    tol = (min(n, 4096) + 64) * 2.0 ** -24
    assert np.max(np.abs(got - ref)) <= tol * np.abs(ref).max()
