"""Neighbour radii at point counts that one, two, four or eight warps to a leaf
are chosen for: they must equal the k-th smallest canonical float distance."""
import numpy as np
import pytest

from tests.test_gpu_knn_sizes import _d2, _points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["faces", "ties", "clump"])
@pytest.mark.parametrize("n,k", [(257, 24), (5400, 128), (6001, 128), (11000, 32), (12000, 128), (17000, 128),
                                 (15001, 64), (27000, 32), (45000, 24)])
def test_radii(gpu_ready, n, k, kind):
    from skid_gb300 import gpu
    rng = np.random.default_rng(n + k)
    pos = _points(n, kind, rng)
    period = None if kind == "clump" else 1.0
    with gpu.Context(period=period, nSmooth=k) as ctx:
        got = ctx.knn_ball2(pos, k)
    rows = rng.choice(n, min(n, 1500), replace=False)
    want = np.array([np.partition(_d2(pos, i, period), k - 1)[k - 1] for i in rows])
    assert np.array_equal(got[rows], want)
