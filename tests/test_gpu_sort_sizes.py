"""Keys sorted at the edges of the sort's tiles (1024 and 4096 keys) and where
the tile size changes (two tiles of 1024 an SM): the tree over the sorted
points must hold every point once, so the nearest neighbours of all of them
are those a k-d tree in FP64 finds.  A float distance^2 carries at most five
roundings of 2^-24 (difference, square, two sums)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1023, 1024, 1025, 4097, 311295, 311296, 311297, 315393])
def test_radii_across_tile_sizes(gpu_ready, n):
    from scipy.spatial import cKDTree

    from skid_gb300 import gpu
    rng = np.random.default_rng(n)
    pos = rng.uniform(-0.5, 0.5, (n, 3))
    pos[: n // 2] *= 0.1 * rng.random((n // 2, 1))
    pos = rng.permutation(pos).astype(np.float32)
    with gpu.Context() as ctx:
        got = ctx.knn_ball2(pos, 8)
    want = cKDTree(pos.astype(np.float64)).query(pos.astype(np.float64), k=8, workers=-1)[0][:, -1] ** 2
    np.testing.assert_allclose(got, want, rtol=5.5 * 2.0**-24, atol=0)
