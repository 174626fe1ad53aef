"""Neighbour radii where many distances are equal but for rounding: a lattice
whose spacing is no power of two, shells of it, groups of coincident points.
Radii must equal the k-th smallest canonical float distance; the counts of
points make 8, 4, 2 and 1 warps share a leaf."""
import numpy as np
import pytest

from tests.test_gpu_knn_sizes import _d2

pytestmark = pytest.mark.gpu
F = np.float32


def _points(kind, n, rng):
    if kind == "dup":
        return np.repeat(rng.uniform(-0.5, 0.5, ((n + 15) // 16, 3)), 16, 0)[:n].astype(F)
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3), -1).reshape(-1, 3)
    if kind == "shells":                # around one point, everything the same few distances off
        g = g[np.isin(((g - m // 2) ** 2).sum(1), (0, 9, 14, 17, 26, 29))]
        return np.resize((g + 0.5) / m - 0.5, (n, 3)).astype(F)
    return ((rng.permutation(g)[:n] + 0.5) / m - 0.5).astype(F)


@pytest.mark.parametrize("kind", ["lattice", "shells", "dup"])
@pytest.mark.parametrize("n,k", [(1331, 24), (1331, 128), (3000, 100), (12_000, 64), (12_000, 128), (35_937, 128),
                                 (35_937, 27)])
def test_near_ties(gpu_ready, n, k, kind):
    from skid_gb300 import gpu
    rng = np.random.default_rng(n + k)
    pos = _points(kind, n, rng)
    at = rng.choice(n, 400, replace=False)
    for period in (1.0, None):
        with gpu.Context(period=period) as ctx:
            got = ctx.knn_ball2(pos, k)
        want = np.array([np.partition(_d2(pos, i, period), k - 1)[k - 1] for i in at])
        assert np.array_equal(got[at], want), period
