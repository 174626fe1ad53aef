"""Neighbour radii and densities where the neighbour kernels change form: the k
at which buffers take over from heaps (24, 128), trees of one leaf, a ragged
last leaf, one stride of leaves and two, points at the periodic faces, many
equal distances (buffers that cannot be cut to size), far outliers.  Radii must
equal the k-th smallest canonical float distance, densities an FP64 sum over
all pairs to 1e-5."""
import numpy as np
import pytest

from skid_gb300 import tipsy

pytestmark = pytest.mark.gpu
F = np.float32


def _points(n, kind, rng):
    if kind == "faces":
        p = rng.uniform(-0.5, 0.5, (n, 3))
        p[:, 0] = np.where(rng.random(n) < 0.7, np.sign(p[:, 0]) * (0.5 - 0.02 * rng.random(n)), p[:, 0])
        return np.clip(p, -0.5, 0.49999997).astype(F)
    if kind == "ties":
        return (rng.integers(-3, 4, (n, 3)) * 0.0625).astype(F)
    p = rng.normal(size=(n, 3)) * 0.02 * rng.random((n, 1)) ** 2
    p[: n // 4] = rng.uniform(-0.5, 0.5, (n // 4, 3))
    return rng.permutation(p).astype(F)


def _d2(pos, i, period):
    d = []
    for c in range(3):
        x = pos[i, c] - pos[:, c]
        if period:
            L, h = F(period), F(0.5 * period)
            x = np.where(x > h, (pos[i, c] - L) - pos[:, c], np.where(x < -h, (pos[i, c] + L) - pos[:, c], x))
        d.append(x.astype(F))
    return ((d[0] * d[0] + d[1] * d[1]).astype(F) + d[2] * d[2]).astype(F)


@pytest.mark.parametrize("kind", ["faces", "ties", "clump"])
@pytest.mark.parametrize("n,k", [(24, 24), (33, 23), (33, 32), (129, 128), (130, 129), (1025, 24),
                                 (1500, 64), (3001, 127), (3001, 128)])
def test_radii_and_density_at_edges(gpu_ready, n, k, kind):
    from skid_gb300 import gpu
    rng = np.random.default_rng(n * 1000 + k)
    pos = _points(n, kind, rng)
    mass = rng.uniform(0.5, 1.0, n).astype(F)
    period = None if kind == "clump" else 1.0
    want = np.array([np.partition(_d2(pos, i, period), k - 1)[k - 1] for i in range(n)])
    snap = tipsy.Snapshot(1.0, 0, n, 0, pos, np.zeros((n, 3), F), mass, np.zeros(n, F), np.zeros(n, F))
    with gpu.Context(period=period, nSmooth=k) as ctx:
        assert np.array_equal(ctx.knn_ball2(pos, k), want)
        if kind == "ties":
            return          # a ball of radius 0 has no density
        ctx.set_particles(snap)
        ctx.scatter_active()
        ctx.density()
        rho, b = ctx.get_density()
    assert np.array_equal(b, want)
    b64 = b.astype(float)
    ref = np.zeros(n)
    for i in range(n):
        d2 = _d2(pos, i, period)
        m = d2 < b[i]
        q = np.sqrt(4.0 * d2[m].astype(float) / b64[i])
        w = np.where(q < 1, 1 - 0.75 * (2 - q) * q * q, 0.25 * (2 - q) ** 3)
        w *= 0.5 / np.pi * (4.0 / b64[i]) ** 1.5
        ref[i] += (mass[m] * w).sum()
        ref[m] += mass[i] * w
    assert np.all(np.abs(rho - ref) <= 1e-5 * ref)
