"""Tree boxes where the upward pass changes form -- one leaf, fewer than 32, one
block of 32, two levels of blocks, a ragged last block -- seen through what is
found with them: neighbour radii must equal the k-th smallest canonical float
distance, friends-of-friends at a length that links everything must find one
group, and the ball boxes must find every copy that reaches a position (an FP64
sum, to 1e-5 of the terms' norms, the bound of the other field comparisons)."""
import numpy as np
import pytest

from oracle import oracle
from skid_gb300 import tipsy

pytestmark = pytest.mark.gpu
F = np.float32


def _points(n, rng):
    pos = rng.uniform(-0.5, 0.5, (n, 3))
    pos[: n // 2] = 0.3 + 0.05 * rng.normal(size=(n // 2, 3)) * rng.random((n // 2, 1))
    return rng.permutation(np.clip(pos, -0.5, 0.49999997)).astype(F)


@pytest.mark.parametrize("n", [9, 32, 33, 64, 65, 992, 1023, 1024, 1025, 2049, 32768, 32769, 33793])
def test_radii_and_groups(gpu_ready, n):
    from skid_gb300 import gpu
    rng = np.random.default_rng(n)
    pos = _points(n, rng)
    rows = np.arange(n) if n < 3000 else rng.choice(n, 1000, replace=False)
    with gpu.Context() as ctx:
        got = ctx.knn_ball2(pos, 8)
        grp, ng = ctx.fof_points(pos, 2.0)
    d = [(pos[rows, None, c] - pos[None, :, c]).astype(F) for c in range(3)]
    d2 = ((d[0] * d[0] + d[1] * d[1]).astype(F) + d[2] * d[2]).astype(F)
    assert np.array_equal(got[rows], np.partition(d2, 7, axis=1)[:, 7])
    assert ng == 1 and (grp == 1).all()


@pytest.mark.parametrize("n", [40, 1024, 1025, 20000])
def test_field_from_ball_boxes(gpu_ready, n):
    from skid_gb300 import gpu
    rng = np.random.default_rng(n)
    pos = _points(n, rng)
    zero = np.zeros(n, F)
    snap = tipsy.Snapshot(1.0, 0, n, 0, pos, np.zeros((n, 3), F), np.full(n, 1.0 / n, F), zero + F(1e-3), zero)
    y = pos[rng.choice(n, min(n, 300), replace=False)]
    with gpu.Context(period=1.0, nSmooth=16) as ctx:
        ctx.set_particles(snap)
        ctx.scatter_active(False, False)
        ctx.density()
        _, b2 = ctx.get_density()
        got = ctx.field(y)
    alive = oracle.replica_mask(pos, b2, 1.0)
    want, absterm, _ = oracle.field(snap.pos, snap.mass, b2, alive, y, 1.0)
    assert (np.linalg.norm(got - want, axis=1) <= 1e-5 * np.maximum(np.ravel(absterm), 1e-300)).all()
