"""The move field at every movers-per-warp setting, at sizes where the copy
tree's depth changes (first level of leaves alone, one stride, two) and the
last leaf and the last warp are partly filled, positions in no order, against
FP64 all pairs (open box, so the copies are the scatterers).  The bar is the
field's own: 1e-5 of the sum of the terms' magnitudes."""
import numpy as np
import pytest

from skid_gb300 import tipsy

pytestmark = pytest.mark.gpu


def _field64(x, m, b, y):
    acc = np.empty((len(y), 3))
    mag = np.empty(len(y))
    ih2 = 4.0 / b
    coef = m * ih2**2.5 / np.pi
    for i in range(len(y)):
        d = x - y[i]
        d2 = (d * d).sum(1)
        q2 = d2 * ih2
        q = np.sqrt(np.maximum(q2, 1e-30))
        f = np.where(q2 < 1, 2.25 * q - 3, 3 - 0.75 * q - 3 / q) * coef * (d2 < b)
        t = f[:, None] * d
        acc[i] = t.sum(0)
        mag[i] = np.linalg.norm(t, axis=1).sum()
    return acc, mag


@pytest.mark.parametrize("n,nm", [(33, 1), (97, 33), (512, 31), (1024, 200), (1025, 65), (5000, 700),
                                  (33000, 257)])
def test_field_sizes_and_groupings(gpu_ready, n, nm):
    from skid_gb300 import gpu
    rng = np.random.default_rng(n + nm)
    pos = (rng.normal(size=(n, 3)) * rng.random((n, 1)) * 0.2).astype(np.float32)
    pos[n // 2:] = rng.uniform(-0.5, 0.5, (n - n // 2, 3)).astype(np.float32)
    mass = rng.uniform(0.5, 1.0, n).astype(np.float32)
    snap = tipsy.Snapshot(1.0, 0, n, 0, pos, np.zeros((n, 3), np.float32), mass,
                          np.zeros(n, np.float32), np.zeros(n, np.float32))
    at = rng.integers(0, n, nm)
    y = (pos[at] + (rng.random((nm, 1)) < 0.9) * rng.normal(size=(nm, 3)) * 0.01).astype(np.float32)
    with gpu.Context(period=None, nSmooth=32) as ctx:
        ctx.set_particles(snap)
        ctx.scatter_active()
        ctx.density()
        _, b = ctx.get_density()
        got = {}
        for g in (0, 1, 4, 8, 16, 32, 64):
            ctx.set_option("field_movers_per_warp", g)
            got[g] = ctx.field(y)
    want, mag = _field64(pos.astype(float), mass.astype(float), b.astype(float), y.astype(float))
    for g, a in got.items():
        assert np.all(np.linalg.norm(a - want, axis=1) <= 1e-5 * mag + 1e-30), g
    assert np.array_equal(got[0], got[32]) and np.array_equal(got[64], got[32])
