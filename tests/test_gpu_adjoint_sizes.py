"""The density adjoint from stored neighbour lists against the one that walks
the tree again, on trees of one leaf, with a ragged last leaf, of one 32-leaf
subtree and more, with and without periodic images.  Both take the same pairs in
the same frames with float terms of about 24 roundings, and add the c terms of
a particle in different orders: their difference stays below
2 (c + 24) 2^-24 of the sum of the terms' norms."""
import numpy as np
import pytest

from oracle import oracle
from skid_gb300 import tipsy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("period", [1.0, None])
@pytest.mark.parametrize("n,k", [(25, 24), (33, 8), (64, 63), (1023, 32), (1025, 64), (3000, 17)])
def test_lists_vs_walk(gpu_ready, n, k, period):
    from skid_gb300 import gpu
    rng = np.random.default_rng(n)
    pos = rng.uniform(-0.5, 0.5, (n, 3))
    pos[: n // 2] = 0.49 + 0.05 * rng.normal(size=(n // 2, 3)) * rng.random((n // 2, 1))
    pos -= np.floor(pos + 0.5)
    pos = np.minimum(pos.astype(np.float32), np.float32(0.49999997))
    mass = (rng.uniform(0.5, 1.5, n) / n).astype(np.float32)
    zero = np.zeros(n, np.float32)
    snap = tipsy.Snapshot(1.0, 0, n, 0, pos, np.zeros((n, 3), np.float32), mass, zero + np.float32(1e-3), zero)
    w = rng.standard_normal(n).astype(np.float32)
    _, _, ab = oracle.density_adjoint_check(pos, mass, w, k, period, np.arange(n), h=1e-6)
    with gpu.Context(period=period, nSmooth=k) as ctx:
        ctx.set_particles(snap)
        ctx.scatter_active(False, False)
        ctx.density()
        _, b2 = ctx.get_density()
        lists = ctx.density_adjoint(w, gpu.ADJ_STORED).astype(np.float64)
        walk = ctx.density_adjoint(w, gpu.ADJ_RECOMPUTE).astype(np.float64)
    d = pos[:, None, :].astype(np.float64) - pos[None, :, :]
    if period:
        d -= np.round(d)
    inside = (d * d).sum(-1) <= 1.00001 * b2[:, None].astype(np.float64)
    c = inside.sum(0) + inside.sum(1)
    tol = 2.0 * (c + 24) * 2.0**-24
    assert (np.linalg.norm(lists - walk, axis=1) <= tol * ab).all()
