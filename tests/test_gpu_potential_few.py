"""A potential call launches the same few kernels however small its groups
are, and gives each group what it gives it in any other selection."""
import numpy as np
import pytest

from skid_gb300 import tipsy
from skid_gb300.options import SPLINE

pytestmark = pytest.mark.gpu


def test_small_selections(gpu_ready):
    from skid_gb300 import gpu
    rng = np.random.default_rng(8)
    sizes = [1, 2, 31, 32, 33, 100, 128, 129, 250]
    n = sum(sizes) + 3
    grp = rng.permutation(np.concatenate([np.repeat(np.arange(1, len(sizes) + 1), sizes), [0] * 3])).astype(np.int32)
    pos = rng.normal(0.0, 0.02, (n, 3)).astype(np.float32)
    snap = tipsy.Snapshot(1.0, 0, n, 0, pos, np.zeros((n, 3), np.float32),
                          rng.uniform(0.5, 1.0, n).astype(np.float32), np.full(n, 1e-3, np.float32),
                          np.zeros(n, np.float32))
    v = rng.normal(size=len(sizes)).astype(np.float32)
    with gpu.Context(period=1.0, nSmooth=2) as ctx:
        ctx.set_particles(snap)
        ctx.set_groups(grp)
        E, grad = ctx.potential_adjoint(np.arange(1, len(sizes) + 1), v, soft_type=SPLINE)
        for g in range(1, len(sizes) + 1):
            before = ctx.timings()["kernel_launches"]
            e1, g1 = ctx.potential_adjoint([g], v[g - 1:g], soft_type=SPLINE)
            # pack, pairs, sums
            assert ctx.timings()["kernel_launches"] - before <= 3
            assert e1[0] == E[g - 1] and np.array_equal(g1[grp == g], grad[grp == g])
            assert not g1[grp != g].any()
            assert ctx.potential_adjoint([g], soft_type=SPLINE)[0][0] == E[g - 1]
    assert not grad[grp == 0].any() and E[0] == 0.0
