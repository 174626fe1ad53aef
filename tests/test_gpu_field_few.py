"""Field probes of few positions: at most a few warps' worth cannot gain from
being sorted, and such a call launches nothing for it; the values are the
same on both sides of the count from which positions are sorted."""
import numpy as np
import pytest

from skid_gb300 import tipsy

pytestmark = pytest.mark.gpu


def test_few_positions_are_not_sorted(gpu_ready):
    from skid_gb300 import gpu
    rng = np.random.default_rng(11)
    n = 4000
    pos = rng.uniform(-0.5, 0.5, (n, 3)).astype(np.float32)
    snap = tipsy.Snapshot(1.0, 0, n, 0, pos, np.zeros((n, 3), np.float32), np.full(n, 1.0 / n, np.float32),
                          np.zeros(n, np.float32), np.zeros(n, np.float32))
    y = rng.uniform(-0.5, 0.5, (300, 3)).astype(np.float32)
    w = rng.normal(size=300).astype(np.float32)
    with gpu.Context(period=1.0, nSmooth=32) as ctx:
        ctx.set_particles(snap)
        ctx.scatter_active()
        ctx.density()
        every = ctx.field(y)             # sorted
        for nm in (1, 31, 32, 33, 64, 127, 128, 129):
            before = ctx.timings()["kernel_launches"]
            a = ctx.field(y[:nm])
            launched = ctx.timings()["kernel_launches"] - before
            assert np.array_equal(a, every[:nm]), nm
            # pack, order, field
            assert launched <= 3 or nm >= 128, (nm, launched)
            assert np.array_equal(ctx.field_adjoint(y[:nm], w[:nm]), -w[:nm, None] * a), nm
        # one position per warp: no walk is shared
        ctx.set_option("field_movers_per_warp", 1)
        before = ctx.timings()["kernel_launches"]
        a = ctx.field(y)
        assert ctx.timings()["kernel_launches"] - before <= 3
        assert np.array_equal(ctx.field(y[::-1])[::-1], a)
        ctx.set_option("field_movers_per_warp", 0)
        assert ctx.field(y[:0]).shape == (0, 3)
