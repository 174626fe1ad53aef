"""The .stat columns at the sizes where the 32-member batches of a group's
walk begin and end, with all three species, against the same one-operation-
at-a-time host restatement the golden cases are held to (bit-identical)."""
import numpy as np
import pytest

from skid_gb300 import tipsy
from skid_gb300.options import Options
from tests.test_gpu_stats import host_stats

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(2, 3, 31, 32, 33), (63, 64, 65, 96, 97), (1000, 5003)])
def test_stats_at_batch_edges(gpu_ready, sizes):
    from skid_gb300 import gpu
    rng = np.random.default_rng(sum(sizes))
    n = sum(sizes) + 40
    grp = np.concatenate([np.repeat(np.arange(1, len(sizes) + 1), sizes), np.zeros(40, int)])
    grp = rng.permutation(grp).astype(np.int32)
    centre = rng.uniform(-0.5, 0.5, (len(sizes) + 1, 3))
    pos = centre[grp] + rng.normal(size=(n, 3)) * 0.01 * rng.random((n, 1))
    pos = (pos - np.floor(pos + 0.5)).astype(np.float32)
    mass = (rng.uniform(0.2, 1.0, n) / n).astype(np.float32)
    soft = np.full(n, 2e-4, np.float32)
    snap = tipsy.Snapshot(1.0, n // 3, n // 3, n - 2 * (n // 3), pos,
                          rng.normal(size=(n, 3)).astype(np.float32), mass, soft,
                          rng.uniform(0, 2e4, n).astype(np.float32))
    opts = Options.parse(["-tau", "0.01", "-p", "1", "-H", "2.8944", "-t", "1e4"])
    with gpu.Context(period=1.0, nSmooth=2) as ctx:
        ctx.set_particles(snap)
        ctx.set_groups(grp)
        ctx.unbind(opts.iSoftType, opts.fScoop, False, True, 2**31 - 1, opts.G, opts.z,
                   opts.a_shift, opts.a_hubble)
        ng = ctx.too_small(1)
        out, rec = ctx.get_groups(ng)
        got = ctx.group_stats(ng, opts.G, opts.a_shift, opts.a_hubble, opts.fDensMin, opts.fTempMax)
    assert ng == len(sizes) and np.array_equal(out, grp)
    want = host_stats(snap, out, rec, np.zeros(n, np.float32), opts)
    for g, w in want.items():
        assert tuple(np.float32(x) for x in got[g]) == tuple(np.float32(x) for x in w), g
