"""The .stat columns of a catalogue of many small groups, where the small ones
take a thread each and the larger a warp each, against the same host
restatement the golden cases are held to (bit-identical)."""
import numpy as np
import pytest

from skid_gb300 import tipsy
from skid_gb300.options import Options
from tests.test_gpu_stats import host_stats

pytestmark = pytest.mark.gpu


def test_many_groups(gpu_ready):
    from skid_gb300 import gpu
    rng = np.random.default_rng(41)
    sizes = np.concatenate([rng.integers(2, 6, 19_000), rng.integers(25, 41, 200), [31, 32, 33, 64, 65, 300]])
    sizes = rng.permutation(sizes)
    n = int(sizes.sum()) + 40
    grp = np.concatenate([np.repeat(np.arange(1, len(sizes) + 1), sizes), np.zeros(40, int)])
    grp = rng.permutation(grp).astype(np.int32)
    pos = rng.uniform(-0.5, 0.5, (len(sizes) + 1, 3))[grp] + rng.normal(size=(n, 3)) * 0.01 * rng.random((n, 1))
    pos = (pos - np.floor(pos + 0.5)).astype(np.float32)
    snap = tipsy.Snapshot(1.0, n // 3, n // 3, n - 2 * (n // 3), pos, rng.normal(size=(n, 3)).astype(np.float32),
                          (rng.uniform(0.2, 1.0, n) / n).astype(np.float32),
                          rng.choice([0.0, 2e-4, 5e-3], n).astype(np.float32),
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
    assert len(want) == ng
    for g, w in want.items():
        assert tuple(np.float32(x) for x in got[g]) == tuple(np.float32(x) for x in w), (g, sizes[g - 1])
