"""Scoop lists where the walk of the ungrouped particles' tree changes form --
a single leaf, a ragged one, one subtree of 32 leaves and more -- with a scoop
that takes none, some and nearly all of them, across the periodic faces: the
particles unbound must be those of the oracle's FP64 loop."""
import numpy as np
import pytest

from oracle import oracle
from skid_gb300 import tipsy
from skid_gb300.options import Options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scoop", ["0", "0.02", "0.45"])
@pytest.mark.parametrize("free", [1, 31, 32, 33, 65, 1024, 1025, 2500])
def test_unbound_with_scooped_particles(gpu_ready, free, scoop):
    from skid_gb300 import gpu
    rng = np.random.default_rng(free)
    sizes = [3, 40, 150, 500]
    n = sum(sizes) + free
    grp = rng.permutation(np.concatenate([np.zeros(free, int),
                                          np.repeat(np.arange(1, 5), sizes)])).astype(np.int32)
    centre = np.array([[0, 0, 0], [0.49, 0.49, 0.49], [-0.49, 0.1, 0.2], [0.1, 0.0, -0.1], [0.3, -0.2, 0.49]])
    pos = centre[grp] + 0.02 * rng.normal(size=(n, 3)) * rng.random((n, 1))
    loose = (grp == 0) & (rng.random(n) < 0.7)
    pos[loose] = centre[rng.integers(1, 5, loose.sum())] + 0.05 * rng.normal(size=(loose.sum(), 3))
    pos -= np.floor(pos + 0.5)
    mass = np.full(n, 1.0 / n)
    vel = rng.normal(size=(n, 3)) * np.sqrt(np.bincount(grp)[grp] / n / 0.03)[:, None]
    snap = tipsy.Snapshot(1.0, 0, n, 0, pos.astype(np.float32), vel.astype(np.float32),
                          mass.astype(np.float32), np.full(n, 4e-4, np.float32), np.zeros(n, np.float32))
    opts = Options.parse(["-tau", "0.01", "-p", "1", "-O", "0.3", "-Lambda", "0.7", "-H", "5.28444",
                          "-scoop", scoop])
    want = oracle.run_unbind(snap, opts, grp, None, stop_after=2)
    assert want["nUnbound"] > 0
    with gpu.Context(period=1.0, nSmooth=2) as ctx:
        ctx.set_particles(snap)
        ctx.set_groups(grp)
        nu = ctx.unbind(opts.iSoftType, opts.fScoop, False, False, 2**31 - 1, opts.G, opts.z,
                        opts.a_shift, opts.a_hubble)
        out, _ = ctx.get_groups(4)
    assert nu == want["nUnbound"]
    assert np.array_equal(out, want["grp"])
