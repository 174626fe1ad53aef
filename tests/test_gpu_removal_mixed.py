"""Unbinding's removal with groups on both sides of the warp limit in one
call: the large ones by blocks (or clusters of blocks), the small ones by
warps in a kernel that runs beside them, either kind alone, and groups that
lose every member.  The particles unbound must be the oracle's."""
import numpy as np
import pytest

from oracle import oracle
from skid_gb300 import tipsy
from skid_gb300.options import Options

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 31, 32, 33, 127, 128, 129, 300, 511, 513, 1023, 1024, 1025, 1500, 2100] + [16] * 700


def _case():
    rng = np.random.default_rng(23)
    n = sum(SIZES) + 40
    grp = rng.permutation(np.concatenate([np.repeat(np.arange(1, len(SIZES) + 1), SIZES),
                                          np.zeros(40, int)])).astype(np.int32)
    r = 0.01 * rng.random(n) ** 2
    d = rng.normal(size=(n, 3))
    pos = rng.uniform(-0.5, 0.5, (len(SIZES) + 1, 3))[grp] + r[:, None] * d / np.linalg.norm(d, axis=1)[:, None]
    pos -= np.floor(pos + 0.5)
    sig = np.sqrt(np.array([40] + SIZES)[grp] / n / 0.02)
    vel = rng.normal(size=(n, 3)) * sig[:, None] * np.where(rng.random(n) < 0.1, 2.0, 0.7)[:, None]
    vel[grp == 10] *= 50.0          # falls apart
    return tipsy.Snapshot(1.0, 0, n, 0, pos.astype(np.float32), vel.astype(np.float32),
                          np.full(n, 1.0 / n, np.float32), np.full(n, 4e-4, np.float32),
                          np.zeros(n, np.float32)), grp


@pytest.fixture(scope="module")
def case():
    snap, grp = _case()
    opts = Options.parse(["-tau", "0.01", "-p", "1", "-O", "0.3", "-Lambda", "0.7", "-H", "5.28444"])
    want = oracle.run_unbind(snap, opts, grp, None, stop_after=2)
    left = want["groups"]["nMembers"][1:]
    assert left.max() > 1024 and left.min() <= 1 and np.count_nonzero(left < np.array(SIZES)) > 100
    return snap, grp, opts, want


@pytest.mark.parametrize("tw,bs,clusters", [(0, 512, 0), (32, 128, 0), (128, 256, 0), (512, 512, 0),
                                            (1024, 1024, 0), (1024, 512, 1100), (256, 256, 1024)])
def test_blocks_and_warps_in_one_call(gpu_ready, case, tw, bs, clusters):
    from skid_gb300 import gpu
    snap, grp, opts, want = case
    for nmax in (2**31 - 1, 1000):   # groups from nmax on are left alone: at 1024 none takes a block
        with gpu.Context(period=1.0, nSmooth=2) as ctx:
            ctx.set_option("unbind_warp_max", tw)
            ctx.set_option("unbind_block", bs)
            ctx.set_option("unbind_cluster_min", clusters)
            ctx.set_particles(snap)
            ctx.set_groups(grp)
            nu = ctx.unbind(opts.iSoftType, opts.fScoop, False, False, nmax, opts.G, opts.z,
                            opts.a_shift, opts.a_hubble)
            out, _ = ctx.get_groups(len(SIZES))
        expect = np.where(np.array([40] + SIZES)[grp] < nmax, want["grp"], grp)
        assert np.array_equal(out, expect), nmax
        assert nu == np.count_nonzero(expect != grp)
