"""Unbinding's potentials where tile pairs hold no, some or only pairs inside
the softening, so that their steps run packed, one by one, or both in one
group: what is unbound, and every record, must be the oracle's."""
import numpy as np
import pytest

from oracle import oracle
from skid_gb300 import tipsy
from skid_gb300.options import Options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plummer", [False, True])
@pytest.mark.parametrize("equal", [True, False])
def test_near_and_far_tile_pairs(gpu_ready, equal, plummer):
    from skid_gb300 import gpu
    rng = np.random.default_rng(31 + equal)
    sizes = [129, 256, 300, 700, 1024, 1500, 2000]
    n = sum(sizes) + 50
    # members in file order: spread ones first, then an ever denser core, and
    # one group with the two interleaved
    grp, pos = [], []
    for g, s in enumerate(sizes):
        r = 0.03 * (np.arange(s)[::-1] / s) ** (1.0 + 2.0 * g / len(sizes))
        if g == 4:
            r = rng.permutation(r)
        d = rng.normal(size=(s, 3))
        pos.append(rng.uniform(-0.4, 0.4, 3) + r[:, None] * d / np.linalg.norm(d, axis=1)[:, None])
        grp.append(np.full(s, g + 1))
    pos = np.concatenate(pos + [rng.uniform(-0.5, 0.5, (50, 3))]).astype(np.float32)
    grp = np.concatenate(grp + [np.zeros(50, int)]).astype(np.int32)
    mass = np.full(n, 1.0 / n) * (1.0 if equal else rng.uniform(0.5, 2.0, n))
    soft = np.full(n, 2e-3) * (1.0 if equal else rng.uniform(0.2, 1.0, n))
    sig = np.sqrt(np.array([50] + sizes)[grp] / n / 0.03)
    vel = rng.normal(size=(n, 3)) * sig[:, None] * np.where(rng.random(n) < 0.1, 2.5, 0.8)[:, None]
    snap = tipsy.Snapshot(1.0, 0, n, 0, pos, vel.astype(np.float32), mass.astype(np.float32),
                          soft.astype(np.float32), np.zeros(n, np.float32))
    opts = Options.parse(["-tau", "0.01", "-p", "1", "-O", "0.3", "-Lambda", "0.7", "-H", "5.28444"] +
                         (["-plummer"] if plummer else []))
    want = oracle.run_unbind(snap, opts, grp, None, stop_after=2)
    assert 50 < want["nUnbound"] < n // 2
    with gpu.Context(period=1.0, nSmooth=2) as ctx:
        ctx.set_particles(snap)
        ctx.set_groups(grp)
        nu = ctx.unbind(opts.iSoftType, opts.fScoop, False, False, 2**31 - 1, opts.G, opts.z,
                        opts.a_shift, opts.a_hubble)
        out, rec = ctx.get_groups(len(sizes))
    assert nu == want["nUnbound"] and np.array_equal(out, want["grp"])
    assert np.abs(rec["rBound"][1:] - want["groups"]["rBound"][1:]).max() < 1e-5
