"""Unbinding's block removal of groups larger than a block's shared memory
(some 7,000 members), where every member's exact potential is asked for in the
middle of the removals -- exact ties among the fast members, a negative mass --
so that members in shared memory and beyond it are brought up to date together
and removed from afterwards; with and without the removed members' potentials
taken off the others (dark particles alone, several species).  The particles
unbound must be the oracle's."""
import numpy as np
import pytest

from oracle import oracle
from skid_gb300 import tipsy
from skid_gb300.options import Options

pytestmark = pytest.mark.gpu


def _case(n, kind, species):
    rng = np.random.default_rng(n + len(kind))
    r = 0.02 * rng.random(n) ** 1.5
    d = rng.normal(size=(n, 3))
    pos = 0.3 + r[:, None] * d / np.linalg.norm(d, axis=1)[:, None]
    vel = rng.normal(size=(n, 3)) * 0.5
    mass = np.full(n, 1.0 / n)
    fast = rng.choice(np.nonzero(r > 0.01)[0], 60, replace=False)
    vel[fast] *= 30.0 / np.linalg.norm(vel[fast], axis=1)[:, None]
    if kind in ("ties", "some ties"):    # sixty members, everything equal, at one place or five
        at = fast[np.arange(60) % (1 if kind == "ties" else 5)]
        pos[fast], vel[fast] = pos[at], vel[at]
    if kind == "negative":
        mass[rng.integers(0, n)] *= -0.5
    if kind == "masses":
        mass *= rng.uniform(0.5, 2.0, n)
    grp = np.ones(n + 20, np.int32)
    grp[rng.choice(n + 20, 20, replace=False)] = 0
    order = np.argsort(grp == 0, kind="stable")
    out = [np.empty((n + 20,) + a.shape[1:], np.float32) for a in (pos, vel, mass)]
    for o, a in zip(out, (pos, vel, mass)):
        o[order[:n]] = a
        o[order[n:]] = 0.1 if a.ndim > 1 else 1.0 / n
    ng, nd = (0, n + 20) if species == "dark" else (n // 3, n // 3)
    return tipsy.Snapshot(1.0, ng, nd, n + 20 - ng - nd, *out, np.full(n + 20, 4e-4, np.float32),
                          np.zeros(n + 20, np.float32)), grp


@pytest.mark.parametrize("species", ["dark", "mixed"])
@pytest.mark.parametrize("n,kind", [(7030, "ties"), (7300, "ties"), (7300, "some ties"), (7300, "negative"),
                                    (9001, "masses"), (12_000, "ties")])
def test_flush_across_the_shared_memory_boundary(gpu_ready, n, kind, species):
    from skid_gb300 import gpu
    snap, grp = _case(n, kind, species)
    opts = Options.parse(["-tau", "0.01", "-p", "1", "-O", "0.3", "-Lambda", "0.7", "-H", "5.28444"])
    want = oracle.run_unbind(snap, opts, grp, None, stop_after=2)
    assert 30 <= want["nUnbound"] < n // 4
    for bs in (128, 512, 1024):
        with gpu.Context(period=1.0, nSmooth=2) as ctx:
            ctx.set_option("unbind_warp_max", 1024)
            ctx.set_option("unbind_block", bs)
            ctx.set_particles(snap)
            ctx.set_groups(grp)
            nu = ctx.unbind(opts.iSoftType, opts.fScoop, False, False, 2**31 - 1, opts.G, opts.z,
                            opts.a_shift, opts.a_hubble)
            out, rec = ctx.get_groups(1)
        assert nu == want["nUnbound"], bs
        assert np.array_equal(out, want["grp"]), bs
        assert np.abs(rec["rBound"][1] - want["groups"]["rBound"][1]).max() < 1e-5, bs
