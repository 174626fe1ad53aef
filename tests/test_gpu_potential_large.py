"""Group potential energies and gradients of calls large enough for the
members' Hilbert order (from 4e8 pairs in large groups) and for column chunks
of 128 to 1024, with tiny and empty groups among the large ones and a selection that is
neither sorted nor complete, against FP64 all pairs in plain torch.

Tolerance: every pair term is a float within a few 2^-23 of its real value,
the energy's row sums are compensated, the gradient's are plain float sums of
at most 1024 columns, combined in FP64; 1e-5 of the sum of the terms'
magnitudes covers all of it several times over."""
import numpy as np
import pytest

from skid_gb300 import tipsy
from skid_gb300.options import PLUMMER, SPLINE

pytestmark = pytest.mark.gpu


def _psi(torch, r, e, plummer):
    if plummer:
        s = r * r + 0.25 * e * e
        return s ** -0.5, -(s ** -1.5)
    u, d = 2.0 * r / e, 2.0 / e
    p = torch.where(u < 1, d * (1.4 - 2 / 3 * u**2 + 0.3 * u**4 - 0.1 * u**5),
                    -1 / (15 * r) + d * (1.6 - 4 / 3 * u**2 + u**3 - 0.3 * u**4 + u**5 / 30))
    g = torch.where(u < 1, d**3 * (-4 / 3 + 1.2 * u**2 - 0.5 * u**3),
                    1 / (15 * r**3) + d**3 * (-8 / 3 + 3 * u - 1.2 * u**2 + u**3 / 6))
    return torch.where(u < 2, p, 1 / r), torch.where(u < 2, g, -(r ** -3.0))


def _all_pairs(torch, x, mass, soft, plummer):
    """Per row: potential sum, gradient sum and the sums of magnitudes."""
    n = len(x)
    x, mass, soft = (torch.from_numpy(a.astype(np.float64)).cuda() for a in (x, mass, soft))
    out = []
    for i in range(0, n, 512):
        d = x[i:i + 512, None, :] - x[None, :, :]
        r = (d * d).sum(-1).sqrt()
        k = torch.arange(min(512, n - i))
        own = torch.zeros_like(r, dtype=torch.bool)
        own[k, k + i] = True
        p, q = _psi(torch, torch.where(own, 1.0, r), soft[i:i + 512, None] + soft[None, :], plummer)
        p = torch.where(own, 0.0, p) * mass * mass[i:i + 512, None]
        q = torch.where(own, 0.0, q) * mass * mass[i:i + 512, None]
        out.append(torch.cat([p.sum(1)[:, None], (q[..., None] * d).sum(1), (q * r).abs().sum(1)[:, None]], 1))
    return torch.cat(out).cpu().numpy()


@pytest.mark.parametrize("sizes,soft_type", [
    ((16_000, 129, 1), SPLINE), ((3_000,) * 100, SPLINE), ((26_000, 13_000, 700, 1), SPLINE), ((31_000, 13_000, 2, 300), SPLINE),
    ((31_000, 13_000, 128), PLUMMER), ((21_000, 30_001, 5, 1000), SPLINE), ((52_000, 127), SPLINE)])
def test_large_calls(gpu_ready, sizes, soft_type):
    import torch
    from skid_gb300 import gpu
    rng = np.random.default_rng(sum(sizes))
    sizes = (0,) + sizes + (40,)       # an empty group, and one that is not selected
    n = sum(sizes) + 7
    grp = np.concatenate([np.repeat(np.arange(1, len(sizes) + 1), sizes), np.zeros(7, int)])
    grp = rng.permutation(grp).astype(np.int32)
    pos = (rng.uniform(-0.1, 0.1, (len(sizes) + 1, 3))[grp] +
           rng.normal(size=(n, 3)) * 0.02 * rng.random((n, 1)) ** 2).astype(np.float32)
    mass = rng.uniform(0.5, 1.0, n).astype(np.float32)
    soft = rng.uniform(1e-4, 1e-3, n).astype(np.float32)
    snap = tipsy.Snapshot(1.0, 0, n, 0, pos, np.zeros((n, 3), np.float32), mass, soft, np.zeros(n, np.float32))
    sel = rng.permutation(np.arange(1, len(sizes))).astype(np.int32)
    v = rng.normal(size=len(sel)).astype(np.float32)
    with gpu.Context(period=1.0, nSmooth=2) as ctx:
        ctx.set_particles(snap)
        ctx.set_groups(grp)
        only, _ = ctx.potential_adjoint(sel, None, soft_type=soft_type)
        E, grad = ctx.potential_adjoint(sel, v, soft_type=soft_type)
        again, grad2 = ctx.potential_adjoint(sel, v, soft_type=soft_type)
    assert np.array_equal(only, E) and np.array_equal(again, E) and np.array_equal(grad2, grad)
    assert not grad[(grp == 0) | (grp == len(sizes))].any()
    for s, g in enumerate(sel):
        m = np.nonzero(grp == g)[0]
        if len(m) == 0:
            assert E[s] == 0.0
            continue
        # coordinates are floats relative to the group's last member
        want = _all_pairs(torch, pos[m] - pos[m[-1]], mass[m], soft[m], soft_type == PLUMMER)
        e = -0.5 * want[:, 0].sum()
        assert abs(E[s] - e) <= 1e-5 * abs(e) + 1e-30, (g, len(m))
        err = np.linalg.norm(grad[m] + want[:, 1:4] * v[s], axis=1)
        assert np.all(err <= 1e-5 * want[:, 4] * abs(v[s]) + 1e-30), (g, len(m))
