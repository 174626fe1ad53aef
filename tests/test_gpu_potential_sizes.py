"""Group potential energies and gradients at the sizes where the pair sums'
row tiles (128) and column chunks begin and end, against FP64 all pairs.

Tolerance: every pair term is a float within a few 2^-23 of its real value
(hardware reciprocal square root, spline in FP32, float coordinates), the
energy's row sums are compensated and the gradient's are plain float sums of
at most 1024 columns, combined in FP64; 1e-5 of the sum of the terms'
magnitudes covers all of it several times over."""
import numpy as np
import pytest

from skid_gb300 import tipsy
from skid_gb300.options import PLUMMER, SPLINE

pytestmark = pytest.mark.gpu


def _psi(r, e, plummer):
    if plummer:
        s = r * r + 0.25 * e * e
        return s ** -0.5, -(s ** -1.5)
    u = 2.0 * r / e
    d = 2.0 / e
    p1 = d * (1.4 - 2 / 3 * u**2 + 0.3 * u**4 - 0.1 * u**5)
    g1 = d**3 * (-4 / 3 + 1.2 * u**2 - 0.5 * u**3)
    with np.errstate(divide="ignore"):
        p2 = -1 / (15 * r) + d * (1.6 - 4 / 3 * u**2 + u**3 - 0.3 * u**4 + u**5 / 30)
        g2 = 1 / (15 * r**3) + d**3 * (-8 / 3 + 3 * u - 1.2 * u**2 + u**3 / 6)
        p3, g3 = 1 / r, -(r ** -3.0)
    return (np.where(u < 1, p1, np.where(u < 2, p2, p3)), np.where(u < 1, g1, np.where(u < 2, g2, g3)))


@pytest.mark.parametrize("soft_type", [SPLINE, PLUMMER])
@pytest.mark.parametrize("sizes", [(1, 2, 127, 128, 129), (255, 257, 1023, 1024, 1025), (9000, 40)])
def test_potential_at_tile_edges(gpu_ready, sizes, soft_type):
    from skid_gb300 import gpu
    rng = np.random.default_rng(sum(sizes))
    n = sum(sizes) + 5
    grp = rng.permutation(np.concatenate([np.repeat(np.arange(1, len(sizes) + 1), sizes),
                                          np.zeros(5, int)])).astype(np.int32)
    pos = (rng.uniform(-0.1, 0.1, (len(sizes) + 1, 3))[grp] +
           rng.normal(size=(n, 3)) * 0.02 * rng.random((n, 1))).astype(np.float32)
    mass = rng.uniform(0.5, 1.0, n).astype(np.float32)
    soft = rng.uniform(1e-4, 3e-3, n).astype(np.float32)
    snap = tipsy.Snapshot(1.0, 0, n, 0, pos, np.zeros((n, 3), np.float32), mass, soft,
                          np.zeros(n, np.float32))
    sel = np.array(list(range(1, len(sizes) + 1)) + [1], np.int32)    # one group twice
    v = rng.normal(size=len(sel)).astype(np.float32)
    v[-1] = v[0]
    with gpu.Context(period=1.0, nSmooth=2) as ctx:
        ctx.set_particles(snap)
        ctx.set_groups(grp)
        only, _ = ctx.potential_adjoint(sel, None, soft_type=soft_type)
        E, grad = ctx.potential_adjoint(sel, v, soft_type=soft_type)
    assert E[-1] == E[0] and np.array_equal(only, E)
    for s, g in enumerate(sel[:-1]):
        m = np.nonzero(grp == g)[0]
        x = (pos[m] - pos[m[-1]]).astype(np.float64)
        e0, mag, gr, gmag = 0.0, 1e-30, np.zeros((len(m), 3)), np.full(len(m), 1e-30)
        for i in range(len(m)):
            j = np.arange(len(m)) != i
            d = x[i] - x[j]
            p, q = _psi(np.sqrt((d * d).sum(1)), soft[m[i]].astype(float) + soft[m[j]], soft_type == PLUMMER)
            mm = float(mass[m[i]]) * mass[m[j]].astype(float)
            e0 -= 0.5 * (mm * p).sum()
            mag += 0.5 * np.abs(mm * p).sum()
            t = (mm * q)[:, None] * d
            gr[i] = -t.sum(0) * v[s]
            gmag[i] += np.linalg.norm(t, axis=1).sum() * abs(v[s])
        assert abs(E[s] - e0) <= 1e-5 * mag
        assert np.all(np.linalg.norm(grad[m] - gr, axis=1) <= 1e-5 * gmag)
