"""Friends-of-friends at ragged counts and tree depths, across the periodic
faces, with equal positions, and at a linking length where one group spans the
box: the groups (numbered by their smallest index) must be the connected
components of the float distance rule, both frames of an image pair counted."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32


def _components(pos, tau, period):
    n = len(pos)
    tau2 = F(tau) * F(tau)
    label = np.arange(n)

    def frame(a, b):
        d = []
        for c in range(3):
            x = a[c] - b[:, c]
            if period:
                L, h = F(period), F(0.5 * period)
                x = np.where(x > h, (a[c] - L) - b[:, c], np.where(x < -h, (a[c] + L) - b[:, c], x))
            d.append(x.astype(F))
        return ((d[0] * d[0] + d[1] * d[1]).astype(F) + d[2] * d[2]).astype(F)

    adj = np.array([frame(pos[i], pos) < tau2 for i in range(n)])
    adj |= adj.T
    for i in range(n):
        if label[i] != i:
            continue
        todo = [i]
        seen = np.zeros(n, bool)
        seen[i] = True
        while todo:
            new = adj[todo].any(0) & ~seen
            seen |= new
            todo = list(np.flatnonzero(new))
        label[seen] = i
    return np.unique(label, return_inverse=True)[1] + 1


@pytest.mark.parametrize("kind", ["box", "clumps", "equal"])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 1000, 1025, 3001])
@pytest.mark.parametrize("f", [0.5, 1.1])
def test_components(gpu_ready, n, kind, f):
    from skid_gb300 import gpu
    rng = np.random.default_rng(n + len(kind))
    pos = rng.uniform(-0.5, 0.5, (n, 3))
    if kind == "clumps":
        pos[: n // 2] = pos[n - 1] + 0.1 * rng.normal(size=(n // 2, 3)) * rng.random((n // 2, 1)) ** 3
    if kind == "equal":
        pos = pos[rng.integers(0, max(1, n // 5), n)]
    pos = (pos - np.floor(pos + 0.5)).astype(F)
    pos = np.minimum(pos, F(0.49999997))
    tau = f * n ** (-1.0 / 3.0) if n > 2 else 0.2
    period = 1.0 if kind != "clumps" else None
    with gpu.Context(period=period) as ctx:
        grp, ng = ctx.fof_points(pos, tau)
    want = _components(pos, tau, period)
    assert ng == want.max()
    assert np.array_equal(grp, want)
