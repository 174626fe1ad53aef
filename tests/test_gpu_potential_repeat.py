"""Group potential energies and gradients are the same bits on every call: a
row's sums over its column chunks are added in chunk order, not in the order
in which blocks finish.  The group is one where the order shows: two heavy
members in different chunks pull the last member with exactly opposite forces
some 2^40 times the rest's, so that the FP64 sum keeps more or fewer of the
rest's bits as they are added before or after."""
import numpy as np
import pytest

from skid_gb300 import tipsy
from skid_gb300.options import PLUMMER, SPLINE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("soft_type", [SPLINE, PLUMMER])
def test_same_bits_on_every_call(gpu_ready, soft_type):
    from skid_gb300 import gpu
    rng = np.random.default_rng(3)
    n = 4000
    pos = rng.uniform(-0.4, 0.4, (n, 3)).astype(np.float32)
    mass = rng.uniform(0.5, 1.5, n).astype(np.float32)
    pos[-1] = 0.0                       # the reference point of the group
    pos[700], pos[2900] = (0.25, 0, 0), (-0.25, 0, 0)
    mass[[700, 2900]] = 2.0**40
    grp = np.ones(n, np.int32)
    snap = tipsy.Snapshot(1.0, 0, n, 0, pos, np.zeros((n, 3), np.float32), mass,
                          np.full(n, 1e-3, np.float32), np.zeros(n, np.float32))
    with gpu.Context(period=None, nSmooth=2) as ctx:
        ctx.set_particles(snap)
        ctx.set_groups(grp)
        runs = [ctx.potential_adjoint([1], [1.0], soft_type=soft_type) for _ in range(100)]
        only = ctx.potential_adjoint([1], soft_type=soft_type)[0]
    E, grad = runs[0]
    assert only == E and 0 < abs(grad[-1]).max() < 2.0**20
    for e, g in runs[1:]:
        assert e == E and np.array_equal(g, grad)
