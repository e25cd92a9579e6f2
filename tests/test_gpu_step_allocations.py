"""Steps allocate no device memory, also those that measure how dense the flock
has become: everything they need is made with the load."""
import numpy as np
import pytest

import krabmaga_gb300 as kg
from krabmaga_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,density", [(6000, 0.025), (6000, 0.5)])
def test_long_runs_allocate_nothing(gpu, n, density):
    side, d = float(np.float32(np.sqrt(n / density))), float(np.float32(10.0) / np.float32(1.5))
    f = kg.Field2D(side, side, d, True)
    f.set_locations(*kg.gen_uniform(n, side, side, 3, 1.0))
    f.lazy_update()
    before = L.allocation_counts()[0]
    p = kg.FlockParams(seed=1)
    for k in range(4):
        f.flock_step(p, 50 * k, 50)
    f.synchronize()
    assert L.allocation_counts()[0] == before
    f.close()
