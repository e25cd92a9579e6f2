"""Offsets of bag matrices at the edges of the scan forms (the cluster scan takes
up to 32,768 bags), through loads and steps against the oracle."""
import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lines", [5, 64, 90, 128, 181, 182, 260])  # 181^2 <= 32768 < 182^2
def test_steps_over_bag_counts_match_oracle(gpu, lines):
    d = 5.0
    side, n = d * (lines - 1), 4000
    ids, xy, dxy = kg.gen_uniform(n, side, side, lines, 1.0)
    xy[-1] = side * (1 - 1e-6)  # the last bags too
    p = kg.FlockParams(seed=lines, arith=kg.KB_ARITH_STRICT, neighbor_radius=7.5)
    f, o = kg.Field2D(side, side, d, True), oracle.OracleField(side, side, d, True)
    f.set_step_options(3)
    f.set_locations(ids, xy, dxy)
    o.set_many(ids, xy, dxy)
    f.lazy_update()
    o.lazy_update()
    f.flock_step(p, 0, 4)
    o.flock_run(oracle.params_from(p), 0, 4)
    gi, gs = f.get_state()
    oi, os_, _ = o.iter(1)
    assert np.array_equal(gi, oi) and np.array_equal(gs.view(np.uint32), os_.view(np.uint32))
    assert f.num_objects() == n and f.moments()[0] == n
    f.close()
