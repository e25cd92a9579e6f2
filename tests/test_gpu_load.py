"""Loading a field (the general stable sort and what it finds out) against the
oracle: bags at the edges of the arrival slots and far past them, removals,
objects placed apart from their positions, and ids of every kind."""
import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("occ", [1, 4, 5, 12, 13, 31, 33, 400])
def test_load_order_of_full_bags(gpu, occ):
    side, d = 60.0, 5.0
    r = np.random.default_rng(occ)
    pts = [r.uniform(0, side * (1 - 1e-6), (90, 2))] + [np.full((occ, 2), c) + r.uniform(0, 4.9, (occ, 2)) for c in (0.0, 25.0, 55.0)]
    xy = r.permutation(np.concatenate(pts).astype(np.float32))
    n = len(xy)
    ids = r.permutation(n).astype(np.uint32)
    dxy = r.uniform(-1, 1, (n, 2)).astype(np.float32)
    f, o = kg.Field2D(side, side, d, True), oracle.OracleField(side, side, d, True)
    f.set_locations(ids, xy, dxy)
    o.set_many(ids, xy, dxy)
    gone = int(ids[n // 2])  # a removed object leaves no gap
    loc = kg.Real2D(float(xy[n // 2, 0]), float(xy[n // 2, 1]))
    f.remove_object_location(kg.Bird(gone, loc), loc)
    f.lazy_update()
    o.lazy_update()
    gi, gs = f.get_state()
    oi, os_, _ = o.iter(1)
    keep = oi != gone
    assert f.num_objects() == n - 1
    assert np.array_equal(gi, oi[keep]) and np.array_equal(gs.view(np.uint32), os_[keep].view(np.uint32))
    f.close()


@pytest.mark.parametrize("kind", ["below", "past", "mixed", "repeat below", "repeat past"])
def test_steps_with_every_kind_of_ids_match_oracle(gpu, kind):
    n, side = 3000, 300.0
    _, xy, dxy = kg.gen_uniform(n, side, side, 9, 1.0)
    ids = np.arange(n, dtype=np.uint32)
    if kind in ("past", "repeat past"):
        ids = ids + np.uint32(0xFFFF0000)
    if kind == "mixed":
        ids[::2] += np.uint32(1 << 20)
    if kind.startswith("repeat"):
        ids[17] = ids[2900]
    p = kg.FlockParams(seed=1, arith=kg.KB_ARITH_STRICT)
    d = float(np.float32(10.0) / np.float32(1.5))
    f, o = kg.Field2D(side, side, d, True), oracle.OracleField(side, side, d, True)
    f.set_step_options(3)
    for k in range(2):  # twice: the second load finds the first one's marks cleared
        f.set_locations(ids, xy, dxy)
        f.lazy_update()
    o.set_many(ids, xy, dxy)
    o.lazy_update()
    f.flock_step(p, 0, 3)
    o.flock_run(oracle.params_from(p), 0, 3)
    gi, gs = f.get_state()
    oi, os_, _ = o.iter(1)
    assert np.array_equal(gi, oi) and np.array_equal(gs.view(np.uint32), os_.view(np.uint32))
    f.close()
