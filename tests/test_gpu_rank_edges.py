"""Fuller bags at every place of a small matrix: the corners, the first and last
lines, the seam's and those beside them, with birds that wrap past both sides, so
that every combination of source lines is read; the last column and row of every
width.  Against the oracle, plain and packed."""
import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle

pytestmark = pytest.mark.gpu
D = 5.0


def birds(side, occ, seed):
    r = np.random.default_rng(seed)
    last = side - 1e-3
    lines = [0.2, D - 0.2, D + 0.2, side / 2, side - 2 * D, side - D - 0.2, side - D + 0.2, last]
    pts = [np.mod(np.array([x, y]) + r.uniform(-0.6, 0.6, (occ, 2)), side) for x in lines for y in lines]
    xy = np.clip(np.concatenate(pts), 0, np.nextafter(np.float32(side), np.float32(0))).astype(np.float32)
    xy = xy[r.permutation(len(xy))]
    a = r.uniform(0, 2 * np.pi, len(xy))
    return np.arange(len(xy), dtype=np.uint32), xy, np.stack([np.cos(a), np.sin(a)], 1).astype(np.float32)


def after(side, state, p, steps):
    o = oracle.OracleField(side, side, D, True)
    o.set_many(*state)
    o.lazy_update()
    o.flock_run(oracle.params_from(p), 0, steps)
    return o.iter(1)[:2]


def same(got, want):
    return np.array_equal(got[0], want[0]) and np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))


# widths that leave a whole, a narrow and a wide last column
@pytest.mark.parametrize("side", [25.0, 40.0, 40.4, 44.8])
@pytest.mark.parametrize("occ", [4, 14, 40])
@pytest.mark.parametrize("jump", [0.7, 4.9])
def test_every_edge_matches_oracle(gpu, side, occ, jump):
    state = birds(side, occ, occ)
    p = kg.FlockParams(seed=1, arith=kg.KB_ARITH_STRICT, neighbor_radius=4.0, jump=jump, cohesion=0.2)
    f = kg.Field2D(side, side, D, True)
    f.set_step_options(3)
    f.set_dense_mode(kg.KB_DENSE_OFF)  # ranks, not segments
    f.set_locations(*state)
    f.lazy_update()
    f.flock_step(p, 0, 4)
    assert same(f.get_state(), after(side, state, p, 4))
    assert f.device_flags() == 0
    f.close()


@pytest.mark.parametrize("occ", [4, 14])
def test_every_edge_of_packed_replicas_matches_oracle(gpu, occ):
    reps = []
    for i, side in enumerate((25.0, 40.4, 44.8, 60.0)):
        p = kg.FlockParams(seed=i, arith=kg.KB_ARITH_STRICT, neighbor_radius=4.0, jump=0.7 + i, cohesion=0.2)
        reps.append(kg.Replica(side, side, D, p, birds(side, occ, 7 * occ + i)))
    with kg.Batch(reps) as b:
        b.step(0, 4)
        for i, r in enumerate(reps):
            assert same(b.get_replica(i), after(r.width, r.state, r.params, 4))
