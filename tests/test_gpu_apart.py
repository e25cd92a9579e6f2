"""Objects that do not stand in the bag of their own column and row: set apart
from their positions, or at positions outside the matrix whose bag index runs
into another column.  Their first step against the oracle, on every path."""
import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle

pytestmark = pytest.mark.gpu
QUERIES = [kg.KB_QUERY_RELAX, kg.KB_QUERY_EXACT]
D = float(np.float32(10.0) / np.float32(1.5))


def outside(n, side, d, seed):
    """Birds of a square field, a third of them below or above its rows."""
    r = np.random.default_rng(seed)
    xy = r.uniform(0.0, side * (1 - 1e-6), (n, 2))
    far = r.random(n) < 1 / 3
    y = np.where(r.random(n) < 0.5, r.uniform(side + 2 * d, 2 * side, n), r.uniform(-side, -2 * d, n))
    # columns in which the index stays inside the matrix
    x = np.where(y > 0, r.uniform(0.0, side / 2, n), r.uniform(side / 2, side * (1 - 1e-6), n))
    xy[far] = np.stack([x, y], 1)[far]
    a = r.uniform(0, 2 * np.pi, n)
    return np.arange(n, dtype=np.uint32), xy.astype(np.float32), np.stack([np.cos(a), np.sin(a)], 1).astype(np.float32)


def oracle_after(side, d, birds, p, steps):
    o = oracle.OracleField(side, side, d, True)
    o.set_many(*birds)
    o.lazy_update()
    o.flock_run(oracle.params_from(p), 0, steps)
    ids, st, _ = o.iter(1)
    return ids, st


def same(got, want):
    return np.array_equal(got[0], want[0]) and np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))


@pytest.mark.parametrize("kind", QUERIES)
@pytest.mark.parametrize("mode", [0, 3, 2])  # the cluster, the separate kernels, the tiled step
@pytest.mark.parametrize("load", ["host", "device", "single"])
@pytest.mark.parametrize("d", [D, 4.0])
def test_positions_outside_the_matrix(gpu, kind, mode, load, d):
    side, n = 200.0, 900
    birds = outside(n, side, d, 3)
    p = kg.FlockParams(seed=1, arith=kg.KB_ARITH_STRICT, query_mode=kind)
    f = kg.Field2D(side, side, d, True)
    f.set_step_options(mode)
    if load == "host":
        f.set_locations(*birds)
    elif load == "device":
        torch = pytest.importorskip("torch")
        st = torch.from_numpy(np.concatenate(birds[1:], 1)).cuda()
        f.set_states_device(torch.from_numpy(birds[0].view(np.int32)).cuda(), st)
    else:
        for i, at, h in zip(*birds):
            at = kg.Real2D(float(at[0]), float(at[1]))
            f.set_object_location(kg.Bird(int(i), at, kg.Real2D(float(h[0]), float(h[1]))), at)
    f.lazy_update()
    for s, k in ((0, 1), (1, 5)):
        f.flock_step(p, s, k)
        assert same(f.get_state(), oracle_after(side, d, birds, p, s + k)), s
    assert f.device_flags() == 0
    f.close()


@pytest.mark.parametrize("kind", QUERIES)
@pytest.mark.parametrize("mode", [0, 2])
def test_packed_replicas_outside_the_matrix(gpu, kind, mode):
    def replica(i, birds):
        return kg.Replica(200.0, 200.0, D, kg.FlockParams(seed=i, arith=kg.KB_ARITH_STRICT, query_mode=kind), birds)

    reps = [replica(0, kg.gen_uniform(700, 200.0, 200.0, 5, 1.0)), replica(1, outside(600, 200.0, D, 6))]
    late = replica(2, outside(500, 200.0, D, 7))
    with kg.Batch(reps) as b:
        b.set_step_options(mode)
        b.step(0, 1)
        b.step(1, 4)
        for i, r in enumerate(reps):
            assert same(b.get_replica(i), oracle_after(200.0, D, r.state, r.params, 5))
        b.add_replica(late, 5)
        b.step(5, 3)
        assert same(b.get_replica(0), oracle_after(200.0, D, reps[0].state, reps[0].params, 8))
        assert same(b.get_replica(2), oracle_after(200.0, D, late.state, late.params, 3))


@pytest.mark.parametrize("kind", QUERIES)
@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("d,radius", [(D, 10.0), (2.0, 9.0)])
def test_objects_set_anywhere(gpu, kind, mode, d, radius):
    side, n = 100.0, 150
    r = np.random.default_rng(4)
    pos = r.uniform(0, side * (1 - 1e-6), (n, 2)).astype(np.float32)
    loc = np.where(r.random((n, 1)) < 1 / 3, r.uniform(0, side * (1 - 1e-6), (n, 2)), pos).astype(np.float32)
    f, o = kg.Field2D(side, side, d, True), oracle.OracleField(side, side, d, True)
    f.set_step_options(mode)
    for i in range(n):
        b = kg.Bird(i, kg.Real2D(float(pos[i, 0]), float(pos[i, 1])), kg.Real2D(0.6, 0.8))
        f.set_object_location(b, kg.Real2D(float(loc[i, 0]), float(loc[i, 1])))
        o.set(i, pos[i, 0], pos[i, 1], 0.6, 0.8, loc[i, 0], loc[i, 1])
    f.lazy_update()
    o.lazy_update()
    p = kg.FlockParams(seed=5, arith=kg.KB_ARITH_STRICT, query_mode=kind, neighbor_radius=radius)
    f.flock_step(p, 0, 3)
    o.flock_run(oracle.params_from(p), 0, 3)
    assert same(f.get_state(), o.iter(1)[:2])
    f.close()
