"""Fields wider than high and higher than wide against the oracle.  A bird's y
wraps with the width (bird.rs:147), so on a field wider than high birds stand
beyond the height, in bags of the columns behind their own, and pairs straddle
the seam inside a ring of bags."""
import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle

pytestmark = pytest.mark.gpu
QUERIES = [kg.KB_QUERY_RELAX, kg.KB_QUERY_EXACT]


def flock(n, w, h, seed):
    r = np.random.default_rng(seed)
    xy = (r.random((n, 2)) * [w * (1 - 1e-6), h * (1 - 1e-6)]).astype(np.float32)
    a = r.uniform(0, 2 * np.pi, n)
    return np.arange(n, dtype=np.uint32), xy, np.stack([np.cos(a), np.sin(a)], 1).astype(np.float32)


def plain(w, h, d, birds, mode=0):
    f = kg.Field2D(w, h, d, True)
    f.set_step_options(mode)
    f.set_locations(*birds)
    f.lazy_update()
    return f


def oracle_after(w, h, d, birds, p, steps):
    o = oracle.OracleField(w, h, d, True)
    o.set_many(*birds)
    o.lazy_update()
    o.flock_run(oracle.params_from(p), 0, steps)
    ids, st, _ = o.iter(1)
    return ids, st


def same(got, want):
    return np.array_equal(got[0], want[0]) and np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))


@pytest.mark.parametrize("kind", QUERIES)
@pytest.mark.parametrize("w,h", [(60.0, 40.0), (40.0, 60.0), (41.0, 40.0)])
@pytest.mark.parametrize("repeat", [False, True])
def test_cluster_sends_what_wide_rings_read(gpu, w, h, kind, repeat):
    # rings of 41 columns near half the side, whole steps in the cluster
    birds = flock(3000, w, h, 5)
    if repeat:
        birds[0][17] = birds[0][2900]
    p = kg.FlockParams(seed=2, arith=kg.KB_ARITH_STRICT, query_mode=kind, neighbor_radius=20.0, cohesion=0.0)
    f = plain(w, h, 1.0, birds)
    f.flock_step(p, 0, 1)
    f.flock_step(p, 1, 24)
    assert f.step_path() == kg.KB_PATH_SMALL
    assert same(f.get_state(), oracle_after(w, h, 1.0, birds, p, 25))
    f.close()


D = float(np.float32(10.0) / np.float32(1.5))
SHAPES = [(100.0, 60.0), (60.0, 100.0), (240.0, 200.0), (200.0, 240.0), (102.0, 100.0)]


@pytest.mark.parametrize("kind", QUERIES)
@pytest.mark.parametrize("w,h", SHAPES)
@pytest.mark.parametrize("mode", [0, 3])  # whole steps in the cluster, the separate kernels
@pytest.mark.parametrize("d,dense", [(D, False), (4.0, False), (1.5, False), (D, True)])
def test_steps_match_oracle(gpu, mode, w, h, kind, d, dense):
    birds = flock(900, w, h, int(w))
    p = kg.FlockParams(seed=4, arith=kg.KB_ARITH_STRICT, query_mode=kind)
    f = plain(w, h, d, birds, mode)
    f.set_dense_mode(kg.KB_DENSE_ON if dense else kg.KB_DENSE_OFF)
    f.flock_step(p, 0, 1)
    f.flock_step(p, 1, 14)
    assert same(f.get_state(), oracle_after(w, h, d, birds, p, 15))
    f.close()


@pytest.mark.parametrize("kind", QUERIES)
@pytest.mark.parametrize("w,h", [(480.0, 400.0), (400.0, 480.0)])
def test_larger_flocks_match_oracle(gpu, w, h, kind):
    birds = flock(6000, w, h, 1)
    p = kg.FlockParams(seed=4, arith=kg.KB_ARITH_STRICT, query_mode=kind)
    f = plain(w, h, D, birds)
    f.flock_step(p, 0, 10)
    assert same(f.get_state(), oracle_after(w, h, D, birds, p, 10))
    f.close()


@pytest.mark.parametrize("kind", QUERIES)
def test_fast_arithmetic_on_both_paths_is_the_same(gpu, kind):
    w, h = 200.0, 130.0
    birds = flock(900, w, h, 2)
    p = kg.FlockParams(seed=4, arith=kg.KB_ARITH_FAST, query_mode=kind)
    out = []
    for mode in (0, 3):
        f = plain(w, h, D, birds, mode)
        f.flock_step(p, 0, 15)
        out.append(f.get_state())
        f.close()
    assert same(*out)


@pytest.mark.parametrize("kind", QUERIES)
@pytest.mark.parametrize("d", [D, 4.0])
def test_packed_rectangles_match_oracle(gpu, kind, d):
    reps = []
    for i, (w, h) in enumerate(SHAPES):
        p = kg.FlockParams(seed=i, arith=kg.KB_ARITH_STRICT, query_mode=kind)
        reps.append(kg.Replica(w, h, d, p, flock(500 + i, w, h, 10 + i)))
    with kg.Batch(reps) as b:
        b.step(0, 12)
        for i, r in enumerate(reps):
            assert same(b.get_replica(i), oracle_after(r.width, r.height, d, r.state, r.params, 12))


@pytest.mark.parametrize("kind", QUERIES)
@pytest.mark.parametrize("w,h", SHAPES)
def test_queries_after_steps_match_oracle(gpu, w, h, kind):
    birds = flock(900, w, h, 7)
    p = kg.FlockParams(seed=4, arith=kg.KB_ARITH_STRICT)
    f = plain(w, h, D, birds)
    f.flock_step(p, 0, 15)
    o = oracle.OracleField(w, h, D, True)
    o.set_many(*birds)
    o.lazy_update()
    o.flock_run(oracle.params_from(p), 0, 15)
    r = np.random.default_rng(1)
    q = np.concatenate([f.get_state()[1][:, :2], r.uniform(-8.0, max(w, h) + 8.0, (300, 2))]).astype(np.float32)
    counts, ids = f.neighbor_lists(kind, 10.0, q)
    want = o.neighbor_lists(kind, 10.0, q)
    assert np.array_equal(counts, want[0]) and np.array_equal(ids, want[1])
    f.close()
