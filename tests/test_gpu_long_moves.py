"""Moves past the neighbouring bag in flocks too large for the ranked rebin of
any move: the general rebuild by a force pass's own counts, with its arrival
slots and without, against the oracle."""
import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dense", [kg.KB_DENSE_OFF, kg.KB_DENSE_ON])  # with arrival slots, without
@pytest.mark.parametrize("occ", [1, 12, 13, 40, 300])
def test_general_rebuild_of_a_pass_matches_oracle(gpu, occ, dense):
    n, side, d = 32769, 600.0, 5.0
    r = np.random.default_rng(occ)
    xy = r.uniform(0, side * (1 - 1e-6), (n, 2)).astype(np.float32)
    for k, c in enumerate(((2.5, 2.5), (302.5, 77.5), (597.5, 597.5))):
        xy[k * occ:(k + 1) * occ] = np.asarray(c) + r.uniform(-2.0, 2.0, (occ, 2))
    order = r.permutation(n)
    xy = xy[order]
    a = r.uniform(0, 2 * np.pi, n)
    birds = np.arange(n, dtype=np.uint32), xy, np.stack([np.cos(a), np.sin(a)], 1).astype(np.float32)
    # a short sight keeps the crowds together while each bird moves past a bag
    p = kg.FlockParams(seed=occ, arith=kg.KB_ARITH_STRICT, neighbor_radius=4.0, jump=6.0)
    f = kg.Field2D(side, side, d, True)
    f.set_dense_mode(dense)
    f.set_locations(*birds)
    f.lazy_update()
    f.flock_step(p, 0, 2)
    f.flock_compute(p, 2)
    f.lazy_update()
    f.flock_step(p, 3, 5)  # replayed from a graph
    got = f.get_state()
    assert f.device_flags() == 0
    f.close()
    o = oracle.OracleField(side, side, d, True)
    o.set_many(*birds)
    o.lazy_update()
    o.flock_run(oracle.params_from(p), 0, 8)
    ids, st, _ = o.iter(1)
    assert np.array_equal(got[0], ids) and np.array_equal(got[1].view(np.uint32), st.view(np.uint32))


@pytest.mark.parametrize("occ", [13, 60])
def test_packed_long_moves_match_oracle(gpu, occ):
    side, d = 100.0, 5.0
    reps = []
    for i in range(3):
        r = np.random.default_rng(10 * occ + i)
        xy = np.concatenate([r.uniform(0, side, (400, 2)), 52.5 + r.uniform(-2, 2, (occ, 2))])
        xy = np.clip(xy, 0, side * (1 - 1e-6)).astype(np.float32)
        a = r.uniform(0, 2 * np.pi, len(xy))
        birds = np.arange(len(xy), dtype=np.uint32), xy, np.stack([np.cos(a), np.sin(a)], 1).astype(np.float32)
        p = kg.FlockParams(seed=i, arith=kg.KB_ARITH_STRICT, neighbor_radius=4.0, jump=6.0 + i)
        reps.append(kg.Replica(side, side, d, p, birds))
    with kg.Batch(reps) as b:
        b.step(0, 5)
        for i, q in enumerate(reps):
            o = oracle.OracleField(side, side, d, True)
            o.set_many(*q.state)
            o.lazy_update()
            o.flock_run(oracle.params_from(q.params), 0, 5)
            ids, st, _ = o.iter(1)
            got = b.get_replica(i)
            assert np.array_equal(got[0], ids) and np.array_equal(got[1].view(np.uint32), st.view(np.uint32))
