"""The ranked rebin (arrival slots of the force pass) against the oracle at the
edges of its rows: bags of 1 to 4, 5 to 12 and more than 12 arrivals, in the
interior, at the field's edge and at the seam, plain and packed."""
import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle

pytestmark = pytest.mark.gpu
D = float(np.float32(10.0) / np.float32(1.5))


def crowded(occ, side, seed):
    """`occ` boids around each of a few bag centres: the corner, the last
    lines (seam moves) and the interior; plus scattered ones."""
    r = np.random.default_rng(seed)
    last = side - 0.4 * D
    centres = [(0.3, 0.3), (0.3, last), (last, last), (side / 2, side / 2), (side / 2, 0.3), (9.5 * D, 12.5 * D)]
    pts = [np.asarray(c) + r.uniform(-0.3, 0.3, (occ, 2)) for c in centres]
    pts.append(r.uniform(0.0, side, (57, 2)))
    xy = np.clip(np.concatenate(pts), 0.0, side * (1 - 1e-6)).astype(np.float32)
    a = r.uniform(0.0, 2 * np.pi, len(xy))
    dxy = np.stack([np.cos(a), np.sin(a)], 1).astype(np.float32)
    order = r.permutation(len(xy))
    return np.arange(len(xy), dtype=np.uint32), xy[order], dxy[order]


def oracle_state(flock, side, p, steps):
    o = oracle.OracleField(side, side, D, True)
    o.set_many(*flock)
    o.lazy_update()
    o.flock_run(oracle.params_from(p), 0, steps)
    ids, st, _ = o.iter(1)
    return ids, st


def same(got, want):
    return np.array_equal(got[0], want[0]) and np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))


@pytest.mark.parametrize("occ", [1, 4, 5, 8, 9, 12, 13, 45, 131, 300])
def test_ranks_at_row_edges_match_oracle(gpu, occ):
    side, steps = 200.0, 4
    flock = crowded(occ, side, occ)
    p = kg.FlockParams(seed=occ, arith=kg.KB_ARITH_STRICT)
    f = kg.Field2D(side, side, D, True)
    f.set_step_options(3)  # the separate kernels whatever the size
    f.set_dense_mode(kg.KB_DENSE_OFF)  # ranks, not segments
    f.set_locations(*flock)
    f.lazy_update()
    f.flock_step(p, 0, steps)
    assert same(f.get_state(), oracle_state(flock, side, p, steps))
    assert f.device_flags() == 0
    f.close()


@pytest.mark.parametrize("occ", [4, 13, 140])
def test_packed_ranks_match_oracle(gpu, occ):
    reps = []
    for i, side in enumerate((200.0, 130.0, 260.0)):
        p = kg.FlockParams(seed=i, arith=kg.KB_ARITH_STRICT)
        reps.append(kg.Replica(side, side, D, p, crowded(occ + i, side, 10 * occ + i)))
    with kg.Batch(reps) as b:
        b.step(0, 4)
        for i, r in enumerate(reps):
            assert same(b.get_replica(i), oracle_state(r.state, r.width, r.params, 4))


@pytest.mark.parametrize("max_cells", [1 << 13, 1 << 24])
def test_server_slots_follow_the_batch(gpu, max_cells):
    """Slots for the whole bag capacity (2^16) and for the bags in use (a
    capacity of 2^27): a batch that grows, grows again and shrinks."""
    reqs = [kg.Request(n, side, D, steps, kg.FlockParams(seed=n, arith=kg.KB_ARITH_FAST), 7 + n)
            for n, side, steps in ((300, 110.0, 40), (5000, 400.0, 21), (2000, 90.0, 33), (9, 500.0, 50))]
    with kg.Server(max_slots=8, quantum_steps=8, max_request_boids=6000, max_request_cells=max_cells) as srv:
        tickets = [srv.submit(reqs[0])]
        srv.wait_idle(60.0)
        tickets += [srv.submit(r) for r in reqs[1:]]
        srv.wait_idle(60.0)
        for t, r in zip(tickets, reqs):
            f = kg.Field2D(r.side, r.side, D, True, capacity_hint=r.nboids)
            f.set_locations(*kg.gen_uniform(r.nboids, r.side, r.side, r.init_seed, r.heading_scale))
            f.lazy_update()
            f.flock_step(r.params, 0, r.steps)
            assert same(srv.result(t, r.nboids), f.get_state())
            f.close()
