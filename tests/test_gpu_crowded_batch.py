"""Batches that are crowded (rebuilt by segments), that become so, that spread out
again and that mix both: every replica follows the oracle through captured and
uncaptured steps, growth and serving."""
import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle
from krabmaga_gb300 import _lib as L

pytestmark = pytest.mark.gpu
D = float(np.float32(10.0) / np.float32(1.5))


def replica(i, n, side, sigma, arith=kg.KB_ARITH_STRICT, **weights):
    birds = kg.gen_clustered(n, side, side, 1, sigma, 3.0, i) if sigma else kg.gen_uniform(n, side, side, i, 1.0)
    return kg.Replica(side, side, D, kg.FlockParams(seed=i, arith=arith, **weights), birds)


def follows(b, i, r, steps):
    o = oracle.OracleField(r.width, r.height, D, True)
    o.set_many(*r.state)
    o.lazy_update()
    o.flock_run(oracle.params_from(r.params), 0, steps)
    ids, st, _ = o.iter(1)
    got = b.get_replica(i)
    return np.array_equal(got[0], ids) and np.array_equal(got[1].view(np.uint32), st.view(np.uint32))


@pytest.mark.parametrize("graphs", [0, 8])
@pytest.mark.parametrize("sigma", [(4.0, 4.0, 4.0), (0.0, 4.0, 0.0), (0.0, 0.0, 0.0)])
def test_steps_of_crowded_batches(gpu, graphs, sigma):
    # a strong avoidance drives crowds apart, a strong cohesion makes them
    pull = dict(cohesion=3.0, avoidance=0.2)
    push = dict(cohesion=0.1, avoidance=5.0)
    reps = [replica(i, 400, 100.0, s, **(push if s else pull)) for i, s in enumerate(sigma)]
    with kg.Batch(reps) as b:
        done = 0
        for k in (30, 70, 60):
            b.step(done, k, graph_launches=graphs)
            done += k
            for i, r in enumerate(reps):
                assert follows(b, i, r, done), (done, i)


def test_a_crowd_joins_and_leaves(gpu):
    reps = [replica(0, 200, 150.0, 0.0), replica(1, 150, 90.0, 0.0)]
    late = replica(2, 1500, 90.0, 5.0)
    with kg.Batch(reps) as b:
        b.step(0, 6, graph_launches=6)
        b.add_replica(late, 6)
        b.step(6, 9, graph_launches=4)
        assert follows(b, 0, reps[0], 15) and follows(b, 2, late, 9)
        b.remove_replica(2)
        b.step(15, 8, graph_launches=8)
        assert follows(b, 0, reps[0], 23) and follows(b, 1, reps[1], 23)


def test_crowded_requests(gpu):
    reqs = [kg.Request(n, side, D, steps, kg.FlockParams(seed=n, arith=kg.KB_ARITH_FAST), 5 + n)
            for n, side, steps in ((2000, 60.0, 150), (3000, 80.0, 200), (300, 200.0, 170))]
    with kg.Server(max_slots=4, quantum_steps=16, max_request_boids=4000, max_request_cells=1 << 14) as srv:
        tickets = [srv.submit(r) for r in reqs]
        srv.wait_idle(60.0)
        for t, r in zip(tickets, reqs):
            f = kg.Field2D(r.side, r.side, D, True, capacity_hint=r.nboids)
            f.set_step_options(3)
            f.set_dense_mode(kg.KB_DENSE_OFF)
            f.set_locations(*kg.gen_uniform(r.nboids, r.side, r.side, r.init_seed, r.heading_scale))
            f.lazy_update()
            f.flock_step(r.params, 0, r.steps)
            got, want = srv.result(t, r.nboids), f.get_state()
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))
            f.close()


def test_a_server_that_cannot_measure_goes_on(gpu):
    """No memory for the measurement's words: the requests run all the same."""
    def ask(n, side, steps):
        return kg.Request(n, side, D, steps, kg.FlockParams(seed=n, arith=kg.KB_ARITH_FAST), n)

    with kg.Server(max_slots=4, quantum_steps=8, max_request_boids=4000, max_request_cells=1 << 14) as srv:
        # a larger batch first, for too few steps to be measured: all tables that the
        # one below needs are there (one request alone, so that both join it)
        srv.submit(ask(4000, 600.0, 16))
        srv.submit(ask(3999, 600.0, 40))
        srv.submit(ask(3998, 600.0, 40))
        srv.wait_idle(60.0)
        reqs = [ask(2000, 200.0, 160), ask(1500, 180.0, 200)]
        L.fail_allocations(1)
        try:
            tickets = [srv.submit(r) for r in reqs]
            srv.wait_idle(60.0)
        finally:
            L.fail_allocations(0)
        for t, r in zip(tickets, reqs):
            assert srv.poll(t)[0] == 2
            ids, st = srv.result(t, r.nboids)
            assert np.array_equal(np.sort(ids), np.arange(r.nboids)) and np.isfinite(st).all()
