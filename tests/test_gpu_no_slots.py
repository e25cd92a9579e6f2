"""Fields and batches that cannot have arrival slots (out of device memory) work
as they do with them: each allocation in turn is made to fail."""
import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle
from krabmaga_gb300 import _lib as L

pytestmark = pytest.mark.gpu
SIDE, D = 200.0, float(np.float32(10.0) / np.float32(1.5))
P = kg.FlockParams(seed=3, arith=kg.KB_ARITH_STRICT)


def counted(make):
    """make()'s result and how many allocations it made."""
    a = L.allocation_counts()[0]
    return make(), L.allocation_counts()[0] - a


def injected(skip, make):
    """(result or None, allocations) with the allocation after `skip` failing."""
    L.fail_allocations(1, skip)
    try:
        return counted(make)
    except kg.KbError as e:
        assert e.status == L.KB_ERR_OOM
        return None, 0
    finally:
        L.fail_allocations(0)


def same(got, want):
    return np.array_equal(got[0], want[0]) and np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))


def oracle_after(birds, steps, side=SIDE, p=P):
    o = oracle.OracleField(side, side, D, True)
    o.set_many(*birds)
    o.lazy_update()
    o.flock_run(oracle.params_from(p), 0, steps)
    return o.iter(1)[:2]


def steps_follow_the_oracle(f):
    birds = kg.gen_uniform(1000, SIDE, SIDE, 1, 1.0)
    f.set_step_options(3)
    f.set_locations(*birds)
    f.lazy_update()
    assert same(f.get_state(), oracle_after(birds, 0))
    f.flock_step(P, 0, 3)
    f.flock_compute(P, 3)
    f.lazy_update()
    f.flock_step(P, 4, 5)
    assert same(f.get_state(), oracle_after(birds, 9))
    assert f.device_flags() == 0
    f.close()


def test_a_field_without_slots(gpu):
    def make():
        return kg.Field2D(SIDE, SIDE, D, True, capacity_hint=1000)

    f, usual = counted(make)
    f.close()
    fewer = 0
    for skip in range(usual):
        f, made = injected(skip, make)
        if f is not None:
            fewer += made < usual
            steps_follow_the_oracle(f)
    assert fewer == 1  # only the slots may be missing


def test_a_load_that_needs_their_memory(gpu):
    f = kg.Field2D(SIDE, SIDE, D, True)
    L.fail_allocations(1)  # the load's own storage: the slots make room for it
    try:
        steps_follow_the_oracle(f)
    finally:
        L.fail_allocations(0)


def test_a_batch_that_grows_without_slots(gpu):
    def replica(i, side, n):
        return kg.Replica(side, side, D, kg.FlockParams(seed=i, arith=kg.KB_ARITH_STRICT),
                          kg.gen_uniform(n, side, side, i, 1.0))

    first, late = replica(0, 100.0, 300), replica(1, 300.0, 900)

    def start():
        b = kg.Batch([first])
        b.step(0, 2)
        return b

    b = start()
    _, usual = counted(lambda: b.add_replica(late, 2))
    b.close()
    fewer = 0
    for skip in range(usual):
        b = start()
        got, made = injected(skip, lambda: b.add_replica(late, 2))
        if got is not None:
            fewer += made < usual
            b.step(2, 6)
            assert same(b.get_replica(0), oracle_after(first.state, 8, 100.0, first.params))
            assert same(b.get_replica(1), oracle_after(late.state, 6, 300.0, late.params))
        b.close()
    assert fewer >= 1


@pytest.mark.parametrize("max_cells", [1 << 14, 1 << 24])
def test_a_server_keeps_slots_within_its_budget(gpu, max_cells):
    """A request that fills the budget runs by segments; with room, by ranks."""
    n, side = 3000, 400.0
    r = kg.Request(n, side, D, 40, kg.FlockParams(seed=5, arith=kg.KB_ARITH_FAST), 11)
    cells = (int(np.ceil(np.float32(side) / np.float32(D))) + 1) ** 2
    one = 120 * n + 16 * cells
    out = []
    for budget in (one + 47 * cells, one + 48 * cells):
        with kg.Server(max_slots=8, quantum_steps=8, max_request_boids=n, max_request_cells=max_cells,
                       hbm_budget_bytes=budget) as srv:
            a = L.allocation_counts()[0]
            t = srv.submit(r)
            srv.wait_idle(60.0)
            out.append((srv.result(t, n), L.allocation_counts()[0] - a))
    assert same(out[0][0], out[1][0])
    assert out[1][1] == out[0][1] + 1
