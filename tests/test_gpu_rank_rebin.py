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


@pytest.mark.parametrize("occ", [1, 4, 5, 8, 9, 12, 13, 45])
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


@pytest.mark.parametrize("occ", [4, 13])
def test_packed_ranks_match_oracle(gpu, occ):
    reps = []
    for i, side in enumerate((200.0, 130.0, 260.0)):
        p = kg.FlockParams(seed=i, arith=kg.KB_ARITH_STRICT)
        reps.append(kg.Replica(side, side, D, p, crowded(occ + i, side, 10 * occ + i)))
    with kg.Batch(reps) as b:
        b.step(0, 4)
        for i, r in enumerate(reps):
            assert same(b.get_replica(i), oracle_state(r.state, r.width, r.params, 4))
