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
