"""Wide rings (radius of many bags) on the warp-per-boid force kernel, and the
ranked rebin of moves longer than a bag, against the oracle: ring widths at a
warp's 32 columns, lists past 32 candidates, bags
of more arrivals than the slots hold."""
import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [kg.KB_QUERY_RELAX, kg.KB_QUERY_EXACT])
@pytest.mark.parametrize("n,side,d,radius,jump", [
    (1, 60.0, 0.5, 10.0, 0.7), (33, 60.0, 0.5, 10.0, 0.7), (700, 100.0, 0.5, 10.0, 0.7),
    (900, 90.0, 0.625, 10.0, 0.7),      # 33 columns
    (1200, 100.0, 2.0, 10.0, 2.5),      # moves over a bag, lists over 32
    (4097, 300.0, 3.0, 9.0, 0.7),
    (600, 20.0, 2.0, 4.5, 2.2),         # bags over twelve arrivals, long moves
])
def test_wide_rings_match_oracle(gpu, kind, n, side, d, radius, jump):
    r = np.random.default_rng(n)
    ids = np.arange(n, dtype=np.uint32)
    xy = r.uniform(0, side * (1 - 1e-6), (n, 2)).astype(np.float32)
    edge = r.random((n, 2)) < 0.2
    xy = np.where(edge, np.float32(d) * np.floor(xy / np.float32(d)), xy).astype(np.float32)
    a = r.uniform(0, 2 * np.pi, n)
    dxy = np.stack([np.cos(a), np.sin(a)], 1).astype(np.float32)
    p = kg.FlockParams(seed=n, arith=kg.KB_ARITH_STRICT, query_mode=kind, neighbor_radius=radius, jump=jump)
    f = kg.Field2D(side, side, d, True)
    f.set_step_options(3)
    f.set_dense_mode(kg.KB_DENSE_OFF)
    f.set_locations(ids, xy, dxy)
    f.lazy_update()
    f.flock_step(p, 0, 6)
    got = f.get_state()
    o = oracle.OracleField(side, side, d, True)
    o.set_many(ids, xy, dxy)
    o.lazy_update()
    o.flock_run(oracle.params_from(p), 0, 6)
    oids, ost, _ = o.iter(1)
    assert np.array_equal(got[0], oids) and np.array_equal(got[1].view(np.uint32), ost.view(np.uint32))
    assert f.device_flags() == 0
    f.close()


@pytest.mark.parametrize("kind", [kg.KB_QUERY_RELAX, kg.KB_QUERY_EXACT])
def test_wide_fast_steps_equal_the_general_kernel(gpu, kind):
    # one repeated id keeps the second flock on the general kernel
    n, side, d = 2000, 300.0, 2.0
    ids, xy, dxy = kg.gen_uniform(n, side, side, 5, 1.0)
    far = np.max(np.abs(xy - np.float32(150.0)), axis=1) < 100.0
    xy, dxy = xy[far], dxy[far]
    m = len(xy)
    xy = np.concatenate([xy, [[5.0, 5.0], [295.0, 295.0]]]).astype(np.float32)
    dxy = np.concatenate([dxy, [[1.0, 0.0], [0.0, 1.0]]]).astype(np.float32)
    p = kg.FlockParams(seed=2, arith=kg.KB_ARITH_FAST, query_mode=kind)
    out = []
    for last in (m + 1, m):
        i = np.arange(m + 2, dtype=np.uint32)
        i[-1] = last
        f = kg.Field2D(side, side, d, True)
        f.set_step_options(3)
        f.set_locations(i, xy, dxy)
        f.lazy_update()
        f.flock_step(p, 0, 3)
        gi, gs = f.get_state()
        out.append((gi[gi < m], gs[gi < m].view(np.uint32)))
        f.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
