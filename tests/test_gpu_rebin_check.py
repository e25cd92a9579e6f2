"""The ranked rebin's check of its source lines: an arrival of a fuller bag from
past them is reported, and moves at the limit of the rule are not."""
import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle

pytestmark = pytest.mark.gpu


def crowd(occ, side, d, seed):
    """Bags of `occ` birds at the far corner, at the seam's lines and inside,
    heading every way, with birds on the bags' edges."""
    r = np.random.default_rng(seed)
    far = side - 1.5 * d
    at = [(far, far), (far - 2 * d, far - d), (0.5 * d, far), (far, 0.5 * d), (0.5 * d, 0.5 * d), (side * 0.9, side * 0.8)]
    xy = np.concatenate([np.floor(np.asarray(c) / d) * d + r.choice([0.0, 0.3, 0.9999], (occ, 2)) * d for c in at])
    xy = np.clip(np.concatenate([xy, r.uniform(0, side, (200, 2))]), 0, side * (1 - 1e-6)).astype(np.float32)
    a = r.uniform(0, 2 * np.pi, len(xy))
    return np.arange(len(xy), dtype=np.uint32), xy, np.stack([np.cos(a), np.sin(a)], 1).astype(np.float32)


@pytest.mark.parametrize("occ", [13, 60])
@pytest.mark.parametrize("lines,d", [(40, 5.0), (2500, 1.0), (2500, 0.7)])
def test_moves_at_the_limit_match_oracle(gpu, occ, lines, d):
    d = float(np.float32(d))
    side = float(np.float32(lines) * np.float32(d))
    jump = float(np.nextafter(np.float32(d) / np.float32(1.001), np.float32(0)))
    birds = crowd(occ, side, d, lines)
    p = kg.FlockParams(seed=occ, arith=kg.KB_ARITH_STRICT, neighbor_radius=1.2 * d, jump=jump)
    f = kg.Field2D(side, side, d, True)
    f.set_step_options(3)
    f.set_dense_mode(kg.KB_DENSE_OFF)  # ranks, not segments
    f.set_locations(*birds)
    f.lazy_update()
    f.flock_step(p, 0, 4)
    got = f.get_state()
    assert f.device_flags() == 0
    f.close()
    o = oracle.OracleField(side, side, d, True)
    o.set_many(*birds)
    o.lazy_update()
    o.flock_run(oracle.params_from(p), 0, 4)
    ids, st, _ = o.iter(1)
    assert np.array_equal(got[0], ids) and np.array_equal(got[1].view(np.uint32), st.view(np.uint32))


@pytest.mark.parametrize("at", [(0.5, 0.5), (0.999, 0.999), (0.0, 0.5)])  # inside, at the seam, at the edge
def test_an_arrival_from_past_the_lines_is_reported(gpu, at):
    """A pass of long moves, then the parameters of short ones (another agent's
    query) before the buffers are exchanged: the rebuild trusts those."""
    torch = pytest.importorskip("torch")
    side, d, occ = 200.0, 5.0, 40
    c = np.clip(np.floor(np.asarray(at) * side / d) * d + 2.5, 2.5, side - 2.5)
    r = np.random.default_rng(1)
    here = c + r.uniform(-2.0, 2.0, (occ, 2))
    # birds that one move of 30 brings among them: nobody near, straight ahead
    far = np.mod(c + [30.0, 0.0], side) + r.uniform(-0.5, 0.5, (3, 2))
    xy = np.concatenate([here, far]).astype(np.float32)
    dxy = np.concatenate([np.zeros((occ, 2)), np.tile([[-1.0, 0.0]], (3, 1))]).astype(np.float32)
    f = kg.Field2D(side, side, d, True)
    f.set_dense_mode(kg.KB_DENSE_OFF)
    f.set_locations(np.arange(len(xy), dtype=np.uint32), xy, dxy)
    f.lazy_update()
    still = dict(arith=kg.KB_ARITH_STRICT, cohesion=0.0, avoidance=0.0, consistency=0.0, randomness=0.0,
                 neighbor_radius=1.0)
    f.flock_compute(kg.FlockParams(jump=30.0, **still), 0)
    one = torch.zeros((1, 4), dtype=torch.float32, device="cuda") + 10.0
    f.next_states_device(kg.FlockParams(jump=0.7, **still), 0, torch.zeros(1, dtype=torch.int32, device="cuda"), one)
    f.lazy_update()
    assert f.device_flags(clear=True) & kg.KB_FLAG_REBIN_MISS
    f.close()
