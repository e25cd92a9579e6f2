"""The rules that choose between the warp-per-boid kernel, the general one and
the cluster: on the side that was measured the faster, and the oracle's bits on
both sides of each line."""
import os
import subprocess

import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "krabmaga_gb300", "csrc")
RELAX, EXACT = kg.KB_QUERY_RELAX, kg.KB_QUERY_EXACT
# (bags around the own one, query, boids): sizes timed at which each side was the faster
WIDE = [(2, RELAX, 12000), (3, RELAX, 16000), (10, RELAX, 32768), (2, EXACT, 32768), (3, EXACT, 65536),
        (4, EXACT, 131072), (5, EXACT, 262144), (20, EXACT, 131072)]
GENERAL = [(2, RELAX, 16384), (3, RELAX, 32000), (2, EXACT, 49152), (2, EXACT, 262144), (3, EXACT, 98304),
           (3, EXACT, 262144)]


def test_wide_rule_is_on_the_measured_side(tmp_path):
    src = tmp_path / "rule.cpp"
    src.write_text('#include <cstdio>\n#include "kb_launch.h"\nint main() { int dd, q;\n'
                   'while (std::scanf("%d %d", &dd, &q) == 2) std::printf("%u\\n", kb::wide_max(dd, q)); }\n')
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = str(tmp_path / "rule")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I", cuda + "/include", "-o", exe, str(src)], check=True)
    rows = WIDE + GENERAL
    text = "".join(f"{dd} {q}\n" for dd, q, _ in rows)
    most = subprocess.run([exe], input=text, check=True, capture_output=True, text=True).stdout.split()
    for (dd, q, n), m in zip(rows, most):
        assert (n <= int(m)) == ((dd, q, n) in WIDE), (dd, q, n, m)


def after(side, d, birds, p, steps):
    o = oracle.OracleField(side, side, d, True)
    o.set_many(*birds)
    o.lazy_update()
    o.flock_run(oracle.params_from(p), 0, steps)
    return o.iter(1)[:2]


def same(got, want):
    return np.array_equal(got[0], want[0]) and np.array_equal(got[1].view(np.uint32), want[1].view(np.uint32))


@pytest.mark.gpu
@pytest.mark.parametrize("over", [0, 1])
@pytest.mark.parametrize("n,d,kind", [(12288, 4.0, RELAX), (40000, 4.0, EXACT), (65536, 3.0, EXACT), (131072, 2.5, EXACT)])
def test_both_sides_of_the_wide_rule_match_oracle(gpu, n, d, kind, over):
    n += over
    side = float(np.float32(np.sqrt(n / 0.025)))
    birds = kg.gen_uniform(n, side, side, n, 1.0)
    p = kg.FlockParams(seed=1, arith=kg.KB_ARITH_STRICT, query_mode=kind)
    f = kg.Field2D(side, side, d, True)
    f.set_locations(*birds)
    f.lazy_update()
    f.flock_step(p, 0, 2)
    assert same(f.get_state(), after(side, d, birds, p, 2))
    f.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,kind,path", [(600, RELAX, kg.KB_PATH_SMALL), (600, EXACT, kg.KB_PATH_SMALL),
                                         (1999, RELAX, kg.KB_PATH_SMALL), (2000, RELAX, kg.KB_PATH_DENSE),
                                         (2000, EXACT, kg.KB_PATH_SMALL), (4096, EXACT, kg.KB_PATH_SMALL)])
def test_dense_wide_rings_of_small_fields(gpu, n, kind, path):
    # crowded: the warp-per-boid kernel, for which wide rings leave the cluster, is not taken
    side, d = float(np.float32(np.sqrt(n / 1.0))), 4.0
    side = max(side, 32.0)
    birds = kg.gen_clustered(n, side, side, 1, 6.0, 0.5, 3)
    p = kg.FlockParams(seed=2, arith=kg.KB_ARITH_STRICT, query_mode=kind, neighbor_radius=10.0)
    f = kg.Field2D(side, side, d, True)
    f.set_locations(*birds)
    f.lazy_update()
    f.flock_step(p, 0, 2)
    f.flock_step(p, 2, 2)
    assert f.dense_active() and f.step_path() == path
    assert same(f.get_state(), after(side, d, birds, p, 4))
    f.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [RELAX, EXACT])
@pytest.mark.parametrize("n", [1200, 1201, 4096])
def test_single_steps_and_runs_of_small_fields_mix(gpu, n, kind):
    # one step at a time on either side of the cluster's limit, runs between them
    side, d = float(np.float32(np.sqrt(n / 0.025))), float(np.float32(10.0) / np.float32(1.5))
    birds = kg.gen_uniform(n, side, side, 4, 1.0)
    p = kg.FlockParams(seed=6, arith=kg.KB_ARITH_STRICT, query_mode=kind)
    f = kg.Field2D(side, side, d, True)
    f.set_locations(*birds)
    f.lazy_update()
    done = 0
    for k in (1, 1, 3, 1, 5, 1):
        f.flock_step(p, done, k)
        done += k
    assert same(f.get_state(), after(side, d, birds, p, done))
    f.close()
