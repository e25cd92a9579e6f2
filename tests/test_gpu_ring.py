"""The ring force kernels: their shared-reciprocal quotients against IEEE
division, and whole steps against the oracle where their rules are decided (bag
edges, radii at the exact query's corner rule, list lengths, block edges)."""
import os
import subprocess

import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

QUOTIENTS = r"""
#include <cstdio>
#include "krabmaga_gb300/csrc/kb_device.cuh"
using namespace kb;
__global__ void recips(unsigned long long* bad, unsigned expo) {
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;  // 2^23 threads
    const float q = __uint_as_float((expo << 23) | m);
    if (recip_rn(q) != __frcp_rn(q)) atomicAdd(bad, 1ull);
}
__global__ void quotients(unsigned long long* bad, unsigned seed) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long n = 0;
    for (unsigned k = 0; k < 256; ++k) {
        const U4 u = philox4x32_10(U4{t, k, 0u, 7u}, seed, 0u);
        // any sign and significand; exponents around and past the bounds
        const float x = __uint_as_float((u.x & 0x807fffffu) | ((20u + u.z % 180u) << 23));
        const float y = __uint_as_float((u.y & 0x807fffffu) | ((60u + (u.z >> 8) % 70u) << 23));
        const float q = __uint_as_float((u.w >> 9) | ((127u + (u.z >> 16) % 80u) << 23));
        const float2 d = div2_rn(x, y, q, false);
        n += (__float_as_uint(d.x) != __float_as_uint(__fdiv_rn(x, q))) +
             (__float_as_uint(d.y) != __float_as_uint(__fdiv_rn(y, q)));
    }
    if (n) atomicAdd(bad + 1, n);
}
int main() {
    unsigned long long *d, h[2] = {0, 0};
    cudaMalloc(&d, 16);
    cudaMemset(d, 0, 16);
    for (unsigned e : {127u, 128u, 150u, 186u}) recips<<<(1u << 23) / 256, 256>>>(d, e);
    for (unsigned s = 0; s < 4; ++s) quotients<<<4096, 256>>>(d, s);
    if (cudaMemcpy(h, d, 16, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    printf("%llu %llu\n", h[0], h[1]);
    return 0;
}
"""


def test_shared_reciprocal_quotients_equal_ieee_division(gpu, tmp_path):
    src = tmp_path / "q.cu"
    src.write_text(QUOTIENTS)
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", f"-I{ROOT}",
                    str(src), "-o", str(tmp_path / "q")], check=True, capture_output=True)
    out = subprocess.run([str(tmp_path / "q")], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0", "0"]


def flock(n, side, d, seed):
    """A third of the boids on bag edges (multiples of d, one ulp beside them)."""
    r = np.random.default_rng(seed)
    xy = r.uniform(0.0, side, (n, 2)).astype(np.float32)
    edge = (np.float32(d) * r.integers(0, int(side / d), (n, 2)).astype(np.float32)).astype(np.float32)
    edge = np.where(r.random((n, 2)) < 0.3, np.nextafter(edge, np.float32(0)), edge).astype(np.float32)
    pick = r.random((n, 2)) < 1 / 3
    xy = np.clip(np.where(pick, edge, xy), 0, np.float32(side * (1 - 1e-6))).astype(np.float32)
    a = r.uniform(0, 2 * np.pi, n)
    return np.arange(n, dtype=np.uint32), xy, np.stack([np.cos(a), np.sin(a)], 1).astype(np.float32)


@pytest.mark.parametrize("kind", [kg.KB_QUERY_RELAX, kg.KB_QUERY_EXACT])
@pytest.mark.parametrize("n,ratio", [(1, 1.5), (127, 1.0), (129, 1.118034), (1500, 1.05), (1500, 1.5), (1500, 1.999),
                                     (1500, 0.6), (1500, 0.2), (3000, 1.1)])
def test_ring_steps_match_oracle(gpu, kind, n, ratio):
    side, d = 150.0, 5.0
    p = kg.FlockParams(seed=n, arith=kg.KB_ARITH_STRICT, query_mode=kind, neighbor_radius=d * ratio, jump=0.7)
    ids, xy, dxy = flock(n, side, d, int(100 * ratio))
    f = kg.Field2D(side, side, d, True)
    f.set_step_options(3)  # the separate kernels whatever the size
    f.set_locations(ids, xy, dxy)
    f.lazy_update()
    f.flock_step(p, 0, 3)
    g = f.get_state()
    o = oracle.OracleField(side, side, d, True)
    o.set_many(ids, xy, dxy)
    o.lazy_update()
    o.flock_run(oracle.params_from(p), 0, 3)
    oids, ost, _ = o.iter(1)
    assert np.array_equal(g[0], oids) and np.array_equal(g[1].view(np.uint32), ost.view(np.uint32))
    f.close()


@pytest.mark.parametrize("kind", [kg.KB_QUERY_RELAX, kg.KB_QUERY_EXACT])
@pytest.mark.parametrize("arith", [kg.KB_ARITH_STRICT, kg.KB_ARITH_FAST])
def test_ring_kernels_equal_the_general_kernel(gpu, kind, arith):
    # a repeated id far from every boid keeps the other flock on the general kernel
    side, d, n = 300.0, 10.0 / 1.5, 5000
    ids, xy, dxy = flock(n, side, d, 3)
    p = kg.FlockParams(seed=4, arith=arith, query_mode=kind)
    out = []
    for repeat in (False, True):
        i = ids.copy()
        keep = np.ones(n, bool)
        # two lone boids, opposite corners of the field, cleared around
        for c in ((20.0, 20.0), (280.0, 280.0)):
            keep &= np.max(np.abs(xy - np.float32(c)), axis=1) > 25.0
        i, x, h = i[keep], xy[keep], dxy[keep]
        i = np.concatenate([i, [n, n if repeat else n + 1]]).astype(np.uint32)
        x = np.concatenate([x, [[20.0, 20.0], [280.0, 280.0]]]).astype(np.float32)
        h = np.concatenate([h, [[1.0, 0.0], [0.0, 1.0]]]).astype(np.float32)
        f = kg.Field2D(side, side, d, True)
        f.set_step_options(3)
        f.set_locations(i, x, h)
        f.lazy_update()
        f.flock_step(p, 0, 2)
        gi, gs = f.get_state()
        rest = gi < n
        out.append((gi[rest], gs[rest].view(np.uint32)))
        f.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("d,radius", [(10.0 / 1.5, 10.0), (2.0, 9.0)])
@pytest.mark.parametrize("kind", [kg.KB_QUERY_RELAX, kg.KB_QUERY_EXACT])
def test_objects_apart_from_their_positions_match_oracle(gpu, kind, d, radius):
    # the first step reads bags that objects were set in, from wherever they are
    side, n = 100.0, 150
    r = np.random.default_rng(3)
    pos = r.uniform(0, side * (1 - 1e-6), (n, 2)).astype(np.float32)
    loc = pos.copy()
    # anywhere; under the relaxed query near enough that no pair straddles the seam
    reach = 15.0 if kind == kg.KB_QUERY_RELAX else side
    loc[::3] = np.clip(loc[::3] + r.uniform(-reach, reach, loc[::3].shape), 0, side * (1 - 1e-6)).astype(np.float32)
    f, o = kg.Field2D(side, side, d, True), oracle.OracleField(side, side, d, True)
    f.set_step_options(3)
    for i in range(n):
        b = kg.Bird(i, kg.Real2D(float(pos[i, 0]), float(pos[i, 1])), kg.Real2D(0.6, 0.8))
        f.set_object_location(b, kg.Real2D(float(loc[i, 0]), float(loc[i, 1])))
        o.set(i, pos[i, 0], pos[i, 1], 0.6, 0.8, loc[i, 0], loc[i, 1])
    f.lazy_update()
    o.lazy_update()
    q = r.uniform(-d, side + d, (400, 2)).astype(np.float32)
    gc, gi = f.neighbor_lists(kind, radius, q)
    oc, oi = o.neighbor_lists(kind, radius, q)
    assert np.array_equal(gc, oc) and np.array_equal(gi, oi)
    p = kg.FlockParams(seed=5, arith=kg.KB_ARITH_STRICT, query_mode=kind, neighbor_radius=radius)
    f.flock_step(p, 0, 3)
    o.flock_run(oracle.params_from(p), 0, 3)
    oids, ost, _ = o.iter(1)
    g = f.get_state()
    assert np.array_equal(g[0], oids) and np.array_equal(g[1].view(np.uint32), ost.view(np.uint32))
    f.close()
