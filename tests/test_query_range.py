"""The bags that a query looks at, at the limits of the i32 bag coordinates: a
point may lie anywhere, and a far one's coordinate saturates.  The device's
cell_range compiled on the host, and (on a GPU) far points and far agents."""
import os
import re
import subprocess

import numpy as np
import pytest

import krabmaga_gb300 as kg
import oracle
from conftest import FLOCK_D

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "krabmaga_gb300", "csrc")
FAR = [3e9, 1.4316557e10, 1e12, 3e38]

HOST = r"""
#include <algorithm>
#include <cmath>
#include <climits>
#include <cstdio>
#include "kb_common.h"
#define __device__
#define __forceinline__ inline
using std::max; using std::min;
namespace kb {
inline int32_t disc(float v, const Rep& R) { return as_i32(std::floor(v / R.d)); }
%s
}
int main() {
    using namespace kb;
    const float at[] = {0.f, 1.f, 57.f, 99.f, 100.f, 104.f, -1.f, -7.f, -1e6f, 1e6f, 2.147483e9f, -2.147483e9f,
                        2.2e9f, -2.2e9f, 3e9f, -3e9f, 1e12f, -1e12f, 3e38f, -3e38f, INFINITY, -INFINITY, NAN};
    const int rings[] = {0, 1, 2, 7, INT_MAX};
    int bad = 0, some = 0;
    for (int wrap = 0; wrap < 2; ++wrap)
        for (float x : at)
            for (float y : at)
                for (int dd : rings) {
                    Rep R{};
                    R.w = R.h = 100.f;
                    R.d = 1.f;
                    R.toroidal = wrap ? 0 : 1;
                    R.max_x = R.max_y = 100;
                    R.dw = R.dh = 101;
                    int mi, Mi, mj, Mj;
                    if (!cell_range(R, x, y, dd, &mi, &Mi, &mj, &Mj)) continue;
                    ++some;
                    // a walk may rely on it: lines of the matrix, none out of order
                    if (mi > Mi || mj > Mj || Mi == INT_MAX || Mj == INT_MAX) ++bad;
                    // (a line moved to end the walk is the same one)
                    else if (wrap && dd == 0 && (t_transform(mi, 100) != t_transform(disc(x, R), 100) ||
                                                 t_transform(mj, 100) != t_transform(disc(y, R), 100))) ++bad;
                    else if (!wrap && (mi < 0 || Mi > 99 || mj < 0 || Mj > 99)) ++bad;
                }
    std::printf("%%d %%d\n", bad, some > 0);
    return 0;
}
"""


def test_ranges_are_lines_of_the_matrix(tmp_path):
    text = open(os.path.join(CSRC, "kb_device.cuh")).read()
    fn = re.search(r"__device__ __forceinline__ bool cell_range\(.*?\n}\n", text, re.S).group(0)
    src = tmp_path / "range.cpp"
    src.write_text(HOST % fn)
    exe = str(tmp_path / "range")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fwrapv", "-I", CSRC, "-o", exe, str(src)], check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split() == ["0", "1"]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [kg.KB_QUERY_RELAX, kg.KB_QUERY_EXACT])
@pytest.mark.parametrize("toroidal,dist", [(True, 10.0), (True, 5.0), (True, 20.0), (False, 10.0)])
def test_far_points_find_nothing(gpu, kind, toroidal, dist):
    n, side = 2000, 200.0
    f = kg.Field2D(side, side, FLOCK_D, toroidal)
    birds = kg.gen_uniform(n, side, side, 3, 1.0)
    f.set_locations(*birds)
    f.lazy_update()
    o = oracle.OracleField(side, side, FLOCK_D, toroidal)
    o.set_many(*birds)
    o.lazy_update()
    near = [[100.0, 100.0], [0.0, 199.9]]
    far = [[s * v, y] for v in FAR for s in (1.0, -1.0) for y in (100.0, v)] + [[100.0, v] for v in FAR]
    if not toroidal:  # a bounded field's saturated range wraps into the matrix, as the reference's does
        far = [q for q in far if min(abs(q[0]), abs(q[1])) > 2.2e10]
    q = np.array(far + near, np.float32)
    counts, ids = f.neighbor_lists(kind, dist, q)
    dc, _ = f.neighbor_digest(kind, dist, q)
    assert not counts[:len(far)].any() and np.array_equal(counts, dc)
    want = o.neighbor_lists(kind, dist, near)
    assert np.array_equal(counts[len(far):], want[0]) and np.array_equal(ids, want[1])
    assert f.device_flags() == 0
    f.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [kg.KB_QUERY_RELAX, kg.KB_QUERY_EXACT])
def test_far_agents_see_nobody(gpu, kind):
    """Agents held by the caller may stand anywhere too: far ones move as they
    do in a field of one distant bird."""
    torch = pytest.importorskip("torch")
    n, side = 2000, 200.0
    at = [[s * v, y, 0.6, 0.8] for v in FAR[:3] for s in (1.0, -1.0) for y in (50.0, v)]
    st = torch.tensor(at, dtype=torch.float32, device="cuda")
    ids = torch.arange(len(at), dtype=torch.int32, device="cuda") + n
    p = kg.FlockParams(seed=8, arith=kg.KB_ARITH_STRICT, query_mode=kind)
    out = []
    for flock in (kg.gen_uniform(n, side, side, 3, 1.0), kg.gen_uniform(1, 1.0, 1.0, 3, 1.0)):
        f = kg.Field2D(side, side, FLOCK_D, True)
        f.set_locations(*flock)
        f.lazy_update()
        out.append(f.next_states_device(p, 0, ids, st).cpu().numpy().view(np.uint32))
        f.close()
    assert np.array_equal(out[0], out[1])
