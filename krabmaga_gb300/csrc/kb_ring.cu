// kb_ring.cu -- the force pass of flocks whose query spans at most one bag
// around the boid's own (radius < 2 d, the usual geometry) on a torus with the
// clamped range and distinct ids: k_flock_force's results bit for bit, for
// less issue per candidate.  Flocks of any other kind take k_flock_force.
//
// The walks are written for few instructions and loads:
//   * the boid itself stays in its list: its own terms are exact zeros (its
//     distance is zero, and a sum that starts at +0 never becomes -0), so only
//     its heading has to be held back, by one predicate;
//   * fast arithmetic: x and y travel together in packed f32x2 operations (one
//     issue slot for two IEEE results; the FMA pipe takes two cycles for it,
//     which the fast walk has to spare and the strict one has not);
//   * strict arithmetic: both quotients of a pair share one reciprocal
//     (div2_rn);
//   * exact query: distances are compared squared, with the largest square
//     whose root is within the radius (Rep::thr), and a bag's four corners are
//     classified from the extreme squares of its column and its row.
#include <cuda_runtime.h>
#include <stdint.h>

#include "kb_common.h"
#include "kb_device.cuh"
#include "kb_force.cuh"
#include "kb_launch.h"
#include "kb_walk.cuh"

namespace kb {
namespace {

// Relaxed query: bags mj..Mj of columns mi..Mi (cell_range, at most 3 x 3).
__device__ __forceinline__ void relaxed_runs(const ForceArgs& a, const Rep& R, int mi, int Mi, int mj,
                                             int Mj, Runs& r) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        r.s[k] = r.e[k] = 0u;
        if (mi + k <= Mi) {
            const uint32_t c = R.cell_off + (uint32_t)(mi + k) * (uint32_t)R.dh;
            r.e[k] = min(__ldg(a.start + c + Mj + 1), a.n);
            r.s[k] = min(__ldg(a.start + c + mj), r.e[k]);
        }
    }
}

// Long lists (dense flocks): column after column with a plain pointer, U
// candidates loaded together; only the agent's own column is tested for the
// agent itself.
template <bool STRICT, bool SELF, int U>
__device__ __forceinline__ void walk_run(const float4* st, pair_t<STRICT> me, uint32_t my, uint32_t s,
                                         uint32_t e, Sums<STRICT>& sums) {
    const float4* q = st + s;
    const float4* const end = st + e;
    uint32_t p = s;
    auto take = [&](const Candidate<STRICT>& o, uint32_t at) {
        const pair_t<STRICT> d = sub2(me, o.pos);
        sums.template add<SELF>(d, pair_sq<STRICT>(d), o.heading, at, my);
    };
#pragma unroll 1
    for (; end - q >= U; q += U, p += U) {
        Candidate<STRICT> o[U];
#pragma unroll
        for (int u = 0; u < U; ++u) o[u] = load_candidate<STRICT>(q + u);
#pragma unroll
        for (int u = 0; u < U; ++u) take(o[u], p + u);
    }
#pragma unroll 1
    for (; q < end; ++q, ++p) take(load_candidate<STRICT>(q), p);
}

template <bool STRICT, int U>
__device__ __forceinline__ void walk_runs(const ForceArgs& a, pair_t<STRICT> me, uint32_t my,
                                          const Runs& r, Sums<STRICT>& sums) {
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
        const uint32_t s = k == 0 ? r.s[0] : (k == 1 ? r.s[1] : r.s[2]);
        const uint32_t e = k == 0 ? r.e[0] : (k == 1 ? r.e[1] : r.e[2]);
        sums.vec += e - s;
        if (my - s < e - s) walk_run<STRICT, true, U>(a.st, me, my, s, e, sums);
        else walk_run<STRICT, false, U>(a.st, me, my, s, e, sums);
    }
}

// Long lists in fast arithmetic: the lanes of a warp stand in one bag or two
// neighbouring ones, so their lists overlap.  The warp copies the union of a
// column's runs to shared memory, STAGE records at a time, and every lane walks
// its own part of it there: a 16-byte shared load that most lanes share takes
// 2.4 cycles of the SM, a global one 4.3 (measured; 70 % of the L1 wavefronts of
// the walk from global memory).  Lanes too far apart (a column's end) walk from
// global memory.
constexpr uint32_t STAGE = 256;

template <bool STRICT, bool SELF, int U>
__device__ __forceinline__ void walk_staged(const float4* q, uint32_t n, uint32_t p, pair_t<STRICT> me,
                                            uint32_t my, Sums<STRICT>& sums) {
    auto take = [&](const Candidate<STRICT>& o, uint32_t at) {
        const pair_t<STRICT> d = sub2(me, o.pos);
        sums.template add<SELF>(d, pair_sq<STRICT>(d), o.heading, at, my);
    };
    const float4* const end = q + n;
#pragma unroll 1
    for (; end - q >= U; q += U, p += U) {
        Candidate<STRICT> o[U];
#pragma unroll
        for (int u = 0; u < U; ++u) o[u] = load_candidate<STRICT, false>(q + u);
#pragma unroll
        for (int u = 0; u < U; ++u) take(o[u], p + u);
    }
#pragma unroll 1
    for (; q < end; ++q, ++p) take(load_candidate<STRICT, false>(q), p);
}

// Every lane of the warp calls it (runs may be empty); stage: the warp's.
template <bool STRICT>
__device__ __forceinline__ void walk_shared(const ForceArgs& a, pair_t<STRICT> me, uint32_t my,
                                            const Runs& r, float4* stage, Sums<STRICT>& sums) {
    constexpr int U = 8;
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll 1
    for (int k = 0; k < 3; ++k) {
        const uint32_t s = k == 0 ? r.s[0] : (k == 1 ? r.s[1] : r.s[2]);
        const uint32_t e = k == 0 ? r.e[0] : (k == 1 ? r.e[1] : r.e[2]);
        const uint32_t len = e - s;
        sums.vec += len;
        const uint32_t us = __reduce_min_sync(0xffffffffu, len ? s : 0xFFFFFFFFu);
        const uint32_t ue = __reduce_max_sync(0xffffffffu, len ? e : 0u);
        const uint32_t longest = __reduce_max_sync(0xffffffffu, len);
        if (longest == 0u) continue;
        const bool self = __any_sync(0xffffffffu, my - s < len);
        if (ue - us > 2u * longest + STAGE) {
            if (my - s < len) walk_run<STRICT, true, U>(a.st, me, my, s, e, sums);
            else walk_run<STRICT, false, U>(a.st, me, my, s, e, sums);
            continue;
        }
#pragma unroll 1
        for (uint32_t c = us; c < ue; c += STAGE) {
            const uint32_t n = min(STAGE, ue - c);
            __syncwarp();
#pragma unroll
            for (uint32_t j = 0; j < STAGE; j += 32u)
                if (j + lane < n) stage[j + lane] = __ldg(a.st + c + j + lane);
            __syncwarp();
            const uint32_t lo = max(s, c), hi = min(e, c + n);
            if (lo < hi) {
                if (self) walk_staged<STRICT, true, U>(stage + (lo - c), hi - lo, lo, me, my, sums);
                else walk_staged<STRICT, false, U>(stage + (lo - c), hi - lo, lo, me, my, sums);
            }
        }
    }
}

template <bool STRICT, int BT, int MINB>
__global__ void __launch_bounds__(BT, MINB) k_flock_dense(ForceArgs a) {
    pdl_enter();
    __shared__ float4 s_stage[BT / 32][STAGE];
    const Rep& R = a.rep0;
    const uint32_t i = blockIdx.x * BT + threadIdx.x;
    const bool live = i < a.n;
    float4 me = make_float4(0.f, 0.f, 0.f, 0.f);
    Sums<STRICT> sums;
    Runs r = {{0u, 0u, 0u}, {0u, 0u, 0u}};
    if (live) {
        me = __ldg(a.st + i);
        int mi, Mi, mj, Mj;
        if (cell_range(R, me.x, me.y, R.dd, &mi, &Mi, &mj, &Mj)) relaxed_runs(a, R, mi, Mi, mj, Mj, r);
    }
    pair_t<STRICT> mxy;
    pack2(mxy, me.x, me.y);
    walk_shared<STRICT>(a, mxy, i, r, s_stage[threadIdx.x >> 5], sums);
    if (!live) return;
    const bool self_in = (i - r.s[0] < r.e[0] - r.s[0]) || (i - r.s[1] < r.e[1] - r.s[1]) ||
                         (i - r.s[2] < r.e[2] - r.s[2]);
    sums.count = sums.vec - (self_in ? 1u : 0u);
    force_finish<STRICT, false>(a, R, i, __ldg(a.st + i), __ldg(a.ids + i), *a.step, sums.result());
}

// How the relaxed query's lists are walked: as one flat list, run by run, or
// by the warp's own longest list (packed replicas, whose flocks differ).
enum Walk { WALK_FLAT, WALK_RUNS, WALK_VOTE };
constexpr uint32_t VOTE_LIST = 32;

template <bool STRICT, bool EXACT, Walk WALK, int U>
__device__ __forceinline__ void ring_body(const ForceArgs& a, const Rep& R, uint32_t i) {
    const unsigned long long step = *a.step;
    const float4 me = __ldg(a.st + i);
    const uint32_t my_id = __ldg(a.ids + i);
    Sums<STRICT> sums;
    int mi, Mi, mj, Mj;
    if (cell_range(R, me.x, me.y, R.dd, &mi, &Mi, &mj, &Mj)) {
        if (EXACT) {
            walk_exact<STRICT, U>(a.st, a.start, a.n, R, me, i, mi, Mi, mj, Mj, sums);
        } else {
            pair_t<STRICT> mxy;
            pack2(mxy, me.x, me.y);
            Runs r;
            relaxed_runs(a, R, mi, Mi, mj, Mj, r);
            const bool self_in = (i - r.s[0] < r.e[0] - r.s[0]) || (i - r.s[1] < r.e[1] - r.s[1]) ||
                                 (i - r.s[2] < r.e[2] - r.s[2]);
            const uint32_t T = (r.e[0] - r.s[0]) + (r.e[1] - r.s[1]) + (r.e[2] - r.s[2]);
            if (WALK == WALK_RUNS || (WALK == WALK_VOTE && __any_sync(__activemask(), T >= VOTE_LIST)))
                walk_runs<STRICT, 4>(a, mxy, i, r, sums);
            else
                walk_flat<STRICT, U>(a.st, mxy, i, r, sums);
            sums.count = sums.vec - (self_in ? 1u : 0u);
        }
    }
    force_finish<STRICT, WALK != WALK_RUNS>(a, R, i, me, my_id, step, sums.result());
}

template <bool STRICT, bool EXACT, Walk WALK, bool MULTI, int U, int BT, int MINB>
__global__ void __launch_bounds__(BT, MINB) k_flock_ring(ForceArgs a) {
    pdl_enter();
    if (MULTI) {
        // one replica per block: its record is read once into shared memory
        __shared__ Rep sR;
        const uint2 e = a.blk[blockIdx.x];
        load_rep_shared(&sR, a.reps + e.x);
        __syncthreads();
        const uint32_t k = e.y + threadIdx.x;
        if (k >= sR.boid_off + sR.nboids) return;
        ring_body<STRICT, EXACT, WALK, U>(a, sR, k);
    } else {
        const uint32_t i = blockIdx.x * BT + threadIdx.x;
        if (i >= a.n) return;
        ring_body<STRICT, EXACT, WALK, U>(a, a.rep0, i);
    }
}

// Launch shapes, measured on GB300 (us per step, density 0.025 unless said):
//   * up to SMALL_N boids the pass is bound by latency: 128-thread blocks of up
//     to 64 registers, the strict walk two candidates at a time (20k 8.2, 262k
//     15.3; the throughput shape 8.3 and 16.8; 65k strict 10.8 with two at a
//     time, 11.4 with one; fast 9.0 with one, 9.7 with two);
//   * above it by issue: fast 32 registers and all 64 warps (1M 40.6; 40 and 48
//     registers 42.1), strict 48 registers (1M 54.4; 40 and 64 registers 56 to
//     58).  k_flock_force: 42.6 and 61.7;
//   * exact query, 65k strict: 12.4 against 30 for k_flock_force;
//   * long lists, strict (131k clustered): 115 against 156 with 4 candidates
//     loaded together and 64 registers (2 and 48: 128).  Two boids of a bag per
//     thread, sharing the loads, leave lanes idle where bags end: not kept;
//   * long lists, fast: the walk through shared memory, 256 records a stage, 8
//     together, 64 registers: force pass of 4M clustered boids 662 us, 763 for
//     k_flock_force (1M of them: 193 against 228; stages of 64, 128 and 384
//     records 235, 215 and 193, 4 together 204, 74 registers 196).
//   * packed replicas: 48 registers and the walk by vote.  64 replicas, steps
//     0-100 / 400-500 (condensed flocks): 74.8 / 93.4 us, flat walk 78.7 / 108.6,
//     k_flock_force 78.6 / 106.0; from 24 or 40 candidates the same, from 64
//     79.9 / 98.5; two or eight candidates together 77.9 / 100.0, 78.1 / 94.8.
constexpr uint32_t SMALL_N = 400000;

template <bool STRICT, bool EXACT>
cudaError_t launch_ring(const ForceArgs& a, cudaStream_t s) {
    // resident blocks of 256 threads per SM
    constexpr int MINB = EXACT ? 4 : (STRICT ? 5 : 8);
    constexpr int MM = EXACT ? 4 : 5;  // packed replicas
    if (a.nrep > 1) {
        if (a.block_threads == 128)
            return launch_pdl(k_flock_ring<STRICT, EXACT, WALK_VOTE, true, 1, 128, 2 * MM>, a.nblk, 128, s, a);
        if (a.block_threads == 512)
            return launch_pdl(k_flock_ring<STRICT, EXACT, WALK_VOTE, true, 1, 512, MM / 2>, a.nblk, 512, s, a);
        return launch_pdl(k_flock_ring<STRICT, EXACT, WALK_VOTE, true, 1, 256, MM>, a.nblk, 256, s, a);
    }
    const unsigned g = grid_for(a.n, 128);
    if constexpr (!STRICT && !EXACT)
        if (a.dense) return launch_pdl(k_flock_dense<false, 128, 8>, g, 128, s, a);
    if constexpr (STRICT && !EXACT)
        if (a.dense) return launch_pdl(k_flock_ring<true, false, WALK_RUNS, false, 1, 128, 8>, g, 128, s, a);
    if (a.n <= SMALL_N)
        return launch_pdl(k_flock_ring<STRICT, EXACT, WALK_FLAT, false, STRICT ? 2 : 1, 128, 8>, g, 128, s, a);
    return launch_pdl(k_flock_ring<STRICT, EXACT, WALK_FLAT, false, 1, 128, 2 * MINB>, g, 128, s, a);
}

}  // namespace

cudaError_t launch_flock_ring(const ForceArgs& a, bool strict, int qmode, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    if (a.nrep > 1 && a.blk == nullptr) return cudaErrorInvalidValue;
    if (qmode == 0) return strict ? launch_ring<true, false>(a, s) : launch_ring<false, false>(a, s);
    return strict ? launch_ring<true, true>(a, s) : launch_ring<false, true>(a, s);
}

}  // namespace kb
