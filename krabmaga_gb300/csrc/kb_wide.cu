// kb_wide.cu -- the force pass of small flocks whose query spans many bags
// (radius >= 2 d: the model's default bag of 0.5 makes it 41 x 41), on a torus
// with the clamped range and distinct ids: k_flock_force's results bit for bit.
//
// With a thread per boid the pass is a chain of dependent loads, two offsets
// for each of the ring's columns before the few candidates are known (1,000
// boids, 41 columns: 44 us, now 4).  Here a warp takes a boid: its lanes load the
// bounds of 32 columns at once, then 32 candidates at once, and work out their
// terms in parallel; the sums are then taken over the terms in list order, one
// sum per lane, so every addition is the one the serial walk makes.  A candidate
// that does not count (the boid itself; outside the exact query) leaves zeros,
// which no sum that starts at +0 can tell from nothing.
#include <cuda_runtime.h>
#include <stdint.h>

#include "kb_common.h"
#include "kb_device.cuh"
#include "kb_force.cuh"
#include "kb_launch.h"

namespace kb {
namespace {

constexpr int WIDE_WARPS = 4;  // per block
constexpr uint32_t WIDE_FULL = 0xFFFFFFFFu;

// The class of the bag of column c0 that holds slot p (check_circle): the row
// is the candidate's own unless its bag is another one.
__device__ __forceinline__ int bag_class(const ForceArgs& a, const Rep& R, int bx, uint32_t c0, int mj,
                                         int Mj, uint32_t p, float4 me, float4 o) {
    int by = disc(o.y, R);
    if (by < mj || by > Mj || p < __ldg(a.start + c0 + by) || p >= __ldg(a.start + c0 + by + 1)) {
        int lo = mj, hi = Mj;  // the last row that starts at or before p
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(a.start + c0 + mid) <= p) lo = mid;
            else hi = mid - 1;
        }
        by = lo;
    }
    return check_circle(bx, by, R, me.x, me.y, R.radius);
}

template <bool STRICT, bool EXACT>
__global__ void __launch_bounds__(32 * WIDE_WARPS) k_flock_wide(ForceArgs a) {
    pdl_enter();
    // terms of 32 candidates: two avoidance, two cohesion, two consistency, the
    // avoidance factor (fast arithmetic fuses it into the sum)
    __shared__ float s_term[WIDE_WARPS][7][32];
    const Rep& R = a.rep0;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t i = blockIdx.x * WIDE_WARPS + warp;  // the warp's boid
    if (i >= a.n) return;
    float(*term)[32] = s_term[warp];
    const unsigned long long step = *a.step;
    const float4 me = __ldg(a.st + i);
    float acc = 0.f;  // lane c < 6: sum c
    uint32_t vec = 0, count = 0;
    int mi, Mi, mj, Mj;
    if (cell_range(R, me.x, me.y, R.dd, &mi, &Mi, &mj, &Mj)) {
#pragma unroll 1
        for (int col = mi; col <= Mi; col += 32) {
            const int bx = col + (int)lane;
            const uint32_t c0 = R.cell_off + (uint32_t)bx * (uint32_t)R.dh;
            uint32_t s = 0, len = 0;
            if (bx <= Mi) {
                const uint32_t e = min(__ldg(a.start + c0 + Mj + 1), a.n);
                s = min(__ldg(a.start + c0 + mj), e);
                len = e - s;
            }
            uint32_t incl = len;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(WIDE_FULL, incl, d);
                if (lane >= (uint32_t)d) incl += y;
            }
            const uint32_t T = __shfl_sync(WIDE_FULL, incl, 31);
#pragma unroll 1
            for (uint32_t f0 = 0; f0 < T; f0 += 32u) {
                const uint32_t f = f0 + lane;
                // the column of list entry f: the first whose inclusive count exceeds it
                int k = 0;
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) {
                    const uint32_t y = __shfl_sync(WIDE_FULL, incl, k + d - 1);
                    if (y <= f) k += d;
                }
                k = min(k, 31);
                const uint32_t ks = __shfl_sync(WIDE_FULL, s, k), kl = __shfl_sync(WIDE_FULL, len, k);
                const uint32_t ki = __shfl_sync(WIDE_FULL, incl, k);
                bool in = f < T;
                float t0 = 0.f, t1 = 0.f, dx = 0.f, dy = 0.f, hx = 0.f, hy = 0.f, fac = 1.f;
                bool other = false;
                if (in) {
                    const uint32_t p = ks + (f - (ki - kl));
                    const float4 o = __ldg(a.st + p);
                    const float ox = __fsub_rn(me.x, o.x), oy = __fsub_rn(me.y, o.y);
                    if (EXACT) {
                        const int cls = bag_class(a, R, col + k, R.cell_off + (uint32_t)(col + k) * (uint32_t)R.dh,
                                                  mj, Mj, p, me, o);
                        in = cls == 1 ||
                             (cls == 0 && __fadd_rn(__fmul_rn(ox, ox), __fmul_rn(oy, oy)) <= R.thr);
                    }
                    other = in && p != i;
                    if (other) {
                        dx = ox;
                        dy = oy;
                        hx = o.z;
                        hy = o.w;
                        if (STRICT) {
                            const float sq = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
                            const float q = __fadd_rn(__fmul_rn(sq, sq), 1.0f);
                            t0 = __fdiv_rn(dx, q);
                            t1 = __fdiv_rn(dy, q);
                        } else {
                            const float sq = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
                            fac = rcp_approx(__fmaf_rn(sq, sq, 1.0f));
                            t0 = dx;
                            t1 = dy;
                        }
                    }
                }
                vec += __popc(__ballot_sync(WIDE_FULL, in));
                count += __popc(__ballot_sync(WIDE_FULL, other));
                term[0][lane] = t0;
                term[1][lane] = t1;
                term[2][lane] = dx;
                term[3][lane] = dy;
                term[4][lane] = hx;
                term[5][lane] = hy;
                term[6][lane] = fac;
                __syncwarp();
                const uint32_t m = min(32u, T - f0);
                if (lane < 6u) {
                    // x * 1 + acc rounds as x + acc does
                    const bool fused = !STRICT && lane < 2u;
#pragma unroll 4
                    for (uint32_t j = 0; j < m; ++j)
                        acc = __fmaf_rn(term[lane][j], fused ? term[6][j] : 1.0f, acc);
                }
                __syncwarp();
            }
        }
    }
    Acc<STRICT> r;
    r.xa = __shfl_sync(WIDE_FULL, acc, 0);
    r.ya = __shfl_sync(WIDE_FULL, acc, 1);
    r.xc = __shfl_sync(WIDE_FULL, acc, 2);
    r.yc = __shfl_sync(WIDE_FULL, acc, 3);
    r.xs = __shfl_sync(WIDE_FULL, acc, 4);
    r.ys = __shfl_sync(WIDE_FULL, acc, 5);
    r.vec = vec;
    r.count = (int)count;
    if (lane == 0) force_finish<STRICT, true>(a, R, i, me, __ldg(a.ids + i), step, r);
}

template <bool STRICT, bool EXACT>
cudaError_t launch_w(const ForceArgs& a, cudaStream_t s) {
    return launch_pdl(k_flock_wide<STRICT, EXACT>, grid_for(a.n, WIDE_WARPS), 32 * WIDE_WARPS, s, a);
}

}  // namespace

cudaError_t launch_flock_wide(const ForceArgs& a, bool strict, int qmode, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    if (a.nrep != 1) return cudaErrorInvalidValue;
    if (qmode == 0) return strict ? launch_w<true, false>(a, s) : launch_w<false, false>(a, s);
    return strict ? launch_w<true, true>(a, s) : launch_w<false, true>(a, s);
}

}  // namespace kb
