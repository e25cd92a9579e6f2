// kb_walk.cuh -- the candidate sums of Bird::step in pairs and the walks of the
// relaxed and the exact query's lists, for the kernels of
// one-bag rings (kb_ring.cu, kb_small.cu): no pair straddles the seam and the
// boid itself is known by its slot.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "kb_common.h"
#include "kb_device.cuh"

namespace kb {
namespace {

// ---- pairs of f32: packed into one register pair, or two registers
using f32x2 = unsigned long long;
struct f32two {
    float x = 0.f, y = 0.f;
};
template <bool STRICT>
using pair_t = typename std::conditional<STRICT, f32two, f32x2>::type;

__device__ __forceinline__ void pack2(f32x2& r, float lo, float hi) {
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
}
__device__ __forceinline__ void pack2(f32two& r, float lo, float hi) {
    r.x = lo;
    r.y = hi;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void unpack2(f32two v, float& lo, float& hi) {
    lo = v.x;
    hi = v.y;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32two add2(f32two a, f32two b) {
    return {__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)};
}
// a - b as b * -1 + a (one rounding, the same bits): a packed subtraction is
// two sign flips and an addition
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(0xBF800000BF800000ull), "l"(a));
    return r;
}
__device__ __forceinline__ f32two sub2(f32two a, f32two b) {
    return {__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y)};
}
// v += w unless p == my
__device__ __forceinline__ void add2_unless(f32x2& v, f32x2 w, uint32_t p, uint32_t my) {
    asm("{\n\t.reg .pred other;\n\tsetp.ne.u32 other, %2, %3;\n\t@other add.rn.f32x2 %0, %0, %1;\n\t}"
        : "+l"(v)
        : "l"(w), "r"(p), "r"(my));
}
__device__ __forceinline__ void add2_unless(f32two& v, f32two w, uint32_t p, uint32_t my) {
    if (p != my) v = add2(v, w);
}

// The sums of one agent over its candidates (Acc's, in pairs).
template <bool STRICT>
struct Sums {
    pair_t<STRICT> ch{}, cs{};  // cohesion, consistency
    float ax = 0.f, ay = 0.f;   // avoidance
    uint32_t vec = 0, count = 0;

    // one candidate at d = me - o, slot p, sq its squared distance as
    // Bird::step has it; SELF: p may be the agent's own slot `my`
    template <bool SELF>
    __device__ __forceinline__ void add(pair_t<STRICT> d, float sq, pair_t<STRICT> heading, uint32_t p,
                                        uint32_t my) {
        float dx, dy;
        unpack2(d, dx, dy);
        if (STRICT) {
            const float q = __fadd_rn(__fmul_rn(sq, sq), 1.0f);
            const float2 t = div2_rn(dx, dy, q, SELF && p == my);  // the agent itself: zeros either way
            ax = __fadd_rn(ax, t.x);
            ay = __fadd_rn(ay, t.y);
        } else {
            const float inv = rcp_approx(__fmaf_rn(sq, sq, 1.0f));
            ax = __fmaf_rn(dx, inv, ax);
            ay = __fmaf_rn(dy, inv, ay);
        }
        ch = add2(ch, d);
        if (SELF) add2_unless(cs, heading, p, my);
        else cs = add2(cs, heading);
    }
    __device__ __forceinline__ Acc<STRICT> result() const {
        Acc<STRICT> r;
        r.xa = ax;
        r.ya = ay;
        unpack2(ch, r.xc, r.yc);
        unpack2(cs, r.xs, r.ys);
        r.vec = vec;
        r.count = (int)count;
        return r;
    }
};

// The squared distance of Bird::step's avoidance term / of the exact query.
__device__ __forceinline__ float sq_rn(float dx, float dy) {
    return __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
}
template <bool STRICT>
__device__ __forceinline__ float pair_sq(pair_t<STRICT> d) {
    float dx, dy;
    unpack2(d, dx, dy);
    return STRICT ? sq_rn(dx, dy) : __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
}

template <bool STRICT>
struct Candidate {
    pair_t<STRICT> pos, heading;
};
// GLOBAL: from global memory that nothing writes meanwhile; else from shared.
template <bool STRICT, bool GLOBAL = true>
__device__ __forceinline__ Candidate<STRICT> load_candidate(const float4* q) {
    Candidate<STRICT> c;
    if constexpr (STRICT) {
        const float4 v = GLOBAL ? __ldg(q) : *q;
        c.pos = {v.x, v.y};
        c.heading = {v.z, v.w};
    } else {
        const ulonglong2* const u = reinterpret_cast<const ulonglong2*>(q);
        const ulonglong2 v = GLOBAL ? __ldg(u) : *u;
        c.pos = v.x;
        c.heading = v.y;
    }
    return c;
}

// The candidate runs of up to three columns.
struct Runs {
    uint32_t s[3], e[3];
};

// One flat list over the three runs: a warp iterates its longest lane's total.
// U candidates are loaded together: 1 for large flocks (issue-bound, few
// registers), more for small ones, where too few warps hide the loads.
template <bool STRICT, int U, bool GLOBAL = true>
__device__ __forceinline__ void walk_flat(const float4* st, pair_t<STRICT> me, uint32_t my,
                                          const Runs& r, Sums<STRICT>& sums) {
    const uint32_t P1 = r.e[0] - r.s[0], P2 = P1 + (r.e[1] - r.s[1]), T = P2 + (r.e[2] - r.s[2]);
    const uint32_t j1 = r.s[1] - r.e[0], j2 = r.s[2] - r.e[1];
    uint32_t p = r.s[0];
    for (uint32_t f = 0; f < T;) {
        Candidate<STRICT> o[U];
        uint32_t at[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (f == P1) p += j1;
            if (f == P2) p += j2;
            at[u] = p;
            if (u == 0 || f < T) o[u] = load_candidate<STRICT, GLOBAL>(st + p);
            ++p;
            ++f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u == 0 || f - (uint32_t)(U - u) < T) {
                const pair_t<STRICT> d = sub2(me, o[u].pos);
                sums.template add<true>(d, pair_sq<STRICT>(d), o[u].heading, at[u], my);
            }
    }
    sums.vec = T;
}

// The agent pass of the exact query (check_circle's bag rule, field_2d.rs:
// 934-972, then the distance): the kept bags of each column as one run, with
// the part of it whose bags count as a whole; the three runs as one flat list.
// st, start: the read buffer's records (of which there are nst) and offsets, in
// global memory or shared.
template <bool STRICT, int U, bool GLOBAL = true>
__device__ __forceinline__ void walk_exact(const float4* st, const uint32_t* start, uint32_t nst, const Rep& R,
                                           float4 me4, uint32_t my, int mi, int Mi, int mj, int Mj,
                                           Sums<STRICT>& sums) {
    auto offset = [&](uint32_t c) { return min(GLOBAL ? __ldg(start + c) : start[c], nst); };
    pair_t<STRICT> me;
    pack2(me, me4.x, me4.y);
    float ymin[3], ymax[3];  // the least and greatest squared y distance of a row's corners
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float nw = __fmul_rn((float)(mj + r), R.d);
        const float n0 = __fsub_rn(nw, me4.y), n1 = __fsub_rn(fminf(__fadd_rn(nw, R.d), R.h), me4.y);
        const float q0 = __fmul_rn(n0, n0), q1 = __fmul_rn(n1, n1);
        ymin[r] = fminf(q0, q1);
        ymax[r] = fmaxf(q0, q1);
    }
    uint32_t s[3], e[3], wl[3], wn[3];
    bool apart = false;  // a skipped bag between two kept ones of a column
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        s[k] = e[k] = wl[k] = wn[k] = 0u;
        if (mi + k > Mi) continue;
        const float nw = __fmul_rn((float)(mi + k), R.d);
        const float n0 = __fsub_rn(nw, me4.x), n1 = __fsub_rn(fminf(__fadd_rn(nw, R.d), R.w), me4.x);
        const float q0 = __fmul_rn(n0, n0), q1 = __fmul_rn(n1, n1);
        const float xmin = fminf(q0, q1), xmax = fmaxf(q0, q1);
        const uint32_t c = R.cell_off + (uint32_t)(mi + k) * (uint32_t)R.dh + (uint32_t)mj;
        uint32_t o[4];
#pragma unroll
        for (int r = 3; r >= 0; --r) o[r] = offset(c + (uint32_t)min(r, Mj - mj + 1));
#pragma unroll
        for (int r = 2; r >= 0; --r) o[r] = min(o[r], o[r + 1]);
        uint32_t keep = 0u, whole = 0u;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            if (mj + r > Mj) continue;
            if (!(__fadd_rn(xmin, ymin[r]) > R.thr)) keep |= 1u << r;
            if (__fadd_rn(xmax, ymax[r]) <= R.thr) whole |= 1u << r;
        }
        apart |= keep == 5u || whole == 5u;
        if (keep) {
            s[k] = (keep & 1u) ? o[0] : ((keep & 2u) ? o[1] : o[2]);
            e[k] = (keep & 4u) ? o[3] : ((keep & 2u) ? o[2] : o[1]);
        }
        if (whole) {
            wl[k] = (whole & 1u) ? o[0] : ((whole & 2u) ? o[1] : o[2]);
            wn[k] = ((whole & 4u) ? o[3] : ((whole & 2u) ? o[2] : o[1])) - wl[k];
        }
    }
    auto take = [&](const Candidate<STRICT>& o, uint32_t p, bool all) {
        const pair_t<STRICT> d = sub2(me, o.pos);
        float dx, dy;
        unpack2(d, dx, dy);
        const float sq = sq_rn(dx, dy);
        if (all || sq <= R.thr) {
            sums.template add<true>(d, STRICT ? sq : pair_sq<STRICT>(d), o.heading, p, my);
            sums.vec += 1u;
            sums.count += p != my ? 1u : 0u;
        }
    };
    if (apart) {  // rounding at a bag's edge: bag by bag
#pragma unroll 1
        for (int k = 0; mi + k <= Mi; ++k) {
#pragma unroll 1
            for (int r = 0; mj + r <= Mj; ++r) {
                const int check = check_circle(mi + k, mj + r, R, me4.x, me4.y, R.radius);
                if (check == -1) continue;
                const uint32_t c = R.cell_off + (uint32_t)(mi + k) * (uint32_t)R.dh + (uint32_t)(mj + r);
                const uint32_t end = offset(c + 1u);
#pragma unroll 1
                for (uint32_t p = offset(c); p < end; ++p)
                    take(load_candidate<STRICT, GLOBAL>(st + p), p, check == 1);
            }
        }
        return;
    }
    const uint32_t P1 = e[0] - s[0], P2 = P1 + (e[1] - s[1]), T = P2 + (e[2] - s[2]);
    uint32_t p = s[0], w0 = wl[0], w1 = wn[0];
    for (uint32_t f = 0; f < T;) {
        Candidate<STRICT> o[U];
        uint32_t at[U];
        bool all[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (f == P1) { p = s[1]; w0 = wl[1]; w1 = wn[1]; }
            if (f == P2) { p = s[2]; w0 = wl[2]; w1 = wn[2]; }
            at[u] = p;
            all[u] = p - w0 < w1;
            if (u == 0 || f < T) o[u] = load_candidate<STRICT, GLOBAL>(st + p);
            ++p;
            ++f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u == 0 || f - (uint32_t)(U - u) < T) take(o[u], at[u], all[u]);
    }
}

}  // namespace
}  // namespace kb
