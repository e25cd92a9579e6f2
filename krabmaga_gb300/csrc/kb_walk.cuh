// kb_walk.cuh -- the candidate sums of Bird::step in pairs, for the kernels of
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

}  // namespace
}  // namespace kb
