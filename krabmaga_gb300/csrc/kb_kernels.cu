// kb_kernels.cu -- sm_103a kernels of the continuous-space agent step.
//
// Data layout in HBM (one field, or many replicas packed back to back):
//   read buffer  st[n] float4 {x, y, last_dx, last_dy}, ids[n] u32, sorted by
//                bag index (cell_off + x*dh + y, field_2d.rs:508), each bag in
//                insertion order; start[ncells+1] u32 bag offsets.
//   write list   the same records in arbitrary order plus a u32 bag key each
//                (the write buffer of field_2d.rs:838-846).
// A flock step is: force pass (read buffer -> write list, key histogram and
// arrival slots; here, in kb_ring.cu or kb_wide.cu), scan of the histogram,
// rebin by ranks or by segments (write list -> read buffer).
#include <cuda_runtime.h>
#include <stdint.h>

#include "kb_common.h"
#include "kb_launch.h"
#include "kb_runtime.h"
#include "kb_device.cuh"
#include "kb_force.cuh"

namespace kb {
namespace {

// Accumulate the candidates of one contiguous run [s, e) of the read
// buffer, four at a time so their loads are in flight together.
// Force-kernel launch shape, chosen by timing builds on GB300 (1M boids,
// density 0.025): 2-candidate load groups and 6 resident 256-thread blocks
// per SM (40 registers) beat deeper unrolling at lower occupancy.
#ifndef KB_FORCE_UNROLL
#define KB_FORCE_UNROLL 2
#endif

template <bool STRICT, bool NOWRAP>
__device__ __forceinline__ void accumulate_run_t(const Rep& R, const float4* __restrict__ st,
                                                 const uint32_t* __restrict__ ids, uint32_t s,
                                                 uint32_t e, float4 me, uint32_t my_id,
                                                 Acc<STRICT>& acc) {
    acc.vec += e - s;
    uint32_t q = s;
    constexpr int U = KB_FORCE_UNROLL;  // candidates whose loads are issued together
    for (; q + U <= e; q += U) {
        uint32_t oid[U];
        float4 o[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            oid[u] = __ldg(ids + q + u);
            o[u] = __ldg(st + q + u);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (oid[u] != my_id) acc.template add<NOWRAP>(R, me.x, me.y, o[u]);
    }
    for (; q < e; ++q) {
        const uint32_t oid = __ldg(ids + q);
        const float4 o = __ldg(st + q);
        if (oid != my_id) acc.template add<NOWRAP>(R, me.x, me.y, o);
    }
}
template <bool STRICT>
__device__ __forceinline__ void accumulate_run(const Rep& R, const float4* __restrict__ st,
                                               const uint32_t* __restrict__ ids, uint32_t s,
                                               uint32_t e, float4 me, uint32_t my_id,
                                               Acc<STRICT>& acc) {
    if (R.nowrap) accumulate_run_t<STRICT, true>(R, st, ids, s, e, me, my_id, acc);
    else accumulate_run_t<STRICT, false>(R, st, ids, s, e, me, my_id, acc);
}

// The candidate runs of up to NC columns (one contiguous run of bags per
// column), every run's bounds loaded before any candidate.
template <int NC, bool STRICT>
__device__ __forceinline__ void columns_runs(const ForceArgs& a, const Rep& R, int mi, int Mi,
                                             int mj, int Mj, float4 me, uint32_t my_id,
                                             Acc<STRICT>& acc) {
    uint32_t s[NC], e[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        if (mi + k <= Mi) {
            const uint32_t colbase = R.cell_off + (uint32_t)(mi + k) * (uint32_t)R.dh;
            e[k] = min(__ldg(a.start + colbase + Mj + 1), a.n);
            s[k] = min(__ldg(a.start + colbase + mj), e[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < NC; ++k)
        if (mi + k <= Mi) accumulate_run(R, a.st, a.ids, s[k], e[k], me, my_id, acc);
}
// The three runs of a one-bag ring as one flat list: a warp then iterates
// the longest lane's total instead of the sum of the per-column maxima.
// DENSE: long lists; each run is walked with a plain pointer (one run after
// the other, the same visiting order), which costs fewer instructions per
// candidate once the runs are long enough that the per-run maxima of a warp
// add little.
template <bool STRICT, bool DENSE>
// my_slot: the boid's own read-buffer slot when ids are unique (a candidate
// is the boid itself exactly there), else ~0u and ids are compared.
__device__ __forceinline__ void columns_flat3(const ForceArgs& a, const Rep& R, int mi, int Mi,
                                              int mj, int Mj, float4 me, uint32_t my_id,
                                              Acc<STRICT>& acc, uint32_t my_slot) {
    uint32_t s[3], e[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        s[k] = e[k] = 0u;
        if (mi + k <= Mi) {
            const uint32_t colbase = R.cell_off + (uint32_t)(mi + k) * (uint32_t)R.dh;
            e[k] = min(__ldg(a.start + colbase + Mj + 1), a.n);
            s[k] = min(__ldg(a.start + colbase + mj), e[k]);
        }
    }
    const uint32_t P1 = e[0] - s[0], P2 = P1 + (e[1] - s[1]), T = P2 + (e[2] - s[2]);
    acc.vec += T;
    const uint32_t d1 = s[1] - P1, d2 = s[2] - P2;  // position = f + d (mod 2^32)
    if (R.nowrap && my_slot != 0xFFFFFFFFu) {
        // every candidate but the boid's own slot counts: no count per candidate
        const bool self_in = (my_slot - s[0] < e[0] - s[0]) || (my_slot - s[1] < e[1] - s[1]) ||
                             (my_slot - s[2] < e[2] - s[2]);
        acc.count = (int)(T - (self_in ? 1u : 0u));
    }
    if (DENSE && R.nowrap && my_slot != 0xFFFFFFFFu) {
#pragma unroll 1
        for (int k = 0; k < 3; ++k) {
            const uint32_t ek = e[k];
            for (uint32_t q = s[k]; q < ek; ++q) {
                const float4 o = __ldg(a.st + q);
                if (q != my_slot) acc.template add<true, false>(R, me.x, me.y, o);
            }
        }
    } else if (R.nowrap && my_slot != 0xFFFFFFFFu) {
        for (uint32_t f = 0; f < T; ++f) {
            const uint32_t p = f < P1 ? s[0] + f : (f < P2 ? f + d1 : f + d2);
            const float4 o = __ldg(a.st + p);
            if (p != my_slot) acc.template add<true, false>(R, me.x, me.y, o);
        }
    } else if (R.nowrap) {
        for (uint32_t f = 0; f < T; ++f) {
            const uint32_t p = f < P1 ? s[0] + f : (f < P2 ? f + d1 : f + d2);
            const uint32_t oid = __ldg(a.ids + p);
            const float4 o = __ldg(a.st + p);
            if (oid != my_id) acc.template add<true>(R, me.x, me.y, o);
        }
    } else if (my_slot != 0xFFFFFFFFu) {  // wrapped pairs (a field wider than high)
        for (uint32_t f = 0; f < T; ++f) {
            const uint32_t p = f < P1 ? s[0] + f : (f < P2 ? f + d1 : f + d2);
            const float4 o = __ldg(a.st + p);
            if (p != my_slot) acc.template add<false>(R, me.x, me.y, o);
        }
    } else {
        for (uint32_t f = 0; f < T; ++f) {
            const uint32_t p = f < P1 ? s[0] + f : (f < P2 ? f + d1 : f + d2);
            const uint32_t oid = __ldg(a.ids + p);
            const float4 o = __ldg(a.st + p);
            if (oid != my_id) acc.template add<false>(R, me.x, me.y, o);
        }
    }
}

// The wider ring out of line, so that it does not set the register budget of
// the common one-ring case.
template <bool STRICT>
__device__ __noinline__ void columns_runs_5(const ForceArgs& a, const Rep& R, int mi, int Mi,
                                            int mj, int Mj, float4 me, uint32_t my_id,
                                            Acc<STRICT>& acc) {
    columns_runs<5>(a, R, mi, Mi, mj, Mj, me, my_id, acc);
}


// The candidate sums of one agent at `me` against the read buffer (the
// query of bird.rs:41 and the loop of bird.rs:48-82).  my_slot: the agent's
// own read-buffer slot when self is recognised by slot, else ~0u.
template <bool STRICT, int QMODE, bool DENSE = false>
__device__ __forceinline__ void gather_candidates(const ForceArgs& a, const Rep& R, float4 me,
                                                  uint32_t my_id, uint32_t my_slot,
                                                  Acc<STRICT>& acc) {
    int mi, Mi, mj, Mj;
    if (cell_range(R, me.x, me.y, R.dd, &mi, &Mi, &mj, &Mj)) {
        const bool clamped = R.toroidal && !R.cell_wrap;  // runs never cross the seam
        if (QMODE == 0 && clamped && Mi - mi < 5) {
            // clamped range: each column's bags mj..Mj are one contiguous
            // run; fetch every run's bounds before touching candidates
            // a one-bag ring (the common case) as one flat list; the wider
            // two-bag ring out of line
            if (Mi - mi < 3)
                columns_flat3<STRICT, DENSE>(a, R, mi, Mi, mj, Mj, me, my_id, acc, my_slot);
            else columns_runs_5(a, R, mi, Mi, mj, Mj, me, my_id, acc);
        } else {
            for (int ci = mi; ci <= Mi; ++ci) {
                const int bx = t_transform(ci, R.max_x);
                const uint32_t colbase = R.cell_off + (uint32_t)bx * (uint32_t)R.dh;
                if (QMODE == 0 && clamped) {
                    const uint32_t e = min(__ldg(a.start + colbase + Mj + 1), a.n);
                    accumulate_run(R, a.st, a.ids, min(__ldg(a.start + colbase + mj), e), e, me,
                                   my_id, acc);
                    continue;
                }
                for (int cj = mj; cj <= Mj; ++cj) {
                    const int by = t_transform(cj, R.max_y);
                    const uint32_t c = colbase + (uint32_t)by;
                    const uint32_t e = min(__ldg(a.start + c + 1), a.n);
                    const uint32_t s = min(__ldg(a.start + c), e);
                    if (s == e) continue;
                    if (QMODE == 0) {
                        accumulate_run(R, a.st, a.ids, s, e, me, my_id, acc);
                        continue;
                    }
                    const int check = check_circle(bx, by, R, me.x, me.y, R.radius);
                    if (check == -1) continue;
                    for (uint32_t k = s; k < e; ++k) {
                        const float4 o = __ldg(a.st + k);
                        if (check == 0 &&
                            !(distance(me.x, me.y, o.x, o.y, R.w, R.h, R.toroidal != 0) <= R.radius))
                            continue;
                        acc.vec += 1;
                        if (__ldg(a.ids + k) != my_id) acc.add(R, me.x, me.y, o);
                    }
                }
            }
        }
    }
}

template <bool STRICT, int QMODE, bool DENSE>
__device__ __forceinline__ void force_body(const ForceArgs& a, const Rep& R, uint32_t i) {
    const unsigned long long step = *a.step;
    const float4 me = __ldg(a.st + i);
    const uint32_t my_id = __ldg(a.ids + i);
    Acc<STRICT> acc;
    gather_candidates<STRICT, QMODE, DENSE>(a, R, me, my_id, a.self_by_slot ? i : 0xFFFFFFFFu, acc);
    force_finish<STRICT, !DENSE>(a, R, i, me, my_id, step, acc);
}

#ifndef KB_FORCE_THREADS
#define KB_FORCE_THREADS 256
#endif
static_assert(KB_FORCE_THREADS == FORCE_THREADS, "the host block tables assume this block size");
#ifndef KB_FORCE_MINB
#define KB_FORCE_MINB 6
#endif
#ifndef KB_FORCE_MINB_MULTI
#define KB_FORCE_MINB_MULTI 6
#endif

// BT: threads per block (the packed-replica block table's granularity); the
// same 48 warps per SM at every block size.
template <bool STRICT, int QMODE, bool MULTI, bool DENSE = false, int BT = KB_FORCE_THREADS>
__global__ void __launch_bounds__(BT, (MULTI ? KB_FORCE_MINB_MULTI : KB_FORCE_MINB) * KB_FORCE_THREADS / BT)
    k_flock_force(ForceArgs a) {
    pdl_enter();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (MULTI) {
        // one replica per block: its record is read once into shared memory
        __shared__ Rep sR;
        const uint2 e = a.blk[blockIdx.x];
        load_rep_shared(&sR, a.reps + e.x);
        __syncthreads();
        if (a.apart) {
            if (threadIdx.x == 0) sR.nowrap = 0;
            __syncthreads();
        }
        const uint32_t k = e.y + threadIdx.x;
        if (k >= sR.boid_off + sR.nboids) return;
        force_body<STRICT, QMODE, false>(a, sR, k);
        return;
    }
    if (i >= a.n) return;
    force_body<STRICT, QMODE, DENSE>(a, a.rep0, i);
}

// Bird::step for agents given by the caller rather than read from the read
// buffer (agents that join the schedule, schedule.rs:283-303): agent j reads
// its neighbours from the read buffer, skips candidates with its own id
// (bird.rs:50) and writes its next state to slot j of the outputs.
template <bool STRICT, int QMODE>
__global__ void __launch_bounds__(KB_FORCE_THREADS)
    k_flock_agents(ForceArgs a, const float4* __restrict__ in_st, const uint32_t* __restrict__ in_ids,
                   uint32_t nin) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nin) return;
    const unsigned long long step = *a.step;
    const float4 me = in_st[j];
    const uint32_t my_id = in_ids[j];
    Acc<STRICT> acc;
    gather_candidates<STRICT, QMODE>(a, a.rep0, me, my_id, 0xFFFFFFFFu, acc);
    force_finish<STRICT, false>(a, a.rep0, j, me, my_id, step, acc);
}

// Mark every live write-list entry whose id is in sorted[0..m) removed.
__global__ void k_remove_ids(const uint32_t* __restrict__ ids, uint8_t* dead, uint32_t n,
                             const uint32_t* __restrict__ sorted, uint32_t m, uint32_t* removed) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || dead[i]) return;
    const uint32_t id = ids[i];
    uint32_t lo = 0, hi = m;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (sorted[mid] < id) lo = mid + 1;
        else hi = mid;
    }
    if (lo < m && sorted[lo] == id) {
        dead[i] = 1;
        atomicAdd(removed, 1u);
    }
}

// first[j] = the smallest index i < n with ids[i] == sorted[j] (live entries
// only when dead != nullptr); first[] starts at ~0u.
__global__ void k_find_ids(const uint32_t* __restrict__ ids, const uint8_t* __restrict__ dead,
                           uint32_t n, const uint32_t* __restrict__ sorted, uint32_t m,
                           uint32_t* first) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || (dead && dead[i])) return;
    const uint32_t id = ids[i];
    uint32_t lo = 0, hi = m;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (sorted[mid] < id) lo = mid + 1;
        else hi = mid;
    }
    if (lo < m && sorted[lo] == id) atomicMin(&first[lo], i);
}

__global__ void k_gather_found(const float4* __restrict__ st, const uint32_t* __restrict__ first,
                               uint32_t m, float4* __restrict__ out) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= m) return;
    const uint32_t i = first[j];
    out[j] = i == 0xFFFFFFFFu ? make_float4(0.f, 0.f, 0.f, 0.f) : st[i];
}

// ---------------------------------------------------------- scan
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr unsigned long long FLAG_AGG = 1ull, FLAG_INC = 2ull;
constexpr uint32_t SPIN_LIMIT = 1u << 20;

__device__ __forceinline__ unsigned long long pack_tile(uint32_t epoch, unsigned long long flag,
                                                        uint32_t v) {
    return ((unsigned long long)(epoch & 0x3FFFFFFFu) << 34) | (flag << 32) | v;
}

__global__ void __launch_bounds__(SCAN_THREADS)
    k_scan(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint32_t n, ScanCtl* ctl,
           unsigned long long* tstate, uint32_t* err, int zero_in, uint32_t ntiles, WaitCfg wait) {
    pdl_enter();
    const uint32_t spin_limit = wait.spin_limit ? wait.spin_limit : SPIN_LIMIT;
    __shared__ uint32_t s_tile, s_epoch, s_prefix;
    __shared__ uint32_t s_warp[SCAN_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        s_tile = atomicAdd(&ctl->tile_counter, 1u);
        s_epoch = *((volatile uint32_t*)&ctl->epoch);
    }
    __syncthreads();
    const uint32_t tile = s_tile, epoch = s_epoch;
    const uint64_t base = (uint64_t)tile * SCAN_TILE + (uint64_t)tid * SCAN_ITEMS;

    uint32_t v[SCAN_ITEMS];
    if (base + SCAN_ITEMS <= n) {
        const uint4* p = reinterpret_cast<const uint4*>(in + base);
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS / 4; ++k) {
            const uint4 w = p[k];
            v[4 * k] = w.x; v[4 * k + 1] = w.y; v[4 * k + 2] = w.z; v[4 * k + 3] = w.w;
        }
        if (zero_in) {
            uint4* q = reinterpret_cast<uint4*>(const_cast<uint32_t*>(in + base));
#pragma unroll
            for (int k = 0; k < SCAN_ITEMS / 4; ++k) q[k] = make_uint4(0, 0, 0, 0);
        }
    } else {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k) {
            v[k] = (base + k < n) ? in[base + k] : 0u;
            if (zero_in && base + k < n) const_cast<uint32_t*>(in)[base + k] = 0u;
        }
    }
    uint32_t tsum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) tsum += v[k];
    // block exclusive scan of the per-thread sums
    uint32_t x = tsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = (lane < SCAN_THREADS / 32) ? s_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < SCAN_THREADS / 32) s_warp[lane] = w;  // inclusive warp prefixes
    }
    __syncthreads();
    const uint32_t agg = s_warp[SCAN_THREADS / 32 - 1];
    const uint32_t texcl = x - tsum + (warp > 0 ? s_warp[warp - 1] : 0u);

    // decoupled look-back across tiles, 256 predecessors per round trip
    __shared__ int s_jinc;
    __shared__ uint32_t s_sum[SCAN_THREADS / 32];
    const bool publish = tile != wait.withhold;  // the test hook withholds one tile's words
    if (tile == 0) {
        if (tid == 0) {
            if (publish) atomicExch(&tstate[0], pack_tile(epoch, FLAG_INC, agg));
            s_prefix = 0;
        }
    } else {
        if (tid == 0) {
            if (publish) atomicExch(&tstate[tile], pack_tile(epoch, FLAG_AGG, agg));
            s_jinc = -0x7fffffff;
        }
        __syncthreads();
        uint32_t prefix = 0;
        int64_t pred = (int64_t)tile - 1;
        for (;;) {
            const int64_t j = pred - tid;
            unsigned long long word = pack_tile(epoch, FLAG_INC, 0u);  // below tile 0
            if (j >= 0) {
                uint32_t spins = 0;
                while (true) {
                    word = *((volatile unsigned long long*)&tstate[j]);
                    if ((uint32_t)(word >> 34) == (epoch & 0x3FFFFFFFu) && ((word >> 32) & 3ull) != 0ull)
                        break;
                    if (++spins > spin_limit) {
                        atomicOr(err, ERR_SPIN_TIMEOUT);
                        word = pack_tile(epoch, FLAG_INC, 0u);
                        break;
                    }
                    __nanosleep(32);
                }
            }
            const bool inc = ((word >> 32) & 3ull) == FLAG_INC;
            // the nearest inclusive predecessor in this window: the smallest tid
            if (inc) atomicMax(&s_jinc, -(int)tid);
            __syncthreads();
            const int stop = -s_jinc;  // tid of the nearest inclusive word, or huge
            uint32_t v = ((int)tid <= stop) ? (uint32_t)word : 0u;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) s_sum[warp] = v;
            __syncthreads();
            uint32_t tot = 0;
#pragma unroll
            for (int w = 0; w < SCAN_THREADS / 32; ++w) tot += s_sum[w];
            prefix += tot;
            const bool done = stop < SCAN_THREADS;
            __syncthreads();
            if (done) break;
            if (tid == 0) s_jinc = -0x7fffffff;
            pred -= SCAN_THREADS;
            __syncthreads();
        }
        if (tid == 0) {
            if (publish) atomicExch(&tstate[tile], pack_tile(epoch, FLAG_INC, prefix + agg));
            s_prefix = prefix;
        }
    }
    __syncthreads();
    const uint32_t prefix = s_prefix;
    uint32_t run = prefix + texcl;
    if (base + SCAN_ITEMS <= n) {
        uint32_t o[SCAN_ITEMS];
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k) {
            o[k] = run;
            run += v[k];
        }
        uint4* p = reinterpret_cast<uint4*>(out + base);
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS / 4; ++k)
            p[k] = make_uint4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
    } else {
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k) {
            if (base + k < n) out[base + k] = run;
            run += v[k];
        }
    }
    if (tile == ntiles - 1 && tid == 0) out[n] = prefix + agg;
    // the last CTA to finish re-arms the control block for the next launch
    if (tid == 0) {
        __threadfence();
        const uint32_t d = atomicAdd(&ctl->done_counter, 1u);
        if (d == ntiles - 1) {
            ctl->tile_counter = 0u;
            ctl->done_counter = 0u;
            __threadfence();
            atomicAdd(&ctl->epoch, 1u);
        }
    }
}

// ---------------------------------------------------------- rebin
// The arrivals of bag c in write-list order from the records [s, e).
__device__ __forceinline__ void rebin_run(const RebinArgs& a, const Rep& R, uint32_t c, uint32_t s,
                                          uint32_t e, uint32_t& dst, uint32_t end) {
    for (uint32_t p = s; p < e; ++p) {
        uint32_t k;
        if (a.key) {
            k = __ldg(a.key + p);
        } else {  // key from the record's own position
            const float4 r = __ldg(a.a_st + p);
            const int64_t b = bag_index(R, disc(r.x, R), disc(r.y, R));
            k = b >= 0 ? R.cell_off + (uint32_t)b : 0xFFFFFFFFu;
        }
        if (k == c) {
            if (dst < end) {
                a.s_st[dst] = __ldg(a.a_st + p);
                a.s_ids[dst] = __ldg(a.a_ids + p);
            }
            ++dst;
        }
    }
}

__device__ __forceinline__ void rebin_cell(const RebinArgs& a, const Rep& R, uint32_t c) {
    const uint32_t end = min(__ldg(a.start_next + c + 1), a.n);
    uint32_t dst = min(__ldg(a.start_next + c), end);
    if (dst == end) return;
    const uint32_t local = c - R.cell_off;
    const uint32_t Xu = div_dh(local, R);
    const int X = (int)Xu, Y = (int)(local - Xu * (uint32_t)R.dh);
    if (X > 0 && X < R.seam && Y > 0 && Y < R.seam) {
        // interior bag: three source columns, rows Y-1..Y+1 contiguous in each
        uint32_t s[3], e[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const uint32_t base = R.cell_off + (uint32_t)(X - 1 + k) * (uint32_t)R.dh + (uint32_t)Y;
            e[k] = min(__ldg(a.start_cur + base + 2), a.n);
            s[k] = min(__ldg(a.start_cur + base - 1), e[k]);
        }
        if (a.key) {
            // the first keys of every run in flight together
            uint32_t kk[3][4];
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    kk[k][u] = (s[k] + u < e[k]) ? __ldg(a.key + s[k] + u) : 0xFFFFFFFFu;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (kk[k][u] == c) {
                        if (dst < end) {
                            a.s_st[dst] = __ldg(a.a_st + s[k] + u);
                            a.s_ids[dst] = __ldg(a.a_ids + s[k] + u);
                        }
                        ++dst;
                    }
                }
                if (s[k] + 4 < e[k]) rebin_run(a, R, c, s[k] + 4, e[k], dst, end);
            }
        } else {
#pragma unroll
            for (int k = 0; k < 3; ++k) rebin_run(a, R, c, s[k], e[k], dst, end);
        }
    } else {
        int lastx = -1;
#pragma unroll 1
        for (int kx = 0; kx < SRC_LINES; ++kx) {
            const int sx = src_line(kx, X, R.max_x, R.seam);
            if (sx < 0 || sx > R.max_x || sx <= lastx) continue;
            lastx = sx;
            const uint32_t colbase = R.cell_off + (uint32_t)sx * (uint32_t)R.dh;
            int lasty = -1;
#pragma unroll 1
            for (int ky = 0; ky < SRC_LINES; ++ky) {
                const int sy = src_line(ky, Y, R.max_y, R.seam);
                if (sy < 0 || sy > R.max_y || sy <= lasty) continue;
                lasty = sy;
                const uint32_t re = min(__ldg(a.start_cur + colbase + sy + 1), a.n);
                rebin_run(a, R, c, min(__ldg(a.start_cur + colbase + sy), re), re, dst, end);
            }
        }
    }
    if (dst != end) atomicOr(a.err, ERR_REBIN_MISS | ERR_MISS_MATERIALIZE);
}

template <bool MULTI>
__global__ void __launch_bounds__(256) k_rebin(RebinArgs a) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c == 0 && a.step != nullptr) *a.step += 1ull;
    if (c >= a.ncells) return;
    if (MULTI) {
        const Rep R = a.reps[rep_of_cell(a.reps, a.nrep, c)];
        rebin_cell(a, R, c);
    } else {
        rebin_cell(a, a.rep0, c);
    }
}

// ---------------------------------------------------------- two-pass scan
// For up to SCAN2_MAX_TILES tiles the offsets are a reduce-then-scan pair of
// launches with no waiting between blocks: per-tile sums, then every tile
// adds the sums before it (at most SCAN2_MAX_TILES / 256 loads a thread),
// scans its items and writes them.  Larger inputs take the single-pass
// look-back kernel above.  The sums go into the look-back state words as
// plain 64-bit values: their flag bits stay zero, so a later look-back
// launch on the same buffer reads them as "not published".
constexpr int S2_ITEMS = KB_SCAN2_ITEMS;

// Exclusive block scan of one value per thread (SCAN_THREADS threads).
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t x, uint32_t* s_warp, uint32_t* total) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t base = 0, tot = 0;
#pragma unroll
    for (int w = 0; w < SCAN_THREADS / 32; ++w) {
        const uint32_t v = s_warp[w];
        if (w < warp) base += v;
        tot += v;
    }
    *total = tot;
    return base + incl - x;
}

template <int ITEMS>
__device__ __forceinline__ void load_items(const uint32_t* in, uint32_t n, uint64_t base,
                                           uint32_t (&v)[ITEMS]) {
    if (base + ITEMS <= n) {
        const uint4* p = reinterpret_cast<const uint4*>(in + base);
#pragma unroll
        for (int k = 0; k < ITEMS / 4; ++k) {
            const uint4 w = p[k];
            v[4 * k] = w.x; v[4 * k + 1] = w.y; v[4 * k + 2] = w.z; v[4 * k + 3] = w.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) v[k] = (base + k < n) ? in[base + k] : 0u;
    }
}

__global__ void __launch_bounds__(SCAN_THREADS)
    k_tile_sums(const uint32_t* __restrict__ in, uint32_t n, unsigned long long* __restrict__ sums) {
    pdl_enter();
    __shared__ uint32_t s_warp[SCAN_THREADS / 32];
    const uint64_t base = (uint64_t)blockIdx.x * SCAN2_TILE + (uint64_t)threadIdx.x * S2_ITEMS;
    uint32_t v[S2_ITEMS];
    load_items<S2_ITEMS>(in, n, base, v);
    uint32_t t = 0;
#pragma unroll
    for (int k = 0; k < S2_ITEMS; ++k) t += v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t s = 0;
#pragma unroll
        for (int w = 0; w < SCAN_THREADS / 32; ++w) s += s_warp[w];
        sums[blockIdx.x] = (unsigned long long)s;
    }
}

// Up to SCAN_CLUSTER_MAX bags one launch: a cluster of eight blocks scans its
// eighths, exchanges their totals through distributed shared memory and adds
// the ones before.  Four bags a thread and no more: a step of 20k boids (18k
// bags) takes 7.7 us with it and 8.2 with the pair of launches below, one of 65k
// boids (60k bags, eight a thread) 10.0 and 8.8, since eight SMs then move what
// the pair spreads over the chip.
__global__ void __cluster_dims__(SCAN_CLUSTER) __launch_bounds__(1024)
    k_scan_cluster(uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint32_t n, int zero_in) {
    // a block's shared memory may be written only once that block runs: every
    // block says so here, and the stores below wait for it (the loads and the
    // block scan hide the wait)
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    pdl_enter();
    constexpr int ITEMS = (int)(SCAN_CLUSTER_MAX / (SCAN_CLUSTER * 1024u));
    __shared__ uint32_t s_warp[32], s_total[SCAN_CLUSTER];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, rank = blockIdx.x;
    const uint64_t base = ((uint64_t)rank * 1024u + tid) * ITEMS;
    uint32_t v[ITEMS], tsum = 0;
    load_items<ITEMS>(in, n, base, v);
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) tsum += v[k];
    uint32_t incl = tsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    if (lane == 31u) s_warp[warp] = incl;
    __syncthreads();
    const uint32_t x = s_warp[lane];
    uint32_t xi = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, xi, o);
        if (lane >= (uint32_t)o) xi += y;
    }
    const uint32_t before = __shfl_sync(0xffffffffu, xi - x, warp), total = __shfl_sync(0xffffffffu, xi, 31);
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (tid < SCAN_CLUSTER) {
        uint32_t at;
        asm("mapa.shared::cluster.u32 %0, %1, %2;"
            : "=r"(at)
            : "r"((uint32_t)__cvta_generic_to_shared(&s_total[rank])), "r"(tid));
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at), "r"(total) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    uint32_t prefix = 0, all = 0;
#pragma unroll
    for (uint32_t q = 0; q < SCAN_CLUSTER; ++q) {
        const uint32_t w = s_total[q];
        if (q < rank) prefix += w;
        all += w;
    }
    uint32_t run = prefix + before + incl - tsum;
    if (base + ITEMS <= n) {
        uint4* p = reinterpret_cast<uint4*>(out + base);
        uint4* q = reinterpret_cast<uint4*>(in + base);
#pragma unroll
        for (int k = 0; k < ITEMS / 4; ++k) {
            uint4 o;
            o.x = run;
            o.y = o.x + v[4 * k];
            o.z = o.y + v[4 * k + 1];
            o.w = o.z + v[4 * k + 2];
            run = o.w + v[4 * k + 3];
            p[k] = o;
            if (zero_in) q[k] = make_uint4(0, 0, 0, 0);
        }
    } else {
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            if (base + k < n) {
                out[base + k] = run;
                if (zero_in) in[base + k] = 0u;
            }
            run += v[k];
        }
    }
    if (rank == 0 && tid == 0) out[n] = all;
}

// The exclusive scan, in place, of ntiles tile sums (one block; large bag
// matrices: the tiles then take their prefix with one load).
constexpr int SUMS_THREADS = 1024;
constexpr int SUMS_ITEMS = 8;
__global__ void __launch_bounds__(SUMS_THREADS) k_scan_sums(unsigned long long* sums, uint32_t ntiles) {
    pdl_enter();
    __shared__ uint32_t s_warp[SUMS_THREADS / 32];
    __shared__ uint32_t s_carry;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    if (tid == 0) s_carry = 0u;
    __syncthreads();
    for (uint64_t chunk = 0; chunk < ntiles; chunk += (uint64_t)SUMS_THREADS * SUMS_ITEMS) {
        const uint64_t base = chunk + (uint64_t)tid * SUMS_ITEMS;
        uint32_t v[SUMS_ITEMS], t = 0;
#pragma unroll
        for (int k = 0; k < SUMS_ITEMS; ++k) {
            v[k] = base + k < ntiles ? (uint32_t)sums[base + k] : 0u;
            t += v[k];
        }
        uint32_t x = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        if (lane == 31u) s_warp[warp] = x;
        __syncthreads();
        if (warp == 0) {
            uint32_t w = s_warp[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= (uint32_t)o) w += y;
            }
            s_warp[lane] = w;  // inclusive warp prefixes
        }
        __syncthreads();
        uint32_t run = s_carry + (warp > 0 ? s_warp[warp - 1] : 0u) + x - t;
#pragma unroll
        for (int k = 0; k < SUMS_ITEMS; ++k) {
            if (base + k < ntiles) sums[base + k] = (unsigned long long)run;
            run += v[k];
        }
        __syncthreads();
        if (tid == 0) s_carry += s_warp[SUMS_THREADS / 32 - 1];
        __syncthreads();
    }
}

// PREFIX: sums[] already holds each tile's exclusive prefix (k_scan_sums);
// otherwise the tile adds up the sums of the tiles before it.
template <bool PREFIX>
__global__ void __launch_bounds__(SCAN_THREADS)
    k_scan_tiles(uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint32_t n,
                 const unsigned long long* __restrict__ sums, int zero_in, uint32_t ntiles) {
    pdl_enter();
    __shared__ uint32_t s_warp[SCAN_THREADS / 32], s_red[SCAN_THREADS / 32];
    const uint32_t tile = blockIdx.x, tid = threadIdx.x;
    // this tile's prefix: the sums of the tiles before it
    uint32_t part = 0;
    if (PREFIX) {
        if (tid == 0) part = (uint32_t)sums[tile];
    } else {
        for (uint32_t k = tid; k < tile; k += SCAN_THREADS) part += (uint32_t)sums[k];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if ((tid & 31) == 0) s_red[tid >> 5] = part;
    const uint64_t base = (uint64_t)tile * SCAN2_TILE + (uint64_t)tid * S2_ITEMS;
    uint32_t v[S2_ITEMS];
    load_items<S2_ITEMS>(in, n, base, v);
    uint32_t tsum = 0;
#pragma unroll
    for (int k = 0; k < S2_ITEMS; ++k) tsum += v[k];
    uint32_t total;
    const uint32_t texcl = block_excl_scan(tsum, s_warp, &total);  // syncs s_red too
    uint32_t prefix = 0;
#pragma unroll
    for (int w = 0; w < SCAN_THREADS / 32; ++w) prefix += s_red[w];
    uint32_t run = prefix + texcl;
    if (base + S2_ITEMS <= n) {
        uint32_t o[S2_ITEMS];
#pragma unroll
        for (int k = 0; k < S2_ITEMS; ++k) {
            o[k] = run;
            run += v[k];
        }
        uint4* p = reinterpret_cast<uint4*>(out + base);
#pragma unroll
        for (int k = 0; k < S2_ITEMS / 4; ++k)
            p[k] = make_uint4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
        if (zero_in) {
            uint4* q = reinterpret_cast<uint4*>(in + base);
#pragma unroll
            for (int k = 0; k < S2_ITEMS / 4; ++k) q[k] = make_uint4(0, 0, 0, 0);
        }
    } else {
#pragma unroll
        for (int k = 0; k < S2_ITEMS; ++k) {
            if (base + k < n) {
                out[base + k] = run;
                if (zero_in) in[base + k] = 0u;
            }
            run += v[k];
        }
    }
    if (tile == ntiles - 1 && tid == 0) out[n] = prefix + total;
}

// ---------------------------------------------------------- segment rebin
// One warp per segment of up to 32 consecutive bags of one column (lane l
// owns bag c0 + l).  The arrivals of those bags sit in the write list inside
// the source runs of the neighbouring columns: rows Y0-1..Y1+1 of columns
// X-1..X+1 (plus the seam lines at the field's edges).  The warp streams
// those runs in ascending bag order, 32 entries at a time with coalesced key
// loads; entries whose key falls in the segment take the next slot of their
// bag: __match_any_sync ranks equal keys within a batch in lane (= list)
// order, a per-bag counter in shared memory carries the rank across batches.
// That is the per-bag insertion order of the reference's lazy_update.
constexpr uint32_t FULL_MASK = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t rep_segments_dev(const Rep& R) {
    const uint32_t rows = R.seg_rows > 0 ? (uint32_t)R.seg_rows : (uint32_t)SEG_ROWS;
    return (uint32_t)R.dw * (((uint32_t)R.dh + rows - 1) / rows);
}

__device__ __forceinline__ int rep_of_seg(const Rep* reps, int nrep, uint32_t g) {
    int lo = 0, hi = nrep - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (__ldg(&reps[mid].seg_off) <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Slot of one write-list entry of a batch of 32 (key k per lane, ~0u for
// none) in its bag of the segment, or ~0u when the key is outside the
// segment.  Every lane of the warp calls it.
// Bag offsets of a segment: lane l holds bag l (lo[0], hi[0]) and, with two
// bags per lane (64-bag segments), bag l + 32 (lo[1], hi[1]).
template <int BPL>
struct SegBags {
    uint32_t lo[BPL], hi[BPL];
};

template <int BPL>
__device__ __forceinline__ uint32_t seg_rank(uint32_t k, uint32_t c0, int nb, const SegBags<BPL>& sb,
                                             uint32_t* cnt, uint32_t lane_lt, bool& bad) {
    const uint32_t local = k - c0;
    const bool in = local < (uint32_t)nb;
    if (__ballot_sync(FULL_MASK, in) == 0u) return 0xFFFFFFFFu;
    const uint32_t peers = __match_any_sync(FULL_MASK, in ? local : 0xFFFFFFFFu);
    const uint32_t rank = __popc(peers & lane_lt);
    const uint32_t src = local & 31u;
    uint32_t blo = __shfl_sync(FULL_MASK, sb.lo[0], src);
    uint32_t bhi = __shfl_sync(FULL_MASK, sb.hi[0], src);
    if (BPL == 2) {
        const uint32_t blo1 = __shfl_sync(FULL_MASK, sb.lo[BPL - 1], src);
        const uint32_t bhi1 = __shfl_sync(FULL_MASK, sb.hi[BPL - 1], src);
        if (local >= 32u) {
            blo = blo1;
            bhi = bhi1;
        }
    }
    const uint32_t slot = BPL == 2 ? local : src;
    const uint32_t base = in ? cnt[slot] : 0u;
    __syncwarp();
    uint32_t dst = 0xFFFFFFFFu;
    if (in) {
        dst = blo + base + rank;
        if (dst >= bhi) {
            bad = true;
            dst = 0xFFFFFFFFu;
        }
        if (rank + 1u == (uint32_t)__popc(peers)) cnt[slot] = base + rank + 1u;
    }
    __syncwarp();
    return dst;
}

// One batch of 32 write-list entries (p, valid per lane): rank and copy.
#ifndef KB_REBIN_BATCHES
#define KB_REBIN_BATCHES 2
#endif

template <int BPL>
__device__ __forceinline__ void seg_batch(const RebinArgs& a, bool valid, uint32_t p, uint32_t c0,
                                          int nb, const SegBags<BPL>& sb, uint32_t* cnt,
                                          uint32_t lane_lt, bool& bad) {
    const uint32_t k = valid ? __ldg(a.key + p) : 0xFFFFFFFFu;
    const uint32_t dst = seg_rank<BPL>(k, c0, nb, sb, cnt, lane_lt, bad);
    if (dst != 0xFFFFFFFFu) {
        a.s_st[dst] = __ldg(a.a_st + p);
        a.s_ids[dst] = __ldg(a.a_ids + p);
    }
}

// ROWS (<= 64) consecutive bags of one column per warp (one or two per lane).
template <int ROWS>
__device__ __forceinline__ void rebin_segment(const RebinArgs& a, const Rep& R, uint32_t g,
                                              uint32_t* cnt) {
    static_assert(ROWS >= 1 && ROWS <= 64, "a segment's bags map to one or two per lane");
    constexpr int BPL = ROWS > 32 ? 2 : 1;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t nsy = ((uint32_t)R.dh + ROWS - 1) / ROWS;
    const uint32_t local = g - R.seg_off;
    const uint32_t Xu = local / nsy;
    const int X = (int)Xu;
    const int Y0 = (int)(local - Xu * nsy) * ROWS;
    const int nb = min(ROWS, R.dh - Y0);
    const int Y1 = Y0 + nb - 1;
    const uint32_t c0 = R.cell_off + Xu * (uint32_t)R.dh + (uint32_t)Y0;
    const bool interior = X > 0 && X < R.seam && Y0 > 0 && Y1 < R.seam;
    // this segment's bag offsets and (interior) the bounds of its three
    // source runs, in one round trip
    SegBags<BPL> sb;
    uint32_t b = 0;
#pragma unroll
    for (int h = 0; h < BPL; ++h) {
        sb.lo[h] = sb.hi[h] = 0u;
        const int bag = (int)lane + 32 * h;
        if (bag < nb) {
            sb.hi[h] = min(__ldg(a.start_next + c0 + bag + 1), a.n);
            sb.lo[h] = min(__ldg(a.start_next + c0 + bag), sb.hi[h]);
        }
    }
    if (interior && lane < 6u) {
        const uint32_t cb = R.cell_off + (uint32_t)(X - 1 + (int)(lane % 3u)) * (uint32_t)R.dh;
        b = min(__ldg(a.start_cur + cb + (lane < 3u ? (uint32_t)(Y0 - 1) : (uint32_t)(Y1 + 2))), a.n);
    }
    {
        const uint32_t first = __shfl_sync(FULL_MASK, sb.lo[0], 0);
        uint32_t last = __shfl_sync(FULL_MASK, sb.hi[0], (nb - 1) & 31);
        if (BPL == 2) {
            const uint32_t last1 = __shfl_sync(FULL_MASK, sb.hi[BPL - 1], (nb - 1) & 31);
            if (nb > 32) last = last1;
        }
        if (first == last) return;  // no arrivals
    }
#pragma unroll
    for (int h = 0; h < BPL; ++h) cnt[lane + 32 * h] = 0u;
    __syncwarp();
    const uint32_t lane_lt = (1u << lane) - 1u;
    bool bad = false;
    if (interior) {
        // columns X-1..X+1, rows Y0-1..Y1+1, as one list of three runs
        const uint32_t s0 = __shfl_sync(FULL_MASK, b, 0), s1 = __shfl_sync(FULL_MASK, b, 1);
        const uint32_t s2 = __shfl_sync(FULL_MASK, b, 2), e0 = __shfl_sync(FULL_MASK, b, 3);
        const uint32_t e1 = __shfl_sync(FULL_MASK, b, 4), e2 = __shfl_sync(FULL_MASK, b, 5);
        // run bounds out of order (only after a failed step) read as empty runs
        const uint32_t P1 = e0 - min(s0, e0), P2 = P1 + (e1 - min(s1, e1)), T = P2 + (e2 - min(s2, e2));
        // KB_REBIN_BATCHES batches of 32 list entries per round: every key of
        // the round in flight at once, then the ranks in list order, then every
        // record of the round in flight at once
        for (uint32_t f0 = 0; f0 < T; f0 += 32u * KB_REBIN_BATCHES) {
            uint32_t p[KB_REBIN_BATCHES], dst[KB_REBIN_BATCHES];
#pragma unroll
            for (int b = 0; b < KB_REBIN_BATCHES; ++b) {
                const uint32_t ff = f0 + 32u * b + lane;
                p[b] = ff < P1 ? s0 + ff : (ff < P2 ? s1 + (ff - P1) : s2 + (ff - P2));
                dst[b] = ff < T ? __ldg(a.key + p[b]) : 0xFFFFFFFFu;
            }
#pragma unroll
            for (int b = 0; b < KB_REBIN_BATCHES; ++b)
                dst[b] = seg_rank<BPL>(dst[b], c0, nb, sb, cnt, lane_lt, bad);
            float4 rec[KB_REBIN_BATCHES];
            uint32_t rid[KB_REBIN_BATCHES];
#pragma unroll
            for (int b = 0; b < KB_REBIN_BATCHES; ++b) {
                if (dst[b] != 0xFFFFFFFFu) {
                    rec[b] = __ldg(a.a_st + p[b]);
                    rid[b] = __ldg(a.a_ids + p[b]);
                }
            }
#pragma unroll
            for (int b = 0; b < KB_REBIN_BATCHES; ++b) {
                if (dst[b] != 0xFFFFFFFFu) {
                    a.s_st[dst[b]] = rec[b];
                    a.s_ids[dst[b]] = rid[b];
                }
            }
        }
    } else {
        // a segment at the seam or the field's edge: the source lines of
        // src_line on both axes, run by run in ascending bag order
        const int mlo = max(0, Y0 - 1), mhi = min(R.max_y, Y1 + 1);
        int lastx = -1;
#pragma unroll 1
        for (int kx = 0; kx < SRC_LINES; ++kx) {
            const int sx = src_line(kx, X, R.max_x, R.seam);
            if (sx < 0 || sx > R.max_x || sx <= lastx) continue;
            lastx = sx;
            const uint32_t cb = R.cell_off + (uint32_t)sx * (uint32_t)R.dh;
            int ra[3], rb[3], nr = 0;
            if (Y1 >= R.seam && mlo > 0) { ra[nr] = 0; rb[nr] = 0; ++nr; }   // bags >= seam take row 0
            ra[nr] = mlo; rb[nr] = mhi; ++nr;
            if (Y0 == 0) {  // row 0 takes rows seam..seam+3
                const int l2 = max(R.seam, mhi + 1), h2 = min(R.seam + SRC_LINES - 5, R.max_y);
                if (l2 <= h2) { ra[nr] = l2; rb[nr] = h2; ++nr; }
            }
#pragma unroll 1
            for (int r = 0; r < nr; ++r) {
                const uint32_t e = min(__ldg(a.start_cur + cb + (uint32_t)rb[r] + 1u), a.n);
                const uint32_t s = min(__ldg(a.start_cur + cb + (uint32_t)ra[r]), e);
#pragma unroll 1
                for (uint32_t f = s; f < e; f += 32u)
                    seg_batch<BPL>(a, f + lane < e, f + lane, c0, nb, sb, cnt, lane_lt, bad);
            }
        }
    }
#pragma unroll
    for (int h = 0; h < BPL; ++h) {
        const int bag = (int)lane + 32 * h;
        if (bag < nb && cnt[bag] != sb.hi[h] - sb.lo[h]) bad = true;
    }
    if (__any_sync(FULL_MASK, bad) && lane == 0u) atomicOr(a.err, ERR_REBIN_MISS | ERR_MISS_MATERIALIZE);
}

#ifndef KB_REBIN_MINB
#define KB_REBIN_MINB 6
#endif

#ifndef KB_REBIN_MINB_MULTI
#define KB_REBIN_MINB_MULTI 6
#endif

template <bool MULTI, int ROWS = SEG_ROWS>
__global__ void __launch_bounds__(32 * REBIN_SEG_WARPS, MULTI ? KB_REBIN_MINB_MULTI : KB_REBIN_MINB)
    k_rebin_seg(RebinArgs a) {
    pdl_enter();
    __shared__ uint32_t s_cnt[REBIN_SEG_WARPS][MULTI ? PACKED_SEG_ROWS : 32];
    const uint32_t w = threadIdx.x >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0 && a.step != nullptr) *a.step += 1ull;
    if (MULTI) {
        // one replica per block: its record is read once into shared memory
        __shared__ Rep sR;
        const uint2 e = a.sblk[blockIdx.x];
        load_rep_shared(&sR, a.reps + e.x);
        __syncthreads();
        const uint32_t g = e.y + w;
        // packed replicas always carry seg_rows == PACKED_SEG_ROWS (assign_segments)
        if (g >= sR.seg_off + rep_segments_dev(sR)) return;  // whole warps
        rebin_segment<PACKED_SEG_ROWS>(a, sR, g, s_cnt[w]);
        return;
    }
    const uint32_t g = blockIdx.x * REBIN_SEG_WARPS + w;
    if (g >= a.nsegs) return;  // whole warps
    rebin_segment<ROWS>(a, a.rep0, g, s_cnt[w]);
}

// ---------------------------------------------------------- ranked rebin
// Each write-list entry: its place in its next bag is the bag's
// next offset plus the number of arrivals of that bag that come before it in
// the list (the insertion order of the reference's lazy_update).  The force
// pass left the first RANK_SLOTS arrivals of every bag in a.slots, in no
// particular order, so a bag of at most RANK_ROW needs one 16-byte load and
// four compares, one of at most RANK_SLOTS two loads more.  The arrivals of a
// fuller bag are counted in the source lines of src_line, as the segment rebin
// does.  Bound by load latency and, at 1M boids, by the L2's capacity: the
// segment rebin's dependent rounds (offsets, keys, ranks, records) become two
// (key and record, read while the scan still runs; offsets and slots).
// Measured per step, force and scan
// included (us, segments against ranks): 20k boids 13.2 / 8.9, 262k 24.2 /
// 17.0, 1M 53.3 / 44.3, 1M at density 0.06 59.6 / 52.8; 512 packed replicas
// (8.4M boids) 592 / 511.  The force pass pays 1.5 of the 1M step's us for
// the slots (its counting atomics return a value).
//
// Fuller bags: the warp takes its distinct keys in turn; for each it reads the
// bag's source lines, and every lane of that key counts the arrivals before its
// own entry.  A chain of dependent loads bounds it, so the lanes look their own
// bags' replicas and columns up together before the first key, an interior
// bag's three columns are read as one list, 128 entries in flight (bounds and
// columns in turn per key, 32 entries at a time: 32 requests 21.5 ms against
// 20.6), and a bag at the seam or the edge has the bounds of all its lines
// loaded at once, a run per lane (line by line, up to 64 pairs of dependent
// loads, such bags held the whole step up as soon as a few were fuller: 64 x
// 4,096 boids at density 0.25 103 us a step, now 48, 64-bag segments 45; 16 x
// 65,536 with four crowded ones 162, 130, 167; 64 condensing replicas 96, 89,
// 101).  Every lane of the warp calls it with its
// entry i (over: the entry's bag is a fuller one).  Out of line and after the
// others are written, so that it costs them no registers.
// The source lines hold every arrival unless one has moved past them.  Each
// entry looks for its own place in its bag's lines; one that is not there would
// be missing from the other arrivals' counts, and raises the error word.
template <bool MULTI>
__device__ __noinline__ void place_by_lines(const RebinArgs& a, bool over, uint32_t i) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t key = 0, first = 0, rank = 0;
    int rep = 0;
    // an interior bag's source columns, entries [s, e) each, ascending
    uint32_t s0 = 0, e0 = 0, s1 = 0, e1 = 0, s2 = 0, e2 = 0;
    bool inner = false, seen = a.any_move != 0;
    if (over) {
        key = __ldcg(a.key + i);
        first = __ldg(a.start_next + key);
        if (!a.any_move) {
            if (MULTI) rep = rep_of_cell(a.reps, a.nrep, key);
            const Rep& R = MULTI ? a.reps[rep] : a.rep0;
            const uint32_t local = key - R.cell_off, dh = (uint32_t)R.dh;
            const uint32_t Xu = div_dh(local, R);
            const int X = (int)Xu, Y = (int)(local - Xu * dh);
            inner = X > 0 && X < R.seam && Y > 0 && Y < R.seam;
            if (inner) {
                const uint32_t* c = a.start_cur + key;
                e0 = min(__ldg(c - dh + 2), a.n), s0 = min(__ldg(c - dh - 1), e0);
                e1 = min(__ldg(c + 2), a.n), s1 = min(__ldg(c - 1), e1);
                e2 = min(__ldg(c + dh + 2), a.n), s2 = min(__ldg(c + dh - 1), e2);
                seen = i - s0 < e0 - s0 || i - s1 < e1 - s1 || i - s2 < e2 - s2;
            }
        }
    }
    uint32_t pending = __ballot_sync(FULL_MASK, over);
    while (pending) {
        const uint32_t leader = __ffs(pending) - 1;
        const uint32_t k = __shfl_sync(FULL_MASK, key, leader);
        const bool mine = over && key == k;
        pending &= ~__ballot_sync(FULL_MASK, mine);
        // nothing behind the last entry of this key matters
        const uint32_t last = __reduce_max_sync(FULL_MASK, mine ? i : 0u);
        if (__shfl_sync(FULL_MASK, inner ? 1 : 0, leader)) {
            // the three columns as one list, 128 entries in flight
            const uint32_t S0 = __shfl_sync(FULL_MASK, s0, leader), E0 = __shfl_sync(FULL_MASK, e0, leader);
            const uint32_t S1 = __shfl_sync(FULL_MASK, s1, leader), E1 = __shfl_sync(FULL_MASK, e1, leader);
            const uint32_t S2 = __shfl_sync(FULL_MASK, s2, leader), E2 = __shfl_sync(FULL_MASK, e2, leader);
            auto before = [&](uint32_t x) {  // entries of the list below index x
                return min(max(x, S0), E0) - S0 + (min(max(x, S1), E1) - S1) + (min(max(x, S2), E2) - S2);
            };
            const uint32_t L0 = E0 - S0, L1 = E1 - S1, T = before(last), own = before(i);
#pragma unroll 1
            for (uint32_t p = 0; p < T; p += 128u) {
                bool hit[4];
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    const uint32_t f = p + 32u * u + lane;
                    const uint32_t e = f < L0 ? S0 + f : (f - L0 < L1 ? S1 + (f - L0) : S2 + (f - L0 - L1));
                    hit[u] = f < T && __ldg(a.key + e) == k;
                }
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    const uint32_t m = __ballot_sync(FULL_MASK, hit[u]), q = p + 32u * u;
                    const uint32_t d = own > q ? own - q : 0u;
                    rank += mine ? __popc(d >= 32u ? m : m & ((1u << d) - 1u)) : 0;
                }
            }
            continue;
        }
        if (a.any_move) {
#pragma unroll 2
            for (uint32_t p = 0; p < last; p += 32u) {
                const bool hit = p + lane < last && __ldg(a.key + p + lane) == k;
                const uint32_t m = __ballot_sync(FULL_MASK, hit);
                // entries p .. i-1 of this batch
                const uint32_t d = i > p ? i - p : 0u;
                rank += mine ? __popc(d >= 32u ? m : m & ((1u << d) - 1u)) : 0;
            }
            continue;
        }
        // a bag at the seam or the field's edge: its source lines are up to
        // three runs of rows in up to six columns (src_line's, ascending), a
        // run per lane, and together one list, 64 entries in flight
        const Rep& R = MULTI ? a.reps[__shfl_sync(FULL_MASK, rep, leader)] : a.rep0;
        const uint32_t local = k - R.cell_off;
        const uint32_t Xu = div_dh(local, R);
        const int X = (int)Xu, Y = (int)(local - Xu * (uint32_t)R.dh);
        const int sx = src_line((int)(lane >> 2), X, R.max_x, R.seam), part = (int)(lane & 3u);
        int ra = 0, rb = -1;
        if (part == 0 && Y >= R.seam) rb = 0;  // bags from the seam on take row 0
        if (part == 1) ra = max(0, Y - 1), rb = min(R.max_y, Y + 1);
        if (part == 2 && Y == 0) ra = R.seam, rb = min(R.seam + SRC_LINES - 5, R.max_y);  // row 0 takes the seam's rows
        uint32_t s = 0, len = 0;
        if (sx >= 0 && sx <= R.max_x && ra <= rb) {
            const uint32_t* c = a.start_cur + R.cell_off + (uint32_t)sx * (uint32_t)R.dh;
            const uint32_t e = min(min(__ldg(c + rb + 1), a.n), last + 1u);
            s = min(__ldg(c + ra), e);
            len = e - s;
        }
        uint32_t incl = len;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL_MASK, incl, d);
            if (lane >= (uint32_t)d) incl += y;
        }
        const uint32_t T = __shfl_sync(FULL_MASK, incl, 31);
        s -= incl - len;  // entry f of the list is s + f, of the run that holds it
#pragma unroll 1
        for (uint32_t p = 0; p < T; p += 64u) {
            uint32_t at[2];
            bool hit[2];
#pragma unroll
            for (uint32_t u = 0; u < 2; ++u) {
                const uint32_t f = p + 32u * u + lane;
                // the first run whose inclusive count exceeds f
                uint32_t q = 0;
#pragma unroll
                for (uint32_t d = 16; d > 0; d >>= 1) {
                    const uint32_t y = __shfl_sync(FULL_MASK, incl, q + d - 1u);
                    if (y <= f) q += d;
                }
                const uint32_t base = __shfl_sync(FULL_MASK, s, q);
                at[u] = f < T ? base + f : 0xFFFFFFFFu;
                hit[u] = f < T && __ldg(a.key + at[u]) == k;
            }
#pragma unroll
            for (uint32_t u = 0; u < 2; ++u) {
                const uint32_t m = __ballot_sync(FULL_MASK, hit[u]);
                // the list ascends: how many of these 32 stand before entry i
                uint32_t d = 0;
#pragma unroll
                for (uint32_t h = 16; h > 0; h >>= 1) {
                    const uint32_t y = __shfl_sync(FULL_MASK, at[u], d + h - 1u);
                    if (y < i) d += h;
                }
                const uint32_t y = __shfl_sync(FULL_MASK, at[u], d);
                seen |= mine && y == i;
                if (y < i) ++d;
                rank += mine ? __popc(d >= 32u ? m : m & ((1u << d) - 1u)) : 0;
            }
        }
    }
    if (over && !seen) atomicOr(a.err, ERR_REBIN_MISS | ERR_MISS_MOVE);
    if (over && first + rank < a.n) {
        a.s_st[first + rank] = __ldcg(a.a_st + i);
        a.s_ids[first + rank] = __ldcg(a.a_ids + i);
    }
}

// Two entries per thread, their loads in flight together: a block of 256
// entries is over in about the time it takes to launch (1M boids: rebin 15.1 us
// with one entry per thread, 13.0 with two, 15.3 with four; step 43.8 / 41.9 /
// 43.6 us).  Fuller bags by warps rather than by each boid alone: 64 replicas
// whose flocks condense over 500 steps, last 100 steps 105 us each against 113
// for 64-bag segments (per-boid walks: no gain over segments there); with the
// ring force kernels 93, and 89 since a key's count stops at its last entry.
constexpr int RANK_ITEMS = 2;
constexpr int RANK_THREADS = 256;
// The plain form keeps 32 registers: with the 40 that place_by_lines would take
// it has 6 blocks per SM instead of 8 (1M boids, 100 steps: 4331 against 4295 us).
template <bool MULTI>
__global__ void __launch_bounds__(RANK_THREADS, MULTI ? 6 : 8) k_rebin_rank(RebinArgs a) {
    static_assert(RANK_ROW == 4 && RANK_ROW2 == 8, "the rows are read 16 bytes at a time");
    const uint32_t i0 = blockIdx.x * (RANK_THREADS * RANK_ITEMS) + threadIdx.x;
    uint32_t key[RANK_ITEMS], id[RANK_ITEMS];
    float4 rec[RANK_ITEMS];
    // the write list is the force pass's: the offsets scan in between has
    // waited for that pass before it let this kernel start, so the list is
    // read while the scan still runs
#pragma unroll
    for (int t = 0; t < RANK_ITEMS; ++t) {
        const uint32_t i = i0 + t * RANK_THREADS;
        if (i < a.n) {
            key[t] = __ldcg(a.key + i);
            rec[t] = __ldcg(a.a_st + i);
            id[t] = __ldcg(a.a_ids + i);
        }
    }
    pdl_enter();
    if (i0 == 0 && a.step != nullptr) *a.step += 1ull;
    uint32_t s[RANK_ITEMS], cnt[RANK_ITEMS];
#pragma unroll
    for (int t = 0; t < RANK_ITEMS; ++t) {
        s[t] = cnt[t] = 0u;
        if (i0 + t * RANK_THREADS < a.n) {
            const uint32_t e = min(__ldg(a.start_next + key[t] + 1), a.n);
            s[t] = min(__ldg(a.start_next + key[t]), e);
            cnt[t] = e - s[t];
        }
    }
    uint4 row[RANK_ITEMS];
#pragma unroll
    for (int t = 0; t < RANK_ITEMS; ++t)
        if (cnt[t] > 1u) row[t] = __ldg(reinterpret_cast<const uint4*>(a.slots) + key[t]);
#pragma unroll
    for (int t = 0; t < RANK_ITEMS; ++t) {
        const uint32_t i = i0 + t * RANK_THREADS, c = cnt[t];
        if (c > RANK_SLOTS) continue;
        uint32_t rank = 0;
        if (c > 1u) {
            const uint4 v = row[t];
            rank = (v.x < i) + (v.y < i) + (c > 2u && v.z < i) + (c > 3u && v.w < i);
            if (c > RANK_ROW) {
                const uint4* row2 = reinterpret_cast<const uint4*>(a.slots) + (size_t)a.ncells + 2u * (size_t)key[t];
                const uint4 u = __ldg(row2);
                rank += (u.x < i) + (c > 5u && u.y < i) + (c > 6u && u.z < i) + (c > 7u && u.w < i);
                if (c > 8u) {
                    const uint4 w = __ldg(row2 + 1);
                    rank += (w.x < i) + (c > 9u && w.y < i) + (c > 10u && w.z < i) + (c > 11u && w.w < i);
                }
            }
        }
        const uint32_t dst = s[t] + rank;
        if (i < a.n && dst < a.n) {
            a.s_st[dst] = rec[t];
            a.s_ids[dst] = id[t];
        }
    }
#pragma unroll
    for (int t = 0; t < RANK_ITEMS; ++t)
        if (__any_sync(FULL_MASK, cnt[t] > RANK_SLOTS))
            place_by_lines<MULTI>(a, cnt[t] > RANK_SLOTS, i0 + t * RANK_THREADS);
}

// Sum of squared bag occupancies of a read buffer (its offsets), a measure
// of how long the candidate lists are: about 9 * sum / N per boid.
// fuller > 0: the objects in bags of more than `fuller` instead.
__device__ __forceinline__ unsigned long long occupancy_term(unsigned long long o, uint32_t fuller) {
    return fuller ? (o > fuller ? o : 0ull) : o * o;
}
__global__ void k_occupancy_sq(const uint32_t* __restrict__ start, uint32_t ncells, uint32_t fuller,
                               unsigned long long* out) {
    __shared__ unsigned long long s_part[8];
    unsigned long long acc = 0;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < ncells; c += gridDim.x * blockDim.x) {
        const unsigned long long o = (unsigned long long)(start[c + 1] - start[c]);
        acc += occupancy_term(o, fuller);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_down_sync(FULL_MASK, acc, d);
    if ((threadIdx.x & 31u) == 0u) s_part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_part[w];
        atomicAdd(out, t);
    }
}

// ---------------------------------------------------------- general sort
__global__ void k_hist_list(const uint32_t* __restrict__ key, const uint8_t* __restrict__ dead,
                            uint32_t n, uint32_t* __restrict__ hist) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || (dead && dead[i])) return;
    atomicAdd(&hist[key[i]], 1u);
}

__global__ void k_scatter_list(const uint32_t* __restrict__ key, const uint8_t* __restrict__ dead,
                               const float4* __restrict__ st, const uint32_t* __restrict__ ids,
                               uint32_t n, const uint32_t* __restrict__ start,
                               uint32_t* __restrict__ cursor, float4* __restrict__ t_st,
                               uint32_t* __restrict__ t_ids, uint32_t* __restrict__ t_src) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || (dead && dead[i])) return;
    const uint32_t k = key[i];
    const uint32_t slot = start[k] + atomicAdd(&cursor[k], 1u);
    t_st[slot] = st[i];
    t_ids[slot] = ids[i];
    t_src[slot] = i;
}

// One thread per bag: order the bag's members by their write-list index
// (the reference's insertion order), then reset the bag's cursor.
__global__ void k_canon(const uint32_t* __restrict__ start, uint32_t ncells,
                        const float4* __restrict__ t_st, const uint32_t* __restrict__ t_ids,
                        const uint32_t* __restrict__ t_src, uint32_t* __restrict__ cursor,
                        float4* __restrict__ s_st, uint32_t* __restrict__ s_ids) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells) return;
    const uint32_t s = start[c], e = start[c + 1];
    if (s == e) return;
    cursor[c] = 0u;
    for (uint32_t m = s; m < e; ++m) {
        const uint32_t src = t_src[m];
        uint32_t rank = 0;
        for (uint32_t m2 = s; m2 < e; ++m2) rank += (t_src[m2] < src) ? 1u : 0u;
        s_st[s + rank] = t_st[m];
        s_ids[s + rank] = t_ids[m];
    }
}

// ---------------------------------------------------------- general rebuild
// The stable counting sort of any write list: count (k_count_list), offsets
// scan, then every entry to its place.  Arrival slots place the entries of
// bags of at most RANK_SLOTS arrivals at once (as k_rebin_rank); an entry of a
// fuller bag (or of any shared bag, without slots) leaves its index at the
// bag's offset plus its arrival number, and k_place_fuller puts each such bag
// in list order, a warp per bag.  A whole force pass has counted its list and
// kept the slots already; only the entries of fuller bags then take an arrival
// number, from the counts that the scan has zeroed.  Bound by the scattered writes.  Scattering
// every record and then ordering each bag by one thread (quadratic in the bag)
// took 52 us of a load of 1M uniform boids and 570 of 4M clustered ones; loads
// with their steps and reads: 1M x 100 steps 4415 -> 4278 us, 4M clustered x 10
// 10.48 -> 10.10 ms, 262k with no step 262 -> 213 us (k_load_facts included).
__global__ void __launch_bounds__(256)
    k_count_list(const uint32_t* __restrict__ key, const uint8_t* __restrict__ dead, uint32_t n,
                 uint32_t* __restrict__ hist, uint32_t* __restrict__ slots, uint32_t ncells,
                 uint32_t* __restrict__ arrival) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || (dead && dead[i])) return;
    const uint32_t k = key[i];
    const uint32_t r = atomicAdd(&hist[k], 1u);
    arrival[i] = r;
    if (slots) {
        if (r < RANK_ROW) slots[(size_t)k * RANK_ROW + r] = i;
        else if (r < RANK_SLOTS) slots[(size_t)ncells * RANK_ROW + (size_t)k * RANK_ROW2 + (r - RANK_ROW)] = i;
    }
}

__global__ void __launch_bounds__(256) k_place_list(PlaceArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n || (a.dead && a.dead[i])) return;
    const uint32_t key = a.key[i];
    const float4 rec = a.st[i];
    const uint32_t id = a.ids[i], r0 = a.arrival ? a.arrival[i] : 0u;
    // (offsets of a scan whose wait ran out read as k_place_fuller reads them)
    const uint32_t e = min(a.start[key + 1], a.n), s = min(a.start[key], e), c = e - s;
    uint32_t rank = 0;
    if (c > (a.slots ? RANK_SLOTS : 1u)) {
        const uint32_t r = a.arrival ? r0 : atomicAdd(&a.cursor[key], 1u);
        if (s + r < a.n) a.order[s + r] = i;
        return;
    }
    if (c > 1u) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(a.slots) + key);
        rank = (v.x < i) + (v.y < i) + (c > 2u && v.z < i) + (c > 3u && v.w < i);
        if (c > RANK_ROW) {
            const uint4* row2 = reinterpret_cast<const uint4*>(a.slots) + (size_t)a.ncells + 2u * (size_t)key;
            const uint4 u = __ldg(row2);
            rank += (u.x < i) + (c > 5u && u.y < i) + (c > 6u && u.z < i) + (c > 7u && u.w < i);
            if (c > 8u) {
                const uint4 w = __ldg(row2 + 1);
                rank += (w.x < i) + (c > 9u && w.y < i) + (c > 10u && w.z < i) + (c > 11u && w.w < i);
            }
        }
    }
    const uint32_t dst = s + rank;
    if (dst < a.n) {  // offsets of a scan whose wait ran out stay in bounds
        a.s_st[dst] = rec;
        a.s_ids[dst] = id;
    }
}

__global__ void __launch_bounds__(256) k_place_fuller(PlaceArgs a) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    uint32_t first = 0, cnt = 0;
    if (c < a.ncells) {
        const uint32_t e = min(a.start[c + 1], a.n);
        first = min(a.start[c], e);
        cnt = e - first;
    }
    const bool fuller = cnt > (a.slots ? RANK_SLOTS : 1u);
    if (fuller && !a.arrival) a.cursor[c] = 0u;  // zero again for the next count
    uint32_t todo = __ballot_sync(FULL_MASK, fuller);
    // offsets of a scan whose wait ran out can claim bags of any length
    if (todo && (*((volatile uint32_t*)a.err) & ERR_SPIN_TIMEOUT)) return;
    while (todo) {
        const uint32_t b = __ffs(todo) - 1;
        todo &= todo - 1u;
        const uint32_t s = __shfl_sync(FULL_MASK, first, b), m = __shfl_sync(FULL_MASK, cnt, b);
        for (uint32_t j = 0; j < m; j += 32u) {
            const uint32_t src = j + lane < m ? a.order[s + j + lane] : 0xFFFFFFFFu;
            uint32_t rank = 0;
            for (uint32_t q = 0; q < m; q += 32u) {
                const uint32_t o = q + lane < m ? a.order[s + q + lane] : 0xFFFFFFFFu;
#pragma unroll
                for (int l = 0; l < 32; ++l) rank += __shfl_sync(FULL_MASK, o, l) < src ? 1u : 0u;
            }
            if (src < a.n && rank < m) {
                a.s_st[s + rank] = a.st[src];
                a.s_ids[s + rank] = a.ids[src];
            }
        }
    }
}

// What a load of the read buffer has to know, in one launch and one read back
// (an 8 B hash slot per id, cleared each time, took 34 us at 1M ids):
// res[0] the sum of squared bag occupancies (packed replicas: the objects in bags
// of more than RANK_SLOTS; 0 for ncells 0), res[1] bit 0: an id below its replica's boid count repeats (its
// bit in `bits`), bit 1: some id is not below it (the caller compares by
// hashing), res[2] the objects stored.  res and bits are cleared by the caller.
__global__ void __launch_bounds__(256)
    k_load_facts(const Rep* __restrict__ reps, int32_t nrep, uint32_t nboids0, const uint32_t* __restrict__ ids,
                 const uint32_t* __restrict__ start, uint32_t ncells, const uint32_t* __restrict__ total,
                 uint32_t cap, uint32_t* bits, unsigned long long* res) {
    __shared__ unsigned long long s_part[8];
    const uint32_t n = min(*total, cap), g = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    uint32_t flags = 0;
    for (uint32_t k = g; k < n; k += step) {
        const uint32_t id = ids[k];
        uint32_t off = 0, most = nboids0;
        if (nrep > 1) {
            const Rep& R = reps[rep_of_boid(reps, nrep, k)];
            off = R.boid_off;
            most = R.nboids;
        }
        if (id < most && off + id < cap) {
            const uint32_t b = off + id, m = 1u << (b & 31u);
            if (atomicOr(bits + (b >> 5), m) & m) flags |= 1u;
        } else {
            flags |= 2u;
        }
    }
    // one atomic per warp, and none for what is known already: with ids past the
    // count, or repeated, every thread would come (loads of 200,000 such ids 295
    // and 206 us, now 174 and 147)
    flags = __reduce_or_sync(FULL_MASK, flags);
    if ((threadIdx.x & 31u) == 0u && (flags & ~(uint32_t)*((volatile unsigned long long*)(res + 1))))
        atomicOr(res + 1, (unsigned long long)flags);
    if (g == 0) res[2] = *total;
    if (ncells == 0) return;
    unsigned long long acc = 0;
    for (uint32_t c = g; c < ncells; c += step) {
        const unsigned long long o = (unsigned long long)(start[c + 1] - start[c]);
        acc += occupancy_term(o, nrep > 1 ? RANK_SLOTS : 0u);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) acc += __shfl_down_sync(FULL_MASK, acc, d);
    if ((threadIdx.x & 31u) == 0u) s_part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < 8; ++w) t += s_part[w];
        atomicAdd(res, t);
    }
}

// ---------------------------------------------------------- queries
// The query of one point whose range is at most 3 x 3 bags (QueryArgs::ring),
// in the order of the bag walk below.  A point's walk is a chain of loads, so
// the offsets of all its bags are loaded together, then its objects four at a
// time (200,000 exact queries of a 1M field: 60 us bag by bag, 28 so; relaxed
// counts 7, lists 21).  The
// exact query's corner rule compares extreme squares of the column and the row
// (see kb_ring.cu).  False: a skipped bag stands between kept ones (rounding at
// a bag's edge): the caller walks bag by bag.
template <int KIND>
__device__ __forceinline__ bool query_ring(const QueryArgs& a, float2 p, int mi, int Mi, int mj, int Mj,
                                           uint64_t off, bool fill, uint32_t* count, uint32_t* digest) {
    const Rep& R = a.rep;
    float ymin[3], ymax[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float nw = __fmul_rn((float)(mj + r), R.d);
        const float n0 = __fsub_rn(nw, p.y), n1 = __fsub_rn(fminf(__fadd_rn(nw, R.d), R.h), p.y);
        const float q0 = __fmul_rn(n0, n0), q1 = __fmul_rn(n1, n1);
        ymin[r] = fminf(q0, q1);
        ymax[r] = fmaxf(q0, q1);
    }
    uint32_t o[3][4];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const uint32_t c = R.cell_off + (uint32_t)(mi + k) * (uint32_t)R.dh + (uint32_t)mj;
#pragma unroll
        for (int r = 0; r < 4; ++r)
            o[k][r] = mi + k <= Mi ? __ldg(a.start + c + min(r, Mj - mj + 1)) : 0u;
    }
    uint32_t s[3], e[3], wl[3], wn[3];
    bool apart = false;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        s[k] = e[k] = wl[k] = wn[k] = 0u;
        if (mi + k > Mi) continue;
        uint32_t keep = 7u, whole = 7u;
        if (KIND == 1) {
            const float nw = __fmul_rn((float)(mi + k), R.d);
            const float n0 = __fsub_rn(nw, p.x), n1 = __fsub_rn(fminf(__fadd_rn(nw, R.d), R.w), p.x);
            const float q0 = __fmul_rn(n0, n0), q1 = __fmul_rn(n1, n1);
            const float xmin = fminf(q0, q1), xmax = fmaxf(q0, q1);
            keep = whole = 0u;
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                if (mj + r > Mj) continue;
                if (!(__fadd_rn(xmin, ymin[r]) > a.thr)) keep |= 1u << r;
                if (__fadd_rn(xmax, ymax[r]) <= a.thr) whole |= 1u << r;
            }
            apart |= keep == 5u || whole == 5u;
        }
        if (keep) {
            s[k] = (keep & 1u) ? o[k][0] : ((keep & 2u) ? o[k][1] : o[k][2]);
            e[k] = (keep & 4u) ? o[k][3] : ((keep & 2u) ? o[k][2] : o[k][1]);
        }
        if (whole) {
            wl[k] = (whole & 1u) ? o[k][0] : ((whole & 2u) ? o[k][1] : o[k][2]);
            wn[k] = ((whole & 4u) ? o[k][3] : ((whole & 2u) ? o[k][2] : o[k][1])) - wl[k];
        }
    }
    if (apart) return false;
    const uint32_t P1 = e[0] - s[0], P2 = P1 + (e[1] - s[1]), T = P2 + (e[2] - s[2]);
    if (KIND == 0 && !fill && !a.digest) {
        *count = T;
        return true;
    }
    uint32_t cnt = 0, dig = 0, pos = s[0], w0 = wl[0], w1 = wn[0];
    constexpr int U = 4;
    for (uint32_t f = 0; f < T;) {
        uint32_t at[U], id[U];
        float4 st[U];
        bool in[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (f == P1) { pos = s[1]; w0 = wl[1]; w1 = wn[1]; }
            if (f == P2) { pos = s[2]; w0 = wl[2]; w1 = wn[2]; }
            at[u] = pos;
            in[u] = f < T;
            const bool whole = pos - w0 < w1;
            if (in[u]) {
                id[u] = __ldg(a.ids + pos);
                if ((KIND == 1 && !whole) || a.out_st) st[u] = __ldg(a.st + pos);
            }
            if (KIND == 1 && in[u] && !whole) {
                // (an object may stand apart from the bag that it was set in)
                const float dx = toroidal_distance(p.x, st[u].x, R.w), dy = toroidal_distance(p.y, st[u].y, R.h);
                in[u] = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)) <= a.thr;
            }
            ++pos;
            ++f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (!in[u]) continue;
            if (fill && off + cnt < a.cap) {
                a.out_ids[off + cnt] = id[u];
                if (a.out_st) a.out_st[off + cnt] = st[u];
            }
            dig += id_mix(id[u]);
            ++cnt;
        }
    }
    *count = cnt;
    *digest = dig;
    return true;
}

template <int KIND>
__global__ void k_query(QueryArgs a) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= a.nq) return;
    const Rep& R = a.rep;
    const float2 p = a.q[q];
    const bool fill = a.offsets != nullptr;
    const uint64_t off = fill ? a.offsets[q] : 0;
    uint32_t cnt = 0, dig = 0;
    int mi, Mi, mj, Mj;
    const int32_t dd = (a.dist <= 0.0f) ? -1 : disc(a.dist, R);
    if (!cell_range(R, p.x, p.y, dd, &mi, &Mi, &mj, &Mj)) {
        // nothing in range
    } else if (a.ring && Mi - mi < 3 && Mj - mj < 3 &&
               query_ring<KIND>(a, p, mi, Mi, mj, Mj, off, fill, &cnt, &dig)) {
        // done
    } else {
        for (int ci = mi; ci <= Mi; ++ci) {
            const int bx = t_transform(ci, R.max_x);
            for (int cj = mj; cj <= Mj; ++cj) {
                const int by = t_transform(cj, R.max_y);
                const uint32_t c = R.cell_off + (uint32_t)bx * (uint32_t)R.dh + (uint32_t)by;
                const uint32_t s = a.start[c], e = a.start[c + 1];
                if (s == e) continue;
                int check = 1;
                if (KIND == 1) {
                    check = check_circle(bx, by, R, p.x, p.y, a.dist);
                    if (check == -1) continue;
                }
                for (uint32_t k = s; k < e; ++k) {
                    if (KIND == 1 && check == 0) {
                        const float4 o = a.st[k];
                        if (!(distance(p.x, p.y, o.x, o.y, R.w, R.h, R.toroidal != 0) <= a.dist))
                            continue;
                    }
                    const uint32_t id = a.ids[k];
                    if (fill && off + cnt < a.cap) {
                        a.out_ids[off + cnt] = id;
                        if (a.out_st) a.out_st[off + cnt] = a.st[k];
                    }
                    dig += id_mix(id);
                    ++cnt;
                }
            }
        }
    }
    if (!fill) {
        a.counts[q] = cnt;
        if (a.digest) a.digest[q] = dig;
    }
}

// ---------------------------------------------------------- ordered filters
// One block walks the list in chunks, keeping list order (write-buffer
// lookups are API calls, not the per-step path).
constexpr int FILTER_THREADS = 1024;

template <typename Pred, typename Emit>
__device__ void ordered_filter(uint32_t n, Pred pred, Emit emit, uint32_t* out_count) {
    __shared__ uint32_t s_warp[FILTER_THREADS / 32];
    __shared__ uint32_t s_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_base = 0;
    __syncthreads();
    for (uint32_t c0 = 0; c0 < n; c0 += FILTER_THREADS) {
        const uint32_t i = c0 + tid;
        const bool f = i < n && pred(i);
        const uint32_t bal = __ballot_sync(0xffffffffu, f);
        if (lane == 0) s_warp[warp] = __popc(bal);
        __syncthreads();
        uint32_t before = 0, total = 0;
        for (int w = 0; w < FILTER_THREADS / 32; ++w) {
            const uint32_t cw = s_warp[w];
            if (w < warp) before += cw;
            total += cw;
        }
        const uint32_t pos = s_base + before + __popc(bal & ((1u << lane) - 1u));
        if (f) emit(i, pos);
        __syncthreads();
        if (tid == 0) s_base += total;
        __syncthreads();
    }
    if (tid == 0) *out_count = s_base;
}

__global__ void __launch_bounds__(FILTER_THREADS)
    k_filter_key(const uint32_t* key, const uint8_t* dead, const float4* st, const uint32_t* ids,
                 uint32_t n, uint32_t target, uint32_t* out_ids, float4* out_st, uint64_t cap,
                 uint32_t* out_count) {
    ordered_filter(
        n, [&](uint32_t i) { return key[i] == target && !(dead && dead[i]); },
        [&](uint32_t i, uint32_t pos) {
            if (pos < cap) {
                if (out_ids) out_ids[pos] = ids[i];
                if (out_st) out_st[pos] = st[i];
            }
        },
        out_count);
}

__global__ void __launch_bounds__(FILTER_THREADS)
    k_empty_bags(Rep R, const uint32_t* start, float2* out, uint64_t cap, uint32_t* out_count) {
    ordered_filter(
        R.ncells, [&](uint32_t c) { return start[c + 1] == start[c]; },
        [&](uint32_t c, uint32_t pos) {
            if (pos < cap) {
                const uint32_t i = c / (uint32_t)R.dh, j = c % (uint32_t)R.dh;
                out[pos] = make_float2(__fmul_rn((float)i, R.d), __fmul_rn((float)j, R.d));
            }
        },
        out_count);
}

__global__ void k_remove(const uint32_t* key, uint8_t* dead, const uint32_t* ids, uint32_t n,
                         uint32_t target, uint32_t id, uint32_t* removed) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (key[i] == target && ids[i] == id && !dead[i]) {
        dead[i] = 1;
        atomicAdd(removed, 1u);
    }
}

__global__ void k_cell_of(const uint32_t* start, uint32_t ncells, uint32_t* cell_of) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells) return;
    for (uint32_t k = start[c]; k < start[c + 1]; ++k) cell_of[k] = c;
}

__global__ void k_cell_xy(Rep R, const uint32_t* cell_of, uint32_t n, float2* out) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t c = cell_of[k] - R.cell_off;
    const uint32_t i = c / (uint32_t)R.dh, j = c % (uint32_t)R.dh;
    out[k] = make_float2(__fmul_rn((float)i, R.d), __fmul_rn((float)j, R.d));
}

// Initial uniform flock of one boid: kb_gen_uniform (kb_gen.cpp) with every
// operation rounded once, so host and device draw the same bits.
__device__ void gen_uniform_boid(uint32_t id, uint32_t seed_lo, uint32_t seed_hi, float w, float h,
                                 float scale, float4* out) {
    U4 o = philox4x32_10(U4{id, 0u, 0u, STREAM_INIT}, seed_lo, seed_hi);
    const float x = __fmul_rn(w, unit_f32(o.x));
    const float y = __fmul_rn(h, unit_f32(o.y));
    uint32_t z = o.z, ww = o.w;
    float hx = 0.f, hy = 0.f;
    for (uint32_t attempt = 1; attempt < 1000u; ++attempt) {
        const float a = __fsub_rn(__fmul_rn(unit_f32(z), 2.0f), 1.0f);
        const float b = __fsub_rn(__fmul_rn(unit_f32(ww), 2.0f), 1.0f);
        const float r2 = __fadd_rn(__fmul_rn(a, a), __fmul_rn(b, b));
        if (r2 > 0.0f && r2 <= 1.0f) {
            const float r = __fsqrt_rn(r2);
            hx = __fdiv_rn(a, r);
            hy = __fdiv_rn(b, r);
            break;
        }
        o = philox4x32_10(U4{id, attempt, 0u, STREAM_INIT}, seed_lo, seed_hi);
        z = o.z;
        ww = o.w;
    }
    *out = make_float4(x, y, __fmul_rn(hx, scale), __fmul_rn(hy, scale));
}

__global__ void k_repack(const PackEntry* __restrict__ plan, int32_t nplan, uint32_t total,
                         const Rep* __restrict__ reps, const float4* __restrict__ src_st,
                         const uint32_t* __restrict__ src_ids, float4* __restrict__ dst_st,
                         uint32_t* __restrict__ dst_ids, uint32_t* __restrict__ dst_key,
                         uint8_t* __restrict__ dst_dead, uint32_t* err) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    int lo = 0, hi = nplan - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (plan[mid].dst_off <= i) lo = mid;
        else hi = mid - 1;
    }
    const PackEntry e = plan[lo];
    const uint32_t k = i - e.dst_off;
    if (k >= e.n) return;
    const Rep R = reps[e.rep];
    float4 st;
    uint32_t id;
    if (e.kind == 0) {
        st = src_st[e.src_off + k];
        id = src_ids[e.src_off + k];
    } else {
        id = k;
        gen_uniform_boid(k, e.seed_lo, e.seed_hi, R.w, R.h, e.heading_scale, &st);
    }
    const int64_t b = bag_index(R, disc(st.x, R), disc(st.y, R));
    if (b < 0) atomicOr(err, ERR_KEY_RANGE);
    dst_st[i] = st;
    dst_ids[i] = id;
    dst_key[i] = R.cell_off + (uint32_t)(b < 0 ? 0 : b);
    dst_dead[i] = 0;
}

// Per replica (one block each): {count, sum dx, sum dy, sum |(dx, dy)|} of
// the read buffer, in double.
__global__ void __launch_bounds__(256) k_moments(const Rep* __restrict__ reps,
                                                 const uint32_t* __restrict__ start,
                                                 const float4* __restrict__ st, double* out) {
    __shared__ double s_acc[4][8];
    const Rep& R = reps[blockIdx.x];
    const uint32_t lo = start[R.cell_off], hi = start[R.cell_off + R.ncells];
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    for (uint32_t k = lo + threadIdx.x; k < hi; k += blockDim.x) {
        const float4 o = st[k];
        const double dx = (double)o.z, dy = (double)o.w;
        a0 += dx;
        a1 += dy;
        a2 += sqrt(dx * dx + dy * dy);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a0 += __shfl_xor_sync(0xffffffffu, a0, o);
        a1 += __shfl_xor_sync(0xffffffffu, a1, o);
        a2 += __shfl_xor_sync(0xffffffffu, a2, o);
    }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        s_acc[0][w] = a0;
        s_acc[1][w] = a1;
        s_acc[2][w] = a2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t[3] = {0.0, 0.0, 0.0};
        for (int k = 0; k < 3; ++k)
            for (int v = 0; v < 8; ++v) t[k] += s_acc[k][v];
        out[4 * blockIdx.x + 0] = (double)(hi - lo);
        out[4 * blockIdx.x + 1] = t[0];
        out[4 * blockIdx.x + 2] = t[1];
        out[4 * blockIdx.x + 3] = t[2];
    }
}

// One thread per read-buffer slot: insert (replica, id) into an open-
// addressing table; a key that is already there is a repeat.
__global__ void k_dup_check(const Rep* __restrict__ reps, int32_t nrep, const uint32_t* __restrict__ ids,
                            uint32_t n, unsigned long long* table, uint32_t cap, uint32_t* dup) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t r = nrep > 1 ? (uint32_t)rep_of_boid(reps, nrep, k) : 0u;
    const unsigned long long key = ((unsigned long long)r << 32) | ids[k];
    uint32_t h = id_mix(ids[k] ^ (r * 0x9E3779B9u)) & (cap - 1u);
    for (uint32_t probe = 0; probe < cap; ++probe) {  // the table is at most half full
        const unsigned long long prev = atomicCAS(table + h, ~0ull, key);
        if (prev == ~0ull) return;
        if (prev == key) {
            *dup = 1u;
            return;
        }
        h = (h + 1u) & (cap - 1u);
    }
    *dup = 1u;  // no free slot found (cannot happen at half occupancy): be conservative
}

// The first object whose own column or row is no line of the matrix.
__device__ __forceinline__ void note_outside(const Rep& R, float x, float y, uint32_t i, uint32_t* first) {
    const int32_t cx = disc(x, R), cy = disc(y, R);
    if (cx < 0 || cx > R.max_x || cy < 0 || cy > R.max_y) atomicMin(first, i);
}

__global__ void k_pack_locations(Rep R, const float2* __restrict__ xy, const float2* __restrict__ dxy,
                                 uint32_t n, float4* __restrict__ out_st, uint32_t* __restrict__ out_key,
                                 uint8_t* __restrict__ out_dead, uint32_t* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float2 p = xy[i], d = dxy[i];
    const int64_t idx = bag_index(R, disc(p.x, R), disc(p.y, R));
    if (!(isfinite(p.x) && isfinite(p.y) && isfinite(d.x) && isfinite(d.y)) || idx < 0) {
        atomicMin(bad, i);
        return;
    }
    note_outside(R, p.x, p.y, i, bad + 1);
    out_st[i] = make_float4(p.x, p.y, d.x, d.y);
    out_key[i] = R.cell_off + (uint32_t)idx;
    out_dead[i] = 0;
}

// The same for records already packed as {x, y, last_d} (device-resident input).
__global__ void k_pack_states(Rep R, const float4* __restrict__ st, uint32_t n,
                              float4* __restrict__ out_st, uint32_t* __restrict__ out_key,
                              uint8_t* __restrict__ out_dead, uint32_t* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 v = st[i];
    const int64_t idx = bag_index(R, disc(v.x, R), disc(v.y, R));
    if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w)) || idx < 0) {
        atomicMin(bad, i);
        return;
    }
    note_outside(R, v.x, v.y, i, bad + 1);
    out_st[i] = v;
    out_key[i] = R.cell_off + (uint32_t)idx;
    out_dead[i] = 0;
}

__global__ void k_set_rep(Rep* dst, Rep v) { *dst = v; }
__global__ void k_set_u64(unsigned long long* dst, unsigned long long v) { *dst = v; }
__global__ void k_add_u64(unsigned long long* dst, unsigned long long v) { *dst += v; }

}  // namespace

cudaError_t launch_repack(const PackEntry* plan, int32_t nplan, uint32_t total, const Rep* reps,
                          const float4* src_st, const uint32_t* src_ids, float4* dst_st,
                          uint32_t* dst_ids, uint32_t* dst_key, uint8_t* dst_dead, uint32_t* err,
                          cudaStream_t s) {
    if (total == 0 || nplan <= 0) return cudaSuccess;
    k_repack<<<grid_for(total, 256), 256, 0, s>>>(plan, nplan, total, reps, src_st, src_ids, dst_st,
                                                   dst_ids, dst_key, dst_dead, err);
    return cudaGetLastError();
}

cudaError_t launch_moments(const Rep* reps, uint32_t nrep, const uint32_t* start, const float4* st,
                           double* out, cudaStream_t s) {
    if (nrep == 0) return cudaSuccess;
    k_moments<<<nrep, 256, 0, s>>>(reps, start, st, out);
    return cudaGetLastError();
}

cudaError_t launch_dup_check(const Rep* reps, int32_t nrep, const uint32_t* ids, uint32_t n,
                             unsigned long long* table, uint32_t cap, uint32_t* dup,
                             cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(table, 0xFF, sizeof(unsigned long long) * cap, s);
    if (e != cudaSuccess || n == 0) return e;
    k_dup_check<<<grid_for(n, 256), 256, 0, s>>>(reps, nrep, ids, n, table, cap, dup);
    return cudaGetLastError();
}

cudaError_t launch_pack_locations(const Rep& rep, const float2* xy, const float2* dxy, uint32_t n,
                                  float4* out_st, uint32_t* out_key, uint8_t* out_dead,
                                  uint32_t* bad, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_pack_locations<<<grid_for(n, 256), 256, 0, s>>>(rep, xy, dxy, n, out_st, out_key, out_dead, bad);
    return cudaGetLastError();
}

cudaError_t launch_pack_states(const Rep& rep, const float4* st, uint32_t n, float4* out_st,
                               uint32_t* out_key, uint8_t* out_dead, uint32_t* bad, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_pack_states<<<grid_for(n, 256), 256, 0, s>>>(rep, st, n, out_st, out_key, out_dead, bad);
    return cudaGetLastError();
}

cudaError_t launch_set_rep(Rep* dst, const Rep& v, cudaStream_t s) {
    k_set_rep<<<1, 1, 0, s>>>(dst, v);
    return cudaGetLastError();
}
cudaError_t launch_set_u64(unsigned long long* dst, unsigned long long v, cudaStream_t s) {
    k_set_u64<<<1, 1, 0, s>>>(dst, v);
    return cudaGetLastError();
}
cudaError_t launch_add_u64(unsigned long long* dst, unsigned long long v, cudaStream_t s) {
    k_add_u64<<<1, 1, 0, s>>>(dst, v);
    return cudaGetLastError();
}

// ====================================================================== launchers
cudaError_t launch_scan(const uint32_t* in, uint32_t* out, uint32_t n, ScanCtl* ctl,
                        unsigned long long* tile_state, uint32_t* err, bool zero_in,
                        cudaStream_t s, WaitCfg wait) {
    const uint32_t nt = scan_tiles(n);
    if (nt == 0) {
        return cudaMemsetAsync(out, 0, sizeof(uint32_t), s);
    }
    const uint32_t nt2 = (n + SCAN2_TILE - 1) / SCAN2_TILE;
    if (n <= SCAN_CLUSTER_MAX)
        return launch_pdl(k_scan_cluster, SCAN_CLUSTER, 1024, s, const_cast<uint32_t*>(in), out, n, zero_in ? 1 : 0);
    // tile_state holds scan_state_words(n) >= nt2 + 1 words: one sum per tile
    if (nt2 <= SCAN2_MAX_TILES) {
        cudaError_t e = launch_pdl(k_tile_sums, nt2, SCAN_THREADS, s, in, n, tile_state);
        if (e != cudaSuccess) return e;
        return launch_pdl(k_scan_tiles<false>, nt2, SCAN_THREADS, s, const_cast<uint32_t*>(in), out, n,
                          tile_state, zero_in ? 1 : 0, nt2);
    }
    // larger matrices: the tile sums scanned by one block in between (no
    // waits); the single-pass look-back scan below serves the largest ones
    // and the bounded-wait test of its look-back (wait.withhold)
    if (nt2 <= SCAN3_MAX_TILES && wait.withhold == ~0u) {
        cudaError_t e = launch_pdl(k_tile_sums, nt2, SCAN_THREADS, s, in, n, tile_state);
        if (e != cudaSuccess) return e;
        e = launch_pdl(k_scan_sums, 1u, (unsigned)SUMS_THREADS, s, tile_state, nt2);
        if (e != cudaSuccess) return e;
        return launch_pdl(k_scan_tiles<true>, nt2, SCAN_THREADS, s, const_cast<uint32_t*>(in), out, n,
                          tile_state, zero_in ? 1 : 0, nt2);
    }
    return launch_pdl(k_scan, nt, SCAN_THREADS, s, in, out, n, ctl, tile_state, err, zero_in ? 1 : 0, nt,
                      wait);
}

cudaError_t launch_flock_force(const ForceArgs& a, bool strict, int qmode, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    const bool multi = a.nrep > 1;
    if (multi && a.blk == nullptr) return cudaErrorInvalidValue;
    if (a.wide) return launch_flock_wide(a, strict, qmode, s);
    if (a.ring) return launch_flock_ring(a, strict, qmode, s);
    const unsigned g = multi ? a.nblk : grid_for(a.n, KB_FORCE_THREADS);
#define KB_FORCE(S, Q, MU)                                                                      \
    do {                                                                                        \
        if constexpr (MU) {                                                                     \
            if (a.block_threads == 128)                                                         \
                return launch_pdl(k_flock_force<S, Q, MU, false, 128>, g, 128, s, a);           \
            if (a.block_threads == 512)                                                         \
                return launch_pdl(k_flock_force<S, Q, MU, false, 512>, g, 512, s, a);           \
        }                                                                                       \
        return launch_pdl(k_flock_force<S, Q, MU>, g, KB_FORCE_THREADS, s, a);                  \
    } while (0)
    if (a.dense && qmode == 0 && !multi) {
        if (strict) return launch_pdl(k_flock_force<true, 0, false, true>, g, KB_FORCE_THREADS, s, a);
        return launch_pdl(k_flock_force<false, 0, false, true>, g, KB_FORCE_THREADS, s, a);
    }
    if (strict) {
        if (qmode == 0) { if (multi) KB_FORCE(true, 0, true); else KB_FORCE(true, 0, false); }
        else { if (multi) KB_FORCE(true, 1, true); else KB_FORCE(true, 1, false); }
    } else {
        if (qmode == 0) { if (multi) KB_FORCE(false, 0, true); else KB_FORCE(false, 0, false); }
        else { if (multi) KB_FORCE(false, 1, true); else KB_FORCE(false, 1, false); }
    }
#undef KB_FORCE
    return cudaGetLastError();
}

cudaError_t launch_flock_agents(const ForceArgs& a, const float4* in_st, const uint32_t* in_ids,
                               uint32_t nin, bool strict, int qmode, cudaStream_t s) {
    if (nin == 0) return cudaSuccess;
    if (a.nrep != 1) return cudaErrorInvalidValue;
    const unsigned g = grid_for(nin, KB_FORCE_THREADS);
    if (strict) {
        if (qmode == 0) k_flock_agents<true, 0><<<g, KB_FORCE_THREADS, 0, s>>>(a, in_st, in_ids, nin);
        else k_flock_agents<true, 1><<<g, KB_FORCE_THREADS, 0, s>>>(a, in_st, in_ids, nin);
    } else {
        if (qmode == 0) k_flock_agents<false, 0><<<g, KB_FORCE_THREADS, 0, s>>>(a, in_st, in_ids, nin);
        else k_flock_agents<false, 1><<<g, KB_FORCE_THREADS, 0, s>>>(a, in_st, in_ids, nin);
    }
    return cudaGetLastError();
}

cudaError_t launch_find_ids(const uint32_t* ids, const uint8_t* dead, const float4* st, uint32_t n,
                            const uint32_t* sorted, uint32_t m, uint32_t* first, float4* out,
                            cudaStream_t s) {
    if (m == 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(first, 0xFF, sizeof(uint32_t) * m, s);
    if (e != cudaSuccess) return e;
    if (n) k_find_ids<<<grid_for(n, 256), 256, 0, s>>>(ids, dead, n, sorted, m, first);
    k_gather_found<<<grid_for(m, 256), 256, 0, s>>>(st, first, m, out);
    return cudaGetLastError();
}

cudaError_t launch_remove_ids(const uint32_t* ids, uint8_t* dead, uint32_t n, const uint32_t* sorted,
                              uint32_t m, uint32_t* removed, cudaStream_t s) {
    if (n == 0 || m == 0) return cudaSuccess;
    k_remove_ids<<<grid_for(n, 256), 256, 0, s>>>(ids, dead, n, sorted, m, removed);
    return cudaGetLastError();
}

cudaError_t launch_rebin(const RebinArgs& a, cudaStream_t s) {
    if (a.slots != nullptr) {
        if (a.key == nullptr && a.n > 0) return cudaErrorInvalidValue;
        const unsigned gr = grid_for(a.n > 0 ? a.n : 1, RANK_THREADS * RANK_ITEMS);
        return a.nrep > 1 ? launch_pdl(k_rebin_rank<true>, gr, RANK_THREADS, s, a)
                          : launch_pdl(k_rebin_rank<false>, gr, RANK_THREADS, s, a);
    }
    if (a.key != nullptr && a.nsegs > 0 && (a.nrep == 1 || a.sblk != nullptr)) {
        if (a.nrep > 1) return launch_pdl(k_rebin_seg<true>, a.nsblk, 32 * REBIN_SEG_WARPS, s, a);
        const unsigned gs = grid_for(a.nsegs, REBIN_SEG_WARPS);
        if (a.seg_rows == DENSE_SEG_ROWS)
            return launch_pdl(k_rebin_seg<false, DENSE_SEG_ROWS>, gs, 32 * REBIN_SEG_WARPS, s, a);
        if (a.seg_rows != 0 && a.seg_rows != SEG_ROWS) return cudaErrorInvalidValue;
        return launch_pdl(k_rebin_seg<false>, gs, 32 * REBIN_SEG_WARPS, s, a);
    }
    const unsigned g = grid_for(a.ncells > 0 ? a.ncells : 1, 256);
    if (a.nrep > 1) k_rebin<true><<<g, 256, 0, s>>>(a);
    else k_rebin<false><<<g, 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_occupancy_sq(const uint32_t* start, uint32_t ncells, uint32_t fuller, unsigned long long* out,
                                cudaStream_t s) {
    if (ncells == 0) return cudaSuccess;
    const unsigned g0 = grid_for(ncells, 256);
    const unsigned g = g0 < 4u * GB300_SMS ? g0 : 4u * GB300_SMS;  // grid-stride: four blocks per SM
    k_occupancy_sq<<<g, 256, 0, s>>>(start, ncells, fuller, out);
    return cudaGetLastError();
}

cudaError_t launch_count_list(const uint32_t* key, const uint8_t* dead, uint32_t n, uint32_t* hist,
                              uint32_t* slots, uint32_t ncells, uint32_t* arrival, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_count_list<<<grid_for(n, 256), 256, 0, s>>>(key, dead, n, hist, slots, ncells, arrival);
    return cudaGetLastError();
}

cudaError_t launch_place_list(const PlaceArgs& a, cudaStream_t s) {
    if (a.n == 0 || a.ncells == 0) return cudaSuccess;
    k_place_list<<<grid_for(a.n, 256), 256, 0, s>>>(a);
    k_place_fuller<<<grid_for(a.ncells, 256), 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_load_facts(const Rep* reps, int32_t nrep, uint32_t nboids0, const uint32_t* ids,
                              const uint32_t* start, uint32_t ncells, const uint32_t* total, uint32_t cap,
                              uint32_t* bits, unsigned long long* res, cudaStream_t s) {
    const uint64_t most = cap > ncells ? cap : ncells;
    const unsigned g0 = grid_for(most > 0 ? most : 1, 256);
    const unsigned g = g0 < 8u * GB300_SMS ? g0 : 8u * GB300_SMS;  // grid-stride: eight blocks per SM
    k_load_facts<<<g, 256, 0, s>>>(reps, nrep, nboids0, ids, start, ncells, total, cap, bits, res);
    return cudaGetLastError();
}

cudaError_t launch_hist_list(const uint32_t* key, const uint8_t* dead, uint32_t n, uint32_t* hist,
                             cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_hist_list<<<grid_for(n, 256), 256, 0, s>>>(key, dead, n, hist);
    return cudaGetLastError();
}

cudaError_t launch_scatter_list(const uint32_t* key, const uint8_t* dead, const float4* st,
                                const uint32_t* ids, uint32_t n, const uint32_t* start,
                                uint32_t* cursor, float4* t_st, uint32_t* t_ids, uint32_t* t_src,
                                cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_scatter_list<<<grid_for(n, 256), 256, 0, s>>>(key, dead, st, ids, n, start, cursor, t_st,
                                                     t_ids, t_src);
    return cudaGetLastError();
}

cudaError_t launch_canon(const uint32_t* start, uint32_t ncells, const float4* t_st,
                         const uint32_t* t_ids, const uint32_t* t_src, uint32_t* cursor,
                         float4* s_st, uint32_t* s_ids, cudaStream_t s) {
    if (ncells == 0) return cudaSuccess;
    k_canon<<<grid_for(ncells, 256), 256, 0, s>>>(start, ncells, t_st, t_ids, t_src, cursor, s_st,
                                                  s_ids);
    return cudaGetLastError();
}

cudaError_t launch_query(const QueryArgs& a, cudaStream_t s) {
    if (a.nq == 0) return cudaSuccess;
    QueryArgs b = a;
    query_ring_args(&b);
    const unsigned g = grid_for(a.nq, 128);
    if (a.kind == 1) k_query<1><<<g, 128, 0, s>>>(b);
    else k_query<0><<<g, 128, 0, s>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_filter_key(const uint32_t* key, const uint8_t* dead, const float4* st,
                              const uint32_t* ids, uint32_t n, uint32_t target, uint32_t* out_ids,
                              float4* out_st, uint64_t cap, uint32_t* out_count, cudaStream_t s) {
    k_filter_key<<<1, FILTER_THREADS, 0, s>>>(key, dead, st, ids, n, target, out_ids, out_st, cap,
                                              out_count);
    return cudaGetLastError();
}

cudaError_t launch_remove(const uint32_t* key, uint8_t* dead, const uint32_t* ids, uint32_t n,
                          uint32_t target, uint32_t id, uint32_t* removed, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_remove<<<grid_for(n, 256), 256, 0, s>>>(key, dead, ids, n, target, id, removed);
    return cudaGetLastError();
}

cudaError_t launch_empty_bags(const Rep& rep, const uint32_t* start, float2* out, uint64_t cap,
                              uint32_t* out_count, cudaStream_t s) {
    k_empty_bags<<<1, FILTER_THREADS, 0, s>>>(rep, start, out, cap, out_count);
    return cudaGetLastError();
}

cudaError_t launch_cell_of(const uint32_t* start, uint32_t ncells, uint32_t* cell_of,
                           cudaStream_t s) {
    if (ncells == 0) return cudaSuccess;
    k_cell_of<<<grid_for(ncells, 256), 256, 0, s>>>(start, ncells, cell_of);
    return cudaGetLastError();
}

cudaError_t launch_cell_xy(const Rep& rep, const uint32_t* cell_of, uint32_t n, float2* out,
                           cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_cell_xy<<<grid_for(n, 256), 256, 0, s>>>(rep, cell_of, n, out);
    return cudaGetLastError();
}

}  // namespace kb
