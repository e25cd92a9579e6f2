// kb_small.cu -- whole steps of a small field in one thread-block cluster.
//
// A field of at most SMALL_MAX_BOIDS boids and SMALL_MAX_CELLS bags (the
// 1,000-boid Flockers case, the reference's own test fields) is launch-bound
// on the separate-kernel path: four launches per step for a few microseconds
// of work.  Here a cluster of SMALL_CTAS blocks runs every step of the call
// in one launch.  Each block holds the read buffer it needs and all bag offsets
// in shared memory and owns one contiguous chunk of the boids:
//   1. agent pass: half of the threads walk the candidates of the chunk's boids
//      (the same candidate order, accumulator and finish as k_flock_force), the
//      other half draws their jitter meanwhile; next states and ids go to a
//      local write list, and the bag keys, eight to a 16-byte store, into every
//      block's list of keys (distributed shared memory);
//   -- cluster barrier --
//   2. lazy_update: every block counts all keys in its own shared memory and
//      scans the counts into the next bag offsets; a boid's place is its bag's
//      offset, plus the arrivals from lower-ranked blocks (earlier in list
//      order), plus those of earlier warps of its chunk (one byte per warp and
//      bag), plus its rank among its warp's equal keys (__match_any_sync): the
//      reference's insertion order inside a bag.  Each record goes to the blocks
//      whose next chunk can see its column (to all where queries wrap, or birds
//      stand beyond the height);
//   -- cluster barrier --
// and every block writes its chunk of the final read buffer back.  No bound on
// how far a boid moves is needed.
//
// Bound by latency: a step is one pass over some two thousand instructions
// between barriers, by few warps.  us per step at 300 / 1000 / 2048 / 4000 boids,
// fast: 3.6 / 4.0 / 4.9 / 7.6, with one warp ranking the chunk in turn, every
// record sent to all blocks and two candidates at a time without the packed
// walk 6.5 / 7.1 / 9.3 / 13.8; strict at 1000: 4.8 against 8.6.  Exact query,
// strict, 300 / 1000 / 4000: 5.3 / 5.6 / 9.9 against 17.4 / 17.9 / 25.2 bag by
// bag with check_circle (separate kernels: 8.4 / 9.4 / 10.1).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "kb_common.h"
#include "kb_device.cuh"
#include "kb_launch.h"
#include "kb_walk.cuh"

namespace cg = cooperative_groups;

namespace kb {
namespace {

constexpr uint32_t SMALL_FULL = 0xFFFFFFFFu;

// One candidate of the relaxed query in list order: self is skipped (by
// slot when ids are unique, else by id).
template <bool STRICT>
__device__ __forceinline__ void take_small(const Rep& R, const uint32_t* ids, uint32_t p, float4 o,
                                           float4 me, uint32_t my_id, uint32_t my_slot,
                                           Acc<STRICT>& acc) {
    const bool self = my_slot != 0xFFFFFFFFu ? p == my_slot : ids[p] == my_id;
    if (!self) acc.add(R, me.x, me.y, o);
}

// Bird::step's candidate sums for `me` against a read buffer in shared
// memory: the query's cells x-outer / y-inner (t_transform wraps the range
// where the field does), each bag in insertion order, the exact query's
// corner rule (check_circle) for QMODE 1.  Self is the slot my_slot when ids
// are unique, else every candidate with the boid's id.  The relaxed query of
// a clamped one-bag ring (the common case) walks its three column runs as one
// flat list, four candidates per iteration, so that their loads and reciprocals
// overlap (the sums are still taken in list order: the same bits).
template <bool STRICT, int QMODE>
__device__ __forceinline__ void gather_small(const Rep& R, const float4* st, const uint32_t* ids,
                                             const uint32_t* start, float4 me, uint32_t my_id,
                                             uint32_t my_slot, Acc<STRICT>& acc) {
    int mi, Mi, mj, Mj;
    if (!cell_range(R, me.x, me.y, R.dd, &mi, &Mi, &mj, &Mj)) return;
    if (QMODE == 1 && R.nowrap && R.dd <= 1 && my_slot != 0xFFFFFFFFu) {  // nowrap: a clamped torus
        Sums<STRICT> sums;
        walk_exact<STRICT, 2, false>(st, start, start[R.ncells], R, me, my_slot, mi, Mi, mj, Mj, sums);
        acc = sums.result();
        return;
    }
    if (QMODE == 0 && R.toroidal && !R.cell_wrap && Mi - mi < 3) {
        uint32_t s[3], e[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            s[k] = e[k] = 0u;
            if (mi + k <= Mi) {
                const uint32_t colbase = (uint32_t)(mi + k) * (uint32_t)R.dh;
                s[k] = start[colbase + (uint32_t)mj];
                e[k] = start[colbase + (uint32_t)Mj + 1u];
            }
        }
        if (R.nowrap && my_slot != 0xFFFFFFFFu) {
            const Runs r = {{s[0], s[1], s[2]}, {e[0], e[1], e[2]}};
            pair_t<STRICT> mxy;
            pack2(mxy, me.x, me.y);
            Sums<STRICT> sums;
            walk_flat<STRICT, 4, false>(st, mxy, my_slot, r, sums);
            bool self_in = false;
#pragma unroll
            for (int k = 0; k < 3; ++k) self_in |= my_slot - s[k] < e[k] - s[k];
            sums.count = sums.vec - (self_in ? 1u : 0u);
            acc = sums.result();
            return;
        }
#pragma unroll 1
        for (int k = 0; k < 3; ++k) {
            const uint32_t ks = k == 0 ? s[0] : (k == 1 ? s[1] : s[2]), ke = k == 0 ? e[0] : (k == 1 ? e[1] : e[2]);
            acc.vec += ke - ks;
            for (uint32_t q = ks; q < ke; ++q) take_small(R, ids, q, st[q], me, my_id, my_slot, acc);
        }
        return;
    }
    if (QMODE == 0 && R.toroidal && !R.cell_wrap) {  // wider rings: a run per column
        for (int ci = mi; ci <= Mi; ++ci) {
            const uint32_t colbase = (uint32_t)ci * (uint32_t)R.dh;
            const uint32_t e = start[colbase + (uint32_t)Mj + 1u];
            const uint32_t s = start[colbase + (uint32_t)mj];
            if (s < e) acc.vec += e - s;
            for (uint32_t k = s; k < e; ++k) take_small(R, ids, k, st[k], me, my_id, my_slot, acc);
        }
        return;
    }
    for (int ci = mi; ci <= Mi; ++ci) {
        const int bx = t_transform(ci, R.max_x);
        const uint32_t colbase = (uint32_t)bx * (uint32_t)R.dh;
        for (int cj = mj; cj <= Mj; ++cj) {
            const int by = t_transform(cj, R.max_y);
            const uint32_t c = colbase + (uint32_t)by;
            const uint32_t s = start[c], e = start[c + 1];
            if (s == e) continue;
            int check = 1;
            if (QMODE == 1) {
                check = check_circle(bx, by, R, me.x, me.y, R.radius);
                if (check == -1) continue;
            }
            for (uint32_t k = s; k < e; ++k) {
                const float4 o = st[k];
                if (QMODE == 1 && check == 0 &&
                    !(distance(me.x, me.y, o.x, o.y, R.w, R.h, R.toroidal != 0) <= R.radius))
                    continue;
                acc.vec += 1;
                const bool self = my_slot != 0xFFFFFFFFu ? k == my_slot : ids[k] == my_id;
                if (!self) acc.add(R, me.x, me.y, o);
            }
        }
    }
}

// Exclusive scan of v[0..n) in place, v[n] = total, by one block of T threads
// (n <= SMALL_MAX_CELLS; v has room for whole vectors of 4, zero past n).
template <int T>
__device__ __forceinline__ void block_scan_small(uint32_t* v, uint32_t n, uint32_t* warp_sums) {
    constexpr int ITEMS = (int)SMALL_MAX_CELLS / T, NW = T / 32;
    static_assert(ITEMS % 4 == 0 && NW <= 32, "scan tiling");
    const uint32_t t = threadIdx.x, lane = t & 31u, w = t >> 5, b = t * ITEMS;
    uint4 q[ITEMS / 4];
    uint32_t sum = 0;
#pragma unroll
    for (int j = 0; j < ITEMS / 4; ++j) {
        q[j] = make_uint4(0u, 0u, 0u, 0u);
        if (b + 4 * j < n) q[j] = *reinterpret_cast<const uint4*>(v + b + 4 * j);
        sum += q[j].x + q[j].y + q[j].z + q[j].w;
    }
    uint32_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(SMALL_FULL, incl, d);
        if (lane >= (uint32_t)d) incl += y;
    }
    if (lane == 31u) warp_sums[w] = incl;
    __syncthreads();
    // every warp scans the warp sums itself
    const uint32_t x = lane < (uint32_t)NW ? warp_sums[lane] : 0u;
    uint32_t xi = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(SMALL_FULL, xi, d);
        if (lane >= (uint32_t)d) xi += y;
    }
    uint32_t run = __shfl_sync(SMALL_FULL, xi - x, w) + incl - sum;
#pragma unroll
    for (int j = 0; j < ITEMS / 4; ++j) {
        uint4 o;
        o.x = run;
        o.y = o.x + q[j].x;
        o.z = o.y + q[j].y;
        o.w = o.z + q[j].z;
        run = o.w + q[j].w;
        if (b + 4 * j < n) *reinterpret_cast<uint4*>(v + b + 4 * j) = o;
    }
    // the total stands behind the last count (its vector may reach past n)
    const uint32_t total = __shfl_sync(SMALL_FULL, xi, 31);
    __syncthreads();
    if (t == 0) v[n] = total;
}

// Boids per block: the chunk, a multiple of 8 (keys travel eight at a time).
__host__ __device__ inline uint32_t small_chunk(uint32_t n) {
    return ((n + SMALL_CTAS - 1) / SMALL_CTAS + 7u) / 8u * 8u;
}
// Words of warp counters per bag: one byte per warp of the chunk.
__host__ __device__ inline uint32_t small_words(uint32_t chunk) { return ((chunk + 31u) / 32u + 3u) / 4u; }

// Shared-memory layout (byte offsets), the same in every block of the cluster.
struct SmallLayout {
    uint32_t rd_st, wr_st, jit, rd_id, wr_id, wr_key, keys, start, nstart, cur, warps, bytes;
};
__host__ __device__ inline SmallLayout small_layout(uint32_t n, uint32_t ncells, uint32_t chunk) {
    SmallLayout L{};
    uint32_t o = 0;
    const uint32_t cells = (ncells + 8u) / 8u * 8u;  // room for one more word and whole vectors
    L.rd_st = o;  o += n * 16u;
    L.wr_st = o;  o += chunk * 16u;
    L.keys = o;   o += SMALL_CTAS * chunk * 2u;
    L.jit = o;    o += chunk * 8u;
    L.start = o;  o += cells * 4u;
    L.nstart = o; o += cells * 4u;
    L.warps = o;  o += cells * 4u * small_words(chunk);
    L.cur = o;    o += cells * 2u;
    L.rd_id = o;  o += n * 4u;
    L.wr_id = o;  o += chunk * 4u;
    L.wr_key = o; o += chunk * 4u;
    L.bytes = o;
    return L;
}

constexpr uint32_t SMALL_OUTSIDE = 0xFFFFu;  // a key outside the matrix (its boid goes to bag 0)
constexpr uint32_t SMALL_NONE = 0xFFFEu;     // no boid

// Shared memory of the cluster's blocks by 32-bit addresses.
__device__ __forceinline__ uint32_t remote_address(const void* local, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;"
        : "=r"(r)
        : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
    return r;
}
__device__ __forceinline__ void store_remote(uint32_t at, uint4 v) {
    asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void store_remote(uint32_t at, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}

// T: threads per block, at least twice the chunk.
template <bool STRICT, int QMODE, int T>
__global__ void __launch_bounds__(T, 1) k_small_steps(SmallArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    cg::cluster_group cl = cg::this_cluster();
    const Rep& R = a.rep;
    const uint32_t n = a.n, C = R.ncells;
    const uint32_t rank = cl.block_rank();
    const uint32_t chunk = small_chunk(n), words = small_words(chunk);
    const uint32_t lo = min(n, rank * chunk), m = min(n, lo + chunk) - lo;
    const SmallLayout Lo = small_layout(n, C, chunk);
    float4* rd_st = reinterpret_cast<float4*>(smem + Lo.rd_st);
    uint32_t* rd_id = reinterpret_cast<uint32_t*>(smem + Lo.rd_id);
    uint32_t* start = reinterpret_cast<uint32_t*>(smem + Lo.start);
    uint32_t* nstart = reinterpret_cast<uint32_t*>(smem + Lo.nstart);  // arrivals per bag, then offsets
    uint32_t* cur = reinterpret_cast<uint32_t*>(smem + Lo.cur);  // arrivals from lower-ranked blocks, 16 bits a bag
    uint32_t* warps = reinterpret_cast<uint32_t*>(smem + Lo.warps);  // arrivals per warp of the chunk, a byte each
    uint16_t* keys = reinterpret_cast<uint16_t*>(smem + Lo.keys);  // every boid's next bag
    float4* wr_st = reinterpret_cast<float4*>(smem + Lo.wr_st);
    float2* jit = reinterpret_cast<float2*>(smem + Lo.jit);
    uint32_t* wr_id = reinterpret_cast<uint32_t*>(smem + Lo.wr_id);
    uint32_t* wr_key = reinterpret_cast<uint32_t*>(smem + Lo.wr_key);
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t line[2][SMALL_CTAS];  // columns of each block's next first and last boid
    __shared__ uint32_t s_err, s_all;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    const uint32_t walkers = (chunk + 31u) / 32u * 32u;  // whole warps
    for (uint32_t i = t; i < n; i += T) {
        rd_st[i] = a.st[i];
        rd_id[i] = a.ids[i];
    }
    for (uint32_t c = t; c <= C; c += T) start[c] = a.start[c];
    for (uint32_t c = t; c < C * words; c += T) warps[c] = 0u;
    if (t < 2u * SMALL_CTAS) line[t / SMALL_CTAS][t % SMALL_CTAS] = 0u;
    if (t == 0) {
        s_err = 0u;
        // records go to every block where a query can wrap, where birds stand
        // beyond the height (y wraps with the width), in bags of other columns
        // than their positions', and from the step on in which a position fell
        // outside the matrix
        s_all = R.toroidal && !R.cell_wrap && R.w <= R.h ? 0u : 1u;
    }
    // a thread writes to one other block: keys, records and ids of block t % 8
    static_assert(T % SMALL_CTAS == 0 && SMALL_CTAS == 8, "one target block per thread");
    const uint32_t key_q = remote_address(keys, t % SMALL_CTAS);
    const uint32_t st_q = remote_address(rd_st, t % SMALL_CTAS), id_q = remote_address(rd_id, t % SMALL_CTAS);
    unsigned long long step = *a.step;
    // every block of the cluster is running (its shared memory may be written
    // through the cluster) and has its whole copy loaded before any thread
    // reads a neighbour
    cl.sync();
    for (uint32_t s = 0; s < a.nsteps; ++s, ++step) {
        // 1. agent pass over the own chunk: candidates by the first threads,
        //    jitter by the last
        if (t >= walkers) {  // meanwhile: the counters
            // (to the end of the last whole vector, which the scan adds up)
            for (uint32_t c = t - walkers; c < (C + 4u) / 4u * 4u; c += T - walkers) nstart[c] = 0u;
            for (uint32_t c = t - walkers; c < (C + 1u) / 2u; c += T - walkers) cur[c] = 0u;
        }
        Acc<STRICT> acc;
        float4 me = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < m) {
            me = rd_st[lo + t];
            gather_small<STRICT, QMODE>(R, rd_st, rd_id, start, me, rd_id[lo + t],
                                        a.self_by_slot ? lo + t : 0xFFFFFFFFu, acc);
        } else if (t >= T / 2 && t - T / 2 < m) {
            jit[t - T / 2] = bird_jitter<STRICT>(R, rd_id[lo + t - T / 2], step);
        }
        __syncthreads();
        if (t < walkers) {
            uint32_t key = SMALL_NONE;
            if (t < m) {
                const float4 nx = finish_bird_with<STRICT>(R, me, acc, [&] { return jit[t]; });
                const int64_t idx = bag_index(R, disc(nx.x, R), disc(nx.y, R));
                uint32_t flags = 0;
                if (idx < 0) flags |= ERR_KEY_RANGE;
                if (!isfinite(nx.x) || !isfinite(nx.y)) flags |= ERR_NONFINITE;
                if (flags) atomicOr(&s_err, flags);
                key = idx < 0 ? SMALL_OUTSIDE : (uint32_t)idx;
                wr_st[t] = nx;
                wr_id[t] = rd_id[lo + t];
                wr_key[t] = idx < 0 ? 0u : (uint32_t)idx;
            }
            // eight keys a store, lane q of each eight to block q
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t k0 = __shfl_sync(SMALL_FULL, key, (lane & 24u) + 2 * k);
                const uint32_t k1 = __shfl_sync(SMALL_FULL, key, (lane & 24u) + 2 * k + 1);
                w[k] = k0 | (k1 << 16);
            }
            const uint32_t at = t & ~7u;
            if (at < chunk) store_remote(key_q + (rank * chunk + at) * 2u, make_uint4(w[0], w[1], w[2], w[3]));
        }
        cl.sync();  // every copy of the keys is complete; no block reads rd_* any more
        // 2. arrivals per bag, and per bag those of lower-ranked blocks (earlier
        //    in the list)
        for (uint32_t i = t; i < SMALL_CTAS * chunk; i += T) {
            uint32_t k = keys[i];
            if (k == SMALL_NONE) continue;
            if (k == SMALL_OUTSIDE) {
                k = 0u;
                s_all = 1u;
            }
            atomicAdd(&nstart[k], 1u);
            if (i < lo) atomicAdd(&cur[k >> 1], 1u << (16u * (k & 1u)));
        }
        // equal keys of a warp of the chunk
        uint32_t my_key = 0, r = 0;
        if (t < walkers) {
            const bool valid = t < m;
            my_key = valid ? wr_key[t] : 0xFFFFFFFFu;
            const uint32_t peers = __match_any_sync(SMALL_FULL, my_key);
            r = __popc(peers & ((1u << lane) - 1u));
            if (valid && r == 0u)
                atomicAdd(&warps[my_key * words + (warp >> 2)], (uint32_t)__popc(peers) << (8u * (warp & 3u)));
        }
        __syncthreads();
        block_scan_small<T>(nstart, C, warp_sums);
        __syncthreads();
        if (t >= T / 2) {  // the columns of every chunk's first and last boid
            for (uint32_t x = t - T / 2; x < (uint32_t)R.dw; x += T / 2) {
                const uint32_t from = nstart[x * (uint32_t)R.dh], to = nstart[(x + 1u) * (uint32_t)R.dh];
#pragma unroll
                for (uint32_t q = 0; q < SMALL_CTAS; ++q) {
                    const uint32_t first = q * chunk, last = min(n, first + chunk) - 1u;
                    if (first < n && first - from < to - from) line[0][q] = x;
                    if (first < n && last - from < to - from) line[1][q] = x;
                }
            }
        }
        if (t < m) {
            uint32_t before = r;
            for (uint32_t q = 0; q < words; ++q) {
                uint32_t v = warps[my_key * words + q];
                if (q == (warp >> 2)) v &= (1u << (8u * (warp & 3u))) - 1u;
                else if (q > (warp >> 2)) v = 0u;
                before += (uint32_t)__dp4a(v, 0x01010101u, 0u);
            }
            const uint32_t lower = (cur[my_key >> 1] >> (16u * (my_key & 1u))) & 0xFFFFu;
            wr_key[t] = nstart[my_key] + lower + before;  // the key becomes the destination slot
        }
        __syncthreads();
        if (t < m)
            for (uint32_t q = 0; q < words; ++q) warps[my_key * words + q] = 0u;
        // the blocks whose next chunk can see a record get it
        const uint32_t q = t % SMALL_CTAS;
        uint32_t from = 0u, to = n;
        if (s_all == 0u) {
            const uint32_t dd = (uint32_t)max(R.dd, 0), x0 = line[0][q];
            from = nstart[(x0 > dd ? x0 - dd : 0u) * (uint32_t)R.dh];
            to = q * chunk < n ? nstart[(min(line[1][q] + dd, (uint32_t)R.dw - 1u) + 1u) * (uint32_t)R.dh] : from;
        }
        for (uint32_t j = t / SMALL_CTAS; j < m; j += T / SMALL_CTAS) {
            const uint32_t pos = wr_key[j];
            if (pos - from < to - from) {
                store_remote(st_q + pos * 16u, reinterpret_cast<const uint4*>(wr_st)[j]);
                store_remote(id_q + pos * 4u, wr_id[j]);
            }
        }
        uint32_t* const o = start;
        start = nstart;
        nstart = o;
        cl.sync();  // every copy of the next read buffer is complete; counters are free
    }
    if (t < m) {
        a.st[lo + t] = rd_st[lo + t];
        a.ids[lo + t] = rd_id[lo + t];
    }
    if (rank == 0) {
        for (uint32_t c = t; c <= C; c += T) a.start[c] = start[c];
        if (t == 0) *a.step = step;
    }
    __syncthreads();
    if (t == 0 && s_err) atomicOr(a.err, s_err);
}

}  // namespace

size_t small_smem_bytes(uint32_t n, uint32_t ncells) { return small_layout(n, ncells, small_chunk(n)).bytes; }

namespace {

template <int T>
cudaError_t launch_small(const SmallArgs& a, bool strict, int qmode, cudaStream_t s) {
    void (*k)(SmallArgs) = strict ? (qmode == 0 ? k_small_steps<true, 0, T> : k_small_steps<true, 1, T>)
                                  : (qmode == 0 ? k_small_steps<false, 0, T> : k_small_steps<false, 1, T>);
    // the largest layout once per kernel (and device), not per launch
    static thread_local int opted[4] = {-1, -1, -1, -1};
    const int ki = (strict ? 2 : 0) + (qmode == 0 ? 0 : 1);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (opted[ki] != dev) {
        const size_t most = small_smem_bytes(SMALL_MAX_BOIDS, SMALL_MAX_CELLS);
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
        if (e != cudaSuccess) return e;
        opted[ki] = dev;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(SMALL_CTAS, 1, 1);
    cfg.blockDim = dim3(T, 1, 1);
    cfg.dynamicSmemBytes = small_smem_bytes(a.n, a.rep.ncells);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = SMALL_CTAS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, a);
}

}  // namespace

cudaError_t launch_small_steps(const SmallArgs& a, bool strict, int qmode, cudaStream_t s) {
    if (a.nsteps == 0) return cudaSuccess;
    if (a.n == 0 || a.n > SMALL_MAX_BOIDS || a.rep.ncells > SMALL_MAX_CELLS || a.rep.cell_off != 0)
        return cudaErrorInvalidValue;
    // two threads per boid of a chunk: fewer warps at every barrier for small flocks
    return small_chunk(a.n) <= 256u ? launch_small<512>(a, strict, qmode, s)
                                    : launch_small<1024>(a, strict, qmode, s);
}

}  // namespace kb
