// kb_launch.h -- host-side launchers of the kernels in kb_kernels.cu.  Every
// launcher enqueues on the given stream and returns the launch error.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "kb_common.h"

namespace kb {

// Scan workspace: a tile counter, a finish counter and an epoch that tags
// the per-tile look-back words, so the scan needs no reset between launches
// (and replays correctly inside a CUDA graph).
struct ScanCtl {
    uint32_t tile_counter;
    uint32_t done_counter;
    uint32_t epoch;
    uint32_t _pad;
};
constexpr unsigned GB300_SMS = 152;
constexpr uint32_t SCAN_TILE = 4096;  // items per CTA (256 threads x 16)
inline uint32_t scan_tiles(uint32_t n) { return (n + SCAN_TILE - 1) / SCAN_TILE; }
constexpr uint32_t SCAN_CLUSTER = 8;  // blocks of the one-launch cluster scan
constexpr uint32_t SCAN_CLUSTER_MAX = SCAN_CLUSTER * 1024u * 4u;  // its bags
// Items per tile of the two-pass scan (inputs of up to SCAN2_MAX_TILES tiles).
#ifndef KB_SCAN2_ITEMS
#define KB_SCAN2_ITEMS 4
#endif
constexpr uint32_t SCAN2_TILE = 256u * KB_SCAN2_ITEMS;
#ifndef KB_SCAN2_MAX
#define KB_SCAN2_MAX 4096
#endif
constexpr uint32_t SCAN2_MAX_TILES = KB_SCAN2_MAX;
// Above SCAN2_MAX_TILES tiles a third launch scans the tile sums (up to
// SCAN3_MAX_TILES tiles, about 268 M bags); beyond it the look-back scan.
#ifndef KB_SCAN3_MAX
#define KB_SCAN3_MAX 262144
#endif
constexpr uint32_t SCAN3_MAX_TILES = KB_SCAN3_MAX;
// 64-bit state words a scan of n items needs (either form).
inline uint32_t scan_state_words(uint32_t n) {
    const uint32_t a = scan_tiles(n), b = (n + SCAN2_TILE - 1) / SCAN2_TILE;
    return (a > b ? a : b) + 1u;
}

// Bounded device waits: the iterations a wait makes before it gives up and
// raises ERR_SPIN_TIMEOUT (0: the kernel's default), and a test hook that
// makes one publisher (a look-back scan tile, a persistent block at its first
// grid barrier) withhold its signal so that a wait runs out on purpose
// (~0u: none).
struct WaitCfg {
    uint32_t spin_limit;
    uint32_t withhold;
};
constexpr WaitCfg WAIT_DEFAULT = {0u, 0xFFFFFFFFu};

// Exclusive scan of in[0..n) into out[0..n]; out[n] = total.  When zero_in,
// in[] is cleared as it is read (the histogram is ready for the next step).
cudaError_t launch_scan(const uint32_t* in, uint32_t* out, uint32_t n, ScanCtl* ctl,
                        unsigned long long* tile_state, uint32_t* err, bool zero_in,
                        cudaStream_t s, WaitCfg wait = WAIT_DEFAULT);

// Flock step agent pass: reads the canonical read buffer (st, ids, start),
// writes next states into the write list in the same order plus each one's
// new bag key, and counts keys into hist.
struct ForceArgs {
    const Rep* reps;
    int32_t nrep;
    Rep rep0;  // the single replica, read from the parameter bank when nrep == 1
    const float4* st;
    const uint32_t* ids;
    const uint32_t* start;
    uint32_t n;
    const unsigned long long* step;
    float4* out_st;
    uint32_t* out_ids;
    uint32_t* out_key;
    uint32_t* hist;
    // the first RANK_SLOTS arrivals of every bag (their write-list slots, in
    // the order the counts were taken), for the ranked rebin; nullptr: not kept
    uint32_t* slots;
    uint32_t ncells;  // bags over all replicas (the second row of a.slots starts behind them)
    uint32_t* err;
    int32_t apart;  // objects may stand apart from their bags: no replica's nowrap holds
    int32_t check_moves;  // flag moves the stencil-gather rebin cannot follow
    // several replicas: one block per entry {replica, first boid}; no block
    // spans two replicas (built by the host with the replica table)
    const uint2* blk;
    uint32_t nblk;
    // ids are unique within every replica: a candidate is the boid itself
    // exactly when it is the boid's own slot, so no id is loaded per candidate
    int32_t self_by_slot;
    // long candidate lists (dense flocks, single replica): walk each column
    // run with a plain pointer instead of the flat index formula (the same
    // visiting order, fewer instructions per candidate)
    int32_t dense;
    // several replicas: threads per block of the block table (FORCE_BLOCKS_*;
    // 0: FORCE_THREADS), the launch shape the batch autotuner picks
    uint32_t block_threads;
    // every replica is a torus with the clamped range, no pair straddles the
    // seam (Rep::nowrap, and every object in its own position's bag), the ring is at most one bag wide, ids are distinct
    // and n <= 2^26 (byte offsets of three runs in 32 bits): the ring kernels
    int32_t ring;
    // the same with a wider ring, one replica of at most wide_max boids: the
    // warp-per-boid kernel
    int32_t wide;
};
// Up to how many boids the warp-per-boid kernel is the faster one: it gives a
// boid 32 lanes, k_flock_force gives it one and waits for its columns in turn.
// The general kernel's time hardly grows with the flock up to 64k boids and
// grows with the columns, the warp-per-boid kernel's the other way round, so the
// line lies by columns.  us per step, warp / thread per boid, density 0.025:
//   relaxed, 5 columns  8k 10.8 / 13.2, 12k 12.5 / 13.3, 14k 13.7 / 13.7, 16k 15.1 / 14.1
//            (strict 12.4 / 15.9, 15.2 / 16.1, 16.6 / 16.5, 18.2 / 16.8)
//            7          8k 11.3 / 16.1, 16k 15.3 / 15.8, 32k 24.7 / 18.4
//            21         16k 17.9 / 32.7, 32k 27.6 / 35.5
//            41         1k 10.1 / 47, 20k 31 / 59
//   exact,   5          33k 35 / 45, 40k 42 / 45, 49k 50 / 45, 262k 227 / 92 (strict 40k 48 / 48)
//            7          66k 64 / 76, 98k 93 / 84, 262k 231 / 148 (strict 66k 74 / 81)
//            9          131k 124 / 141 (strict 142 / 151)
//            11         262k 243 / 310; 17: 275 / 590; 41: 131k 342 / 1098 (a corner rule per bag)
// The same at densities 0.01 and 0.06.
inline uint32_t wide_max(int32_t dd, int32_t qmode) {
    if (qmode != 0) return dd <= 2 ? 40000u : (dd == 3 ? 65536u : (dd == 4 ? 131072u : 262144u));
    return dd <= 2 ? 12288u : (2 * dd + 1 >= 16 ? 32768u : 16384u);
}
constexpr int FORCE_THREADS = 256;  // the force kernel's block (one replica per block)
// Block sizes of the force pass over packed replicas (one replica per block).
constexpr int FORCE_BLOCK_SIZES[3] = {128, 256, 512};
cudaError_t launch_flock_force(const ForceArgs& a, bool strict, int qmode, cudaStream_t s);
// The same for a.ring flocks (kb_ring.cu); launch_flock_force calls it.
cudaError_t launch_flock_ring(const ForceArgs& a, bool strict, int qmode, cudaStream_t s);
cudaError_t launch_flock_wide(const ForceArgs& a, bool strict, int qmode, cudaStream_t s);
// Whole steps of a small single-replica field in one cluster of SMALL_CTAS
// blocks (kb_small.cu): every block loads the read buffer (st, ids, start
// over rep.ncells bags) into its shared memory, nsteps steps run there, and
// the final read buffer, offsets and step counter (*step += nsteps) are
// written back.
constexpr uint32_t SMALL_CTAS = 8;  // a portable cluster size
// Measured on GB300 (uniform flocks, 400-step calls): 4.5 / 4.0 / 4.9 / 7.6 us
// per step at 16 / 1000 / 2048 / 4000 boids, against 8.0 to 8.3 us for the
// separate kernels; the bound is the shared memory.
constexpr uint32_t SMALL_MAX_BOIDS = 4096;
constexpr uint32_t SMALL_MAX_CELLS = 4096;
constexpr uint32_t SMALL_SINGLE_MAX = 1200;  // boids up to which a single step takes the cluster
constexpr uint32_t SMALL_DENSE_WIDE = 2000;  // from here on crowded wide rings of relaxed queries leave it
struct SmallArgs {
    Rep rep;
    float4* st;
    uint32_t* ids;
    uint32_t* start;
    uint32_t n;
    uint32_t nsteps;
    unsigned long long* step;
    uint32_t* err;
    int32_t self_by_slot;
};
size_t small_smem_bytes(uint32_t n, uint32_t ncells);
cudaError_t launch_small_steps(const SmallArgs& a, bool strict, int qmode, cudaStream_t s);

// Bird::step of nin caller-given agents (in_st {x, y, dx, dy}, in_ids) against
// the read buffer of a single replica; agent j's next state, id and bag key
// go to slot j of a.out_st / a.out_ids / a.out_key, its arrival into a.hist.
cudaError_t launch_flock_agents(const ForceArgs& a, const float4* in_st, const uint32_t* in_ids,
                               uint32_t nin, bool strict, int qmode, cudaStream_t s);

// Stencil-gather rebin: builds the canonical read buffer of the next step
// from the write list (in the previous canonical order) and the scanned
// histogram.  Bumps *step when step != nullptr.  With key == nullptr each
// record's bag is recomputed from its position.
struct RebinArgs {
    const Rep* reps;
    int32_t nrep;
    Rep rep0;  // the single replica when nrep == 1
    const uint32_t* start_cur;
    const uint32_t* start_next;
    const uint32_t* key;
    const float4* a_st;
    const uint32_t* a_ids;
    uint32_t ncells;
    uint32_t nsegs;  // column segments over all replicas (0: per-bag kernel only)
    int32_t seg_rows;  // bags per segment of a single replica: 0 (SEG_ROWS) or DENSE_SEG_ROWS
    // several replicas: one block per entry {replica, first segment}, up to
    // REBIN_SEG_WARPS segments of that replica
    const uint2* sblk;
    uint32_t nsblk;
    float4* s_st;
    uint32_t* s_ids;
    unsigned long long* step;
    uint32_t* err;
    uint32_t n;  // records (every slot index is below it)
    const uint32_t* slots;  // the force pass's arrival slots: the ranked rebin (nullptr: by segments)
    // moves may cross more than one bag: a fuller bag's arrivals are counted in
    // the whole list (ranked rebin only, up to RANK_ANY_MAX records)
    int32_t any_move;
};
// Arrivals per bag whose write-list slots the force pass records: the first
// four of every bag in one array of 16 B per bag, the next eight in a second
// one of 32 B per bag behind it that bags of ordinary occupancy never touch.
// (A single row of 8 or 16 per bag ran the 1M step at 47.2 or 52.0 us against
// 44.6 us for a row of 4: the step's working set is near the L2's size.)
constexpr uint32_t RANK_ROW = 4, RANK_ROW2 = 8;
constexpr uint32_t RANK_SLOTS = RANK_ROW + RANK_ROW2;
// Records up to which the ranked rebin takes flocks whose moves the source
// lines do not cover: a warp then reads the whole list for each of its fuller
// bags (about 10 us at this length).
constexpr uint32_t RANK_ANY_MAX = 32768;
// Bag matrices up to this many bags carry the arrival slots (48 B per bag).
constexpr uint32_t RANK_MAX_CELLS = 1u << 26;
// Bag segments of the segment rebin: SEG_ROWS consecutive bags of one column.
constexpr int SEG_ROWS = 32;
// Shorter segments for dense flocks: a segment's source runs are long there,
// and the warp walks them in order, so fewer rows per warp shorten the tail.
constexpr int DENSE_SEG_ROWS = 8;
constexpr int REBIN_SEG_WARPS = 8;  // segments (warps) per block
// Segments of the replicas of a packed batch: 64 bags (two per lane), half
// as many segments as 32-bag ones (the packed rebin's time follows the
// number of segments; measured on the 512-replica sweep).
constexpr int PACKED_SEG_ROWS = 64;
// rows 0: the replica's own segment height (Rep::seg_rows, else SEG_ROWS).
inline uint32_t rep_segments(const Rep& R, int rows = 0) {
    if (rows == 0) rows = R.seg_rows > 0 ? R.seg_rows : SEG_ROWS;
    return (uint32_t)R.dw * (((uint32_t)R.dh + (uint32_t)rows - 1) / (uint32_t)rows);
}
cudaError_t launch_rebin(const RebinArgs& a, cudaStream_t s);
// *out += sum over bags of (start[c+1] - start[c])^2, or with fuller > 0 the
// objects in bags of more than `fuller` (the caller zeroes *out).
cudaError_t launch_occupancy_sq(const uint32_t* start, uint32_t ncells, uint32_t fuller, unsigned long long* out,
                                cudaStream_t s);
// Whether any (replica, id) pair repeats in the read buffer (n boids, nrep
// replicas by boid_off): an open-addressing table of cap (a power of two,
// >= 2n) 64-bit words, cleared here; *dup is set to 1 on a repeat.
cudaError_t launch_dup_check(const Rep* reps, int32_t nrep, const uint32_t* ids, uint32_t n,
                             unsigned long long* table, uint32_t cap, uint32_t* dup,
                             cudaStream_t s);
// out[4r..4r+3] = {boids, sum dx, sum dy, sum |(dx,dy)|} of replica r's read buffer.
cudaError_t launch_moments(const Rep* reps, uint32_t nrep, const uint32_t* start, const float4* st,
                           double* out, cudaStream_t s);

// Bulk set_object_location on the device: n objects at their own positions
// (xy and dxy as float2 arrays) appended to the write list as records, bag
// keys and live marks; bad[0] takes the smallest index of an object with a
// non-finite value or a location outside the bag matrix, bad[1] that of one
// whose own column or row is no line of the matrix (~0u when none).
cudaError_t launch_pack_locations(const Rep& rep, const float2* xy, const float2* dxy, uint32_t n,
                                  float4* out_st, uint32_t* out_key, uint8_t* out_dead,
                                  uint32_t* bad, cudaStream_t s);
// The same for records already packed as float4 {x, y, last_d} on the device.
cudaError_t launch_pack_states(const Rep& rep, const float4* st, uint32_t n, float4* out_st,
                               uint32_t* out_key, uint8_t* out_dead, uint32_t* bad, cudaStream_t s);

// The general rebuild: counts (hist zero before; arrival[i] = entry i's arrival
// number, the bags' first RANK_SLOTS arrivals into slots unless nullptr), and
// after the offsets scan every live entry to its place in list order.  order:
// n words of scratch.  A list that a force pass counted has no arrival numbers
// (nullptr): fuller bags take them from cursor, zero before and after.
struct PlaceArgs {
    const uint32_t* key;
    const uint8_t* dead;
    const float4* st;
    const uint32_t* ids;
    uint32_t n;
    const uint32_t* arrival;
    uint32_t* cursor;
    const uint32_t* start;
    uint32_t ncells;
    const uint32_t* slots;
    uint32_t* order;
    float4* s_st;
    uint32_t* s_ids;
    const uint32_t* err;
};
cudaError_t launch_count_list(const uint32_t* key, const uint8_t* dead, uint32_t n, uint32_t* hist,
                              uint32_t* slots, uint32_t ncells, uint32_t* arrival, cudaStream_t s);
cudaError_t launch_place_list(const PlaceArgs& a, cudaStream_t s);
// res[0..2] = {sum of squared bag occupancies over ncells bags (several replicas:
// the objects in bags of more than RANK_SLOTS), id flags (1 a
// repeat among the ids below their replica's boid count, 2 an id that is not
// below it), objects stored}; bits: one bit per record (cap of them), cleared
// with res by the caller.  nboids0: the boid count of a single replica.
cudaError_t launch_load_facts(const Rep* reps, int32_t nrep, uint32_t nboids0, const uint32_t* ids,
                              const uint32_t* start, uint32_t ncells, const uint32_t* total, uint32_t cap,
                              uint32_t* bits, unsigned long long* res, cudaStream_t s);

// Stable counting sort of the write list by key (insertion order
// kept inside each bag): histogram, scatter, per-bag canonicalisation.
cudaError_t launch_hist_list(const uint32_t* key, const uint8_t* dead, uint32_t n, uint32_t* hist,
                             cudaStream_t s);
cudaError_t launch_scatter_list(const uint32_t* key, const uint8_t* dead, const float4* st,
                                const uint32_t* ids, uint32_t n, const uint32_t* start,
                                uint32_t* cursor, float4* t_st, uint32_t* t_ids, uint32_t* t_src,
                                cudaStream_t s);
cudaError_t launch_canon(const uint32_t* start, uint32_t ncells, const float4* t_st,
                         const uint32_t* t_ids, const uint32_t* t_src, uint32_t* cursor,
                         float4* s_st, uint32_t* s_ids, cudaStream_t s);

// Field2D queries over the read buffer of a single replica.
//   mode 0: counts only (+ digest when digest != nullptr)
//   mode 1: fill ids/states at offsets[q]
struct QueryArgs {
    Rep rep;
    int32_t kind;  // 0 relax, 1 exact
    float dist;
    const uint32_t* start;
    const float4* st;
    const uint32_t* ids;
    uint32_t nq;
    const float2* q;
    uint32_t* counts;
    uint32_t* digest;
    const uint32_t* offsets;
    uint32_t* out_ids;
    float4* out_st;
    uint64_t cap;
    // set by launch_query: the range is clamped and at most one bag around the
    // point's own, and no distance in it wraps; the largest square within dist
    int32_t ring;
    float thr;
};
// ring and thr of a query by its geometry and distance.
void query_ring_args(QueryArgs* a);
cudaError_t launch_query(const QueryArgs& a, cudaStream_t s);

// Ordered filter of the write list: entries with key == target and not dead,
// in list order; writes ids/states (up to cap) and the count.
cudaError_t launch_filter_key(const uint32_t* key, const uint8_t* dead, const float4* st,
                              const uint32_t* ids, uint32_t n, uint32_t target, uint32_t* out_ids,
                              float4* out_st, uint64_t cap, uint32_t* out_count, cudaStream_t s);
// Mark write-list entries (key == target, id == id, live) dead; adds the
// number marked to *removed.
cudaError_t launch_remove(const uint32_t* key, uint8_t* dead, const uint32_t* ids, uint32_t n,
                          uint32_t target, uint32_t id, uint32_t* removed, cudaStream_t s);
// For each id sorted[j] (ascending, distinct): first[j] = the first index i
// < n with ids[i] == sorted[j] (skipping dead entries when dead != nullptr),
// ~0u when none, and out[j] = st[first[j]] (zeros when none).
cudaError_t launch_find_ids(const uint32_t* ids, const uint8_t* dead, const float4* st, uint32_t n,
                            const uint32_t* sorted, uint32_t m, uint32_t* first, float4* out,
                            cudaStream_t s);
// Mark live write-list entries whose id is in sorted[0..m) (ascending) dead;
// adds the number marked to *removed.
cudaError_t launch_remove_ids(const uint32_t* ids, uint8_t* dead, uint32_t n, const uint32_t* sorted,
                              uint32_t m, uint32_t* removed, cudaStream_t s);
// Empty bags of the read buffer in index order, as (i*d, j*d).
cudaError_t launch_empty_bags(const Rep& rep, const uint32_t* start, float2* out, uint64_t cap,
                              uint32_t* out_count, cudaStream_t s);
// Bag index of every stored object (read buffer), for iteration.
cudaError_t launch_cell_of(const uint32_t* start, uint32_t ncells, uint32_t* cell_of,
                           cudaStream_t s);
// (i*d, j*d) of the bag of each object.
cudaError_t launch_cell_xy(const Rep& rep, const uint32_t* cell_of, uint32_t n, float2* out,
                           cudaStream_t s);

// Repacking plan for a continuous batch: each entry fills write-list slots
// [dst_off, dst_off+n) for replica `rep`, either copying its canonical
// records from the read buffer (kind 0, from src_off) or generating its
// initial uniform flock (kind 1: kb_gen_uniform's draws, bit for bit).
struct PackEntry {
    uint32_t dst_off, n, rep, src_off;
    uint32_t kind, seed_lo, seed_hi;
    float heading_scale;
};
cudaError_t launch_repack(const PackEntry* plan, int32_t nplan, uint32_t total, const Rep* reps,
                          const float4* src_st, const uint32_t* src_ids, float4* dst_st,
                          uint32_t* dst_ids, uint32_t* dst_key, uint8_t* dst_dead, uint32_t* err,
                          cudaStream_t s);

}  // namespace kb
