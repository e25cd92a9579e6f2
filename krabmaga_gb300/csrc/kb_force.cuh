// kb_force.cuh -- what the force kernels share: programmatic dependent
// launch, a replica record in shared memory, and the end of an agent's step.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "kb_common.h"
#include "kb_device.cuh"
#include "kb_launch.h"

namespace kb {
namespace {

// Programmatic dependent launch.  The step's kernels are launched so that
// the next one may be scheduled before the previous one ends; each first
// waits until its predecessor has finished and its writes are visible
// (griddepcontrol.wait, before touching any memory), then lets its own
// successor launch (griddepcontrol.launch_dependents).  Launched without the
// attribute, the wait returns at once.
#ifndef KB_PDL
#define KB_PDL 1
#endif
__device__ __forceinline__ void pdl_enter() {
#if KB_PDL
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#endif
}

template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), unsigned grid, unsigned block, cudaStream_t s,
                       Args... args) {
#if KB_PDL
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
#else
    kernel<<<grid, block, 0, s>>>(static_cast<KArgs>(args)...);
    return cudaGetLastError();
#endif
}

// A replica record into shared memory, one word per thread (blockDim >= words).
__device__ __forceinline__ void load_rep_shared(Rep* dst, const Rep* src) {
    constexpr int WORDS = sizeof(Rep) / 4;
    static_assert(sizeof(Rep) % 4 == 0 && WORDS <= 256, "replica record words");
    if (threadIdx.x < WORDS)
        reinterpret_cast<uint32_t*>(dst)[threadIdx.x] = __ldg(reinterpret_cast<const uint32_t*>(src) + threadIdx.x);
}

// bird.rs:84-153 after the candidate sums: the next state at slot i of the
// write list, its bag key and the arrival count of that bag.  SLOTS: a's
// arrival slots are kept where it has them.
template <bool STRICT, bool SLOTS>
__device__ __forceinline__ void force_finish(const ForceArgs& a, const Rep& R, uint32_t i,
                                             float4 me, uint32_t my_id, unsigned long long step,
                                             const Acc<STRICT>& acc) {
    const float4 nxt = finish_bird<STRICT>(R, me, my_id, step, acc);
    const float nx = nxt.x, ny = nxt.y;
    a.out_st[i] = nxt;
    a.out_ids[i] = my_id;
    const int32_t ncx = disc(nx, R), ncy = disc(ny, R);
    int64_t idx = bag_index(R, ncx, ncy);
    uint32_t flags = 0;
    if (idx < 0) {
        flags |= ERR_KEY_RANGE;
        idx = 0;
    }
    if (!isfinite(nx) || !isfinite(ny)) flags |= ERR_NONFINITE;
    // the rebin gathers a bag's arrivals from the 3x3 old bags around it
    // (plus the seam columns/rows); anything else must take the general sort
    if (a.check_moves) {
        const int32_t ocx = disc(me.x, R), ocy = disc(me.y, R);
        if (!(move_ok(ocx, ncx, R.seam) && move_ok(ocy, ncy, R.seam)))
            flags |= ERR_REBIN_MISS | ERR_MISS_MOVE;
    }
    if (flags) atomicOr(a.err, flags);
    const uint32_t key = R.cell_off + (uint32_t)idx;
    a.out_key[i] = key;
    if (SLOTS && a.slots) {
        const uint32_t r = atomicAdd(&a.hist[key], 1u);
        if (r < RANK_ROW) a.slots[(size_t)key * RANK_ROW + r] = i;
        else if (r < RANK_SLOTS) a.slots[(size_t)a.ncells * RANK_ROW + (size_t)key * RANK_ROW2 + (r - RANK_ROW)] = i;
    } else {
        atomicAdd(&a.hist[key], 1u);
    }
}

inline unsigned grid_for(uint64_t n, unsigned block) { return (unsigned)((n + block - 1) / block); }

}  // namespace
}  // namespace kb
