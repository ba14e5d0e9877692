// wf_launch.cuh -- grid of the persistent wavefront kernels.
#pragma once

#include <algorithm>
#include <cstdint>

#include <cuda_runtime.h>

#include "wf_fields.cuh"
#include "wf_kernels.h"

// Threads per block of a wavefront launch: 4 warps, which the kernels are bounded to, or fewer by the tuning
// (which accepts up to 32; more than 4 give 4).
inline int wave_threads(const WfLaunchCfg& c) { return 32 * (c.walk_warps > 0 ? std::min(c.walk_warps, 4) : 4); }

// Blocks of a persistent wavefront launch and the number of work items dispatched first.
//
// The grid is every block that fits on the device at once (occupancy), capped by the work.
// The longest chains (the plan's trailing long chunks) carry the critical path, so up to half
// of the resident warps take them first; the remaining warps take the other chunks in the plan's
// order. Progress is guaranteed: a chunk only waits for chains before it in that order, which are
// either long chunks already resident or ordinary chunks, which at least half of the resident
// warps keep dispatching in dependency order; and the chains of a chunk, which may share a warp,
// end before another one of the chunk needs their discharge (wf_plan.cpp).
template <class Kernel>
cudaError_t wave_grid(Kernel kernel, int threads, size_t smem, const WfLaunchCfg& c, const WfDevGraph& g, int& blocks,
                      int64_t& prio_items, int64_t items_per_chunk = 0) {
    int per_sm = 0;
    const cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    if (err != cudaSuccess) return err;
    if (per_sm < 1) per_sm = 1;
    blocks = c.walk_blocks > 0 ? c.walk_blocks : c.num_sms * per_sm;
    const int wpb = threads / 32;
    const int64_t ipc = items_per_chunk > 0 ? items_per_chunk : (g.M > 32 ? g.M / 32 : 1);
    const int64_t items = g.n_chunks * ipc;
    const int64_t need = (items + wpb - 1) / wpb;
    if (blocks > need) blocks = (int)(need < 1 ? 1 : need);
    const int64_t resident = (int64_t)std::min(blocks, c.num_sms * per_sm) * wpb;
    prio_items = std::min<int64_t>(g.n_long_chunks * ipc, resident / 2);
    return cudaSuccess;
}

// Chunks of the first-dispatched group that a slim wavefront (wf_wave.cuh) takes first with SL lanes per
// pair: as many as half of the resident warps hold.
inline int64_t first_chunks(const WfDevGraph& g, int SL, int64_t resident) {
    return std::min<int64_t>(g.n_long_chunks, resident / 2 / wf_items_per_chunk(1, g.M, SL));
}

// Lanes per chain-member pair of that group: the most (fewest pairs to a warp, whose members wait for one
// another) that still give each of its warps a scheduler. Eight members of 128 x 128 cells, hourly FP64 river
// sweep: 3.3 ms with all members in a warp, 2.2 by this rule.
inline int first_lanes(const WfDevGraph& g, const WfLaunchCfg& c) {
    int SL = 32;
    while (SL > 1 && g.n_long_chunks * wf_items_per_chunk(1, g.M, SL) > c.num_sms * 4) SL >>= 1;
    return SL;
}

// Sub-step lanes of a diagonal-schedule launch of S sub-steps: the smallest power of two that
// covers S, at most the cap (tuning; 8 by default) and at most 32.
inline int wave_sub_lanes(int S, const WfLaunchCfg& c) {
    const int cap = c.sub_lanes > 0 ? std::min(c.sub_lanes, 32) : 8;
    int sl = 1;
    while (sl < S && sl < cap) sl <<= 1;
    return sl;
}
