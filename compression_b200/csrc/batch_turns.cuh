// batch_turns.cuh -- how the blocks of the batch decoder (batch.cu) take tasks.
//
// A block goes through turns: its warps decode tasks of their own, then the
// whole block decodes the Deflate tasks that they met.  What a turn's start is
// decided by (s_go) is written by warp 0 alone and by nothing that a turn does:
// a word that a warp may change inside the turn, read late by another at its
// start, lost that one's task.  A warp branches on shared words that other
// warps write only through one lane's reading of them, so that its lanes stay
// together at the warp collectives.
#pragma once
#include "gd_common.cuh"

namespace gd {
namespace batch {

// Runs the calling block's share of n tasks.  `order`: the queue (null: as
// numbered); entries out of range are passed over.  Dynamic: tasks are taken
// from the queue through `counter`, which starts at 0; else warp w of W takes
// places w, w + W, ...  The callers' functions: deflate(ti): task ti is for a
// block; warp_task(ti): decode it with the calling warp; block_task(ti): with
// the block.
template <uint32_t WPB, class Deflate, class WarpTask, class BlockTask>
__device__ __forceinline__ void run_turns(uint32_t n, const uint32_t* __restrict__ order, uint32_t* counter,
                                          bool dynamic, Deflate deflate, WarpTask warp_task, BlockTask block_task) {
    __shared__ uint32_t s_list[WPB], s_nd;  // Deflate tasks taken
    __shared__ uint32_t s_go, s_stop, s_soon, s_end;
    constexpr uint32_t NONE = 0xffffffffu, BAD = 0xfffffffeu;
    const uint32_t lane = lane_id(), wid = threadIdx.x >> 5, W = gridDim.x * WPB;
    // task of queue place j: NONE past the end, BAD for an entry out of range
    auto entry = [&](uint32_t j) -> uint32_t {
        if (j >= n) return NONE;
        const uint32_t ti = order ? order[j] : j;
        return ti < n ? ti : BAD;
    };
    // the next task of the queue, for the calling warp; soon: a Deflate task
    // lies in the part of the queue that the blocks will take next
    auto pop = [&](bool& defl, bool& soon) -> uint32_t {
        for (;;) {
            uint32_t i = 0;
            if (lane == 0) i = atomicAdd(counter, 1u);
            i = __shfl_sync(GD_FULL_MASK, i, 0);
            const uint32_t t = entry(i + lane * (W / 16u));
            const uint32_t m = __ballot_sync(GD_FULL_MASK, t < n && deflate(t));
            const uint32_t ti = __shfl_sync(GD_FULL_MASK, t, 0);
            defl = m & 1u;
            soon = (m >> 1) != 0;
            if (ti != BAD) return ti;
        }
    };
    uint32_t at = blockIdx.x * WPB + wid;  // the static mapping's next place
    for (bool begin = true;; begin = false) {
        uint32_t first = NONE;  // warp 0: a task in hand
        if (wid == 0) {
            bool defl = false, soon = false, end = false;
            if (dynamic && (begin || __shfl_sync(GD_FULL_MASK, s_soon, 0))) {
                first = pop(defl, soon);
                end = first == NONE;
            }
            if (lane == 0) {
                s_list[0] = first;
                s_nd = defl;
                s_go = !defl && !end;
                s_stop = 0;
                s_soon = soon;
                s_end = end;
            }
        }
        __syncthreads();
        if (s_go) {
            for (;;) {
                bool defl = false, soon = false;
                uint32_t ti = first;
                first = NONE;
                if (ti == NONE) {
                    uint32_t stop = 0;
                    if (lane == 0) stop = *(volatile uint32_t*)&s_stop;
                    if (__shfl_sync(GD_FULL_MASK, stop, 0)) break;
                    if (dynamic) {
                        ti = pop(defl, soon);
                    } else {
                        do {
                            ti = entry(at);
                            at += W;
                        } while (ti == BAD);
                        defl = ti != NONE && deflate(ti);
                    }
                }
                if (ti != NONE && !defl) warp_task(ti);
                const bool leave = ti == NONE || defl || soon;
                if (lane == 0) {
                    if (ti == NONE && dynamic) s_end = 1;
                    if (soon) s_soon = 1;
                    if (defl) s_list[atomicAdd(&s_nd, 1u)] = ti;
                    // statically, a warp at its end leaves the others going
                    if (leave && (dynamic || defl)) *(volatile uint32_t*)&s_stop = 1;
                }
                if (leave) break;
                __syncwarp();
            }
        }
        __syncthreads();
        const uint32_t nd = s_nd, end = dynamic ? s_end : nd == 0;
        for (uint32_t w = 0; w < nd; ++w) block_task(s_list[w]);
        if (end) break;
        __syncthreads();  // the shared words are set for the next turn
    }
}

}  // namespace batch
}  // namespace gd
