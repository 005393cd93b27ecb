// The turns of the batch decoder's blocks (batch_turns.cuh), with tasks that
// only count the threads that run them.
#include "cuda_runtime.h"

#include "batch_turns.cuh"

template <uint32_t WPB>
static bool go(uint32_t n, const uint8_t* deflate, const uint32_t* order, bool dynamic, uint32_t grid, uint32_t kind,
               uint32_t* warp_runs, uint32_t* block_runs) {
    uint32_t counter = 0;
    for (uint32_t b = 0; b < grid; ++b)
        if (!simt::run(32 * WPB, b, grid, simt::schedule(32 * WPB, kind), [&] {
                gd::batch::run_turns<WPB>(
                    n, order, &counter, dynamic, [&](uint32_t t) { return deflate[t] != 0; },
                    [&](uint32_t t) {
                        ++warp_runs[t];
                        __syncwarp();
                    },
                    [&](uint32_t t) {
                        ++block_runs[t];
                        __syncthreads();
                    });
            }))
            return false;
    return true;
}

// 0: the kernel ended; runs[t]: threads that ran task t as a warp's / a block's
extern "C" int turns(uint32_t wpb, uint32_t n, const uint8_t* deflate, const uint32_t* order, int dynamic, uint32_t grid,
                     uint32_t kind, uint32_t* warp_runs, uint32_t* block_runs) {
    const bool ok = wpb == 8 ? go<8>(n, deflate, order, dynamic, grid, kind, warp_runs, block_runs)
                             : go<4>(n, deflate, order, dynamic, grid, kind, warp_runs, block_runs);
    return ok ? 0 : 1;
}
