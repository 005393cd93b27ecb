// The LZSS column encoder of encode.cu, whose text from LZ_WPB on up to the
// next kernel the test writes to LZSS_COLUMNS.
#include "cuda_runtime.h"

#include "gd_common.cuh"

namespace gd {
namespace encd {
thread_local __align__(16) uint8_t smem[64 << 10];
#include LZSS_COLUMNS
}  // namespace encd
}  // namespace gd

using namespace gd::encd;

// Columns [first, n_cols) of the chunk of chunk_size bytes at `in`, in steps of
// a block's; column q's stream at scratch + q * cap.
extern "C" int lzss_columns(const uint8_t* in, uint64_t chunk_size, uint32_t first, uint32_t n_cols, uint8_t* scratch,
                            uint32_t cap, uint32_t* raw_len, uint32_t kind) {
    const uint32_t wsm = lz_warp_smem((uint32_t)(chunk_size / 32));
    if (LZ_WPB * wsm > sizeof smem) return 2;
    for (uint32_t b = first / LZ_WPB; b < n_cols / LZ_WPB; ++b) {
        memset(smem, 0, sizeof smem);
        if (!simt::run(32 * LZ_WPB, b, 32 / LZ_WPB, simt::schedule(32 * LZ_WPB, kind), [&] {
                if (lz_buckets((uint32_t)(chunk_size / 32)) == LZ_NB)
                    lzss_column_kernel<LZ_NB>(in, chunk_size, chunk_size, 32, scratch, cap, raw_len, wsm);
                else
                    lzss_column_kernel<LZ_NB_SHORT>(in, chunk_size, chunk_size, 32, scratch, cap, raw_len, wsm);
            }))
            return 1;
    }
    return 0;
}
