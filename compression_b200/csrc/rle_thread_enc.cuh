// rle_thread_enc.cuh -- RLE v1 / RLE v2 lane-stream encoders with a thread per
// lane stream and a warp per chunk (sm_100a).
//
// Each thread gathers its lane's values straight from the column (RLE v1:
// COMP_COL_LEN-byte slices at a 32-slice stride; RLE v2: READ_UNIT-value slices)
// and runs the serial writer of lane_enc.h into its own scratch slot, buffering
// 4 bytes in a register so that the scratch is written in whole words (the
// literal-count byte written back later is a byte store or a register edit).
// A lane stream takes as long as its values are many, whatever they hold, and a
// chip full of them costs 2.5 warp instructions where a warp per lane stream
// (rlev1_enc.cuh, rlev2_enc.cuh) pays for every token.  So this one is for short
// lane streams and for large columns of short runs.
#pragma once
#include "gd_common.cuh"
#include "lane_enc.h"

namespace gd {
namespace encd {

constexpr int THREAD_NT = 128;  // threads per block: 4 chunks

// Byte sink over one lane's scratch slot (cap bytes, a multiple of 4).
struct DevSink {
    uint32_t* w;
    uint32_t n, cap, cur;  // bytes put; capacity; bytes [n & ~3, n) not yet stored
    __device__ __forceinline__ void put(uint8_t b) {
        cur |= (uint32_t)b << (8u * (n & 3u));
        ++n;
        if ((n & 3u) == 0) {
            if (n <= cap) w[(n >> 2) - 1] = cur;
            cur = 0;
        }
    }
    __device__ __forceinline__ uint32_t size() const { return n; }
    __device__ __forceinline__ void set(uint64_t i, uint8_t b) {
        if (i >= (n & ~3u)) {
            const uint32_t sh = 8u * ((uint32_t)i & 3u);
            cur = (cur & ~(0xffu << sh)) | ((uint32_t)b << sh);
        } else if (i < cap) {
            reinterpret_cast<uint8_t*>(w)[i] = b;
        }
    }
    // store the last partial word (its unused bytes are zero)
    __device__ __forceinline__ void flush() {
        if ((n & 3u) && n < cap) w[n >> 2] = cur;
    }
};

// Value i of lane t is chunk element (i / unit) * 32 * unit + t * unit + i % unit
// (encoder.h:139-153, encoder_trans.h:40-108); elements past the input are zero.
template <typename T>
struct LaneVals {
    const T* base;
    uint64_t avail;
    uint32_t t, unit;
    __device__ __forceinline__ T operator[](uint64_t i) const {
        const uint32_t q = (uint32_t)i / unit, r = (uint32_t)i - q * unit;
        const uint64_t at = (uint64_t)q * 32u * unit + (uint64_t)t * unit + r;
        return at < avail ? base[at] : (T)0;
    }
};

// One block: *runs = whether SAMPLE windows of 32 values, spread over the
// column's n_values (at least 32 * SAMPLE), hold min_ends ends of runs (three
// values or more of one difference, RLE v1, or equal, RLE v2).
constexpr uint32_t SAMPLE = 512;
template <int CODEC, typename T>
__global__ void __launch_bounds__(1024) sample_runs_kernel(const T* __restrict__ in, uint64_t n_values,
                                                           uint32_t min_ends, uint64_t* __restrict__ runs) {
    constexpr uint32_t PER = SAMPLE / 32u;  // windows a warp
    __shared__ uint32_t s_sum;
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    const uint32_t lane = lane_id();
    T v[PER];
#pragma unroll
    for (uint32_t i = 0; i < PER; ++i)
        v[i] = __ldg(in + n_values / SAMPLE * ((threadIdx.x >> 5) * PER + i) + lane);
    uint32_t ends = 0;
#pragma unroll
    for (uint32_t i = 0; i < PER; ++i) {
        const T b = __shfl_down_sync(GD_FULL_MASK, v[i], 1), c = __shfl_down_sync(GD_FULL_MASK, v[i], 2);
        const bool run = CODEC == GD_CODEC_RLEV1 ? (T)(c - b) == (T)(b - v[i]) : c == b && b == v[i];
        const uint32_t in_run = __ballot_sync(GD_FULL_MASK, lane < 30u && run);
        ends += __popc(in_run & ~(in_run >> 1) & 0x1fffffffu);
    }
    if (lane == 0) atomicAdd(&s_sum, ends);
    __syncthreads();
    if (threadIdx.x == 0) *runs = s_sum >= min_ends;
}

// CODEC: GD_CODEC_RLEV1 (T = uint32_t / uint64_t, unit = values per slice) or
// GD_CODEC_RLEV2 (T = int64_t, unit = read unit).  take null: the chunks' block
// sizes and status are written too.  Else nothing is done if it points at 0, and
// col_len is as the warp encoders' (all ones if a stream outgrew its slot), for
// lane_sizes_kernel.
template <int CODEC, typename T>
__global__ void __launch_bounds__(THREAD_NT) thread_encode_kernel(const uint8_t* __restrict__ in, uint64_t n_bytes,
                                                                  uint32_t n_chunks, uint64_t chunk_size, uint32_t unit,
                                                                  uint8_t* __restrict__ scratch, uint32_t lane_cap,
                                                                  uint64_t* __restrict__ col_len,
                                                                  const uint64_t* __restrict__ take,
                                                                  uint64_t* __restrict__ blk_size,
                                                                  uint32_t* __restrict__ status) {
    const uint32_t c = (blockIdx.x * THREAD_NT + threadIdx.x) >> 5, t = lane_id();
    if (c >= n_chunks || (take && !*take)) return;
    const uint64_t cb = (uint64_t)c * chunk_size;
    const uint64_t have = n_bytes > cb ? (n_bytes - cb < chunk_size ? n_bytes - cb : chunk_size) : 0;
    const LaneVals<T> v{reinterpret_cast<const T*>(in + cb), have / sizeof(T), t, unit};
    DevSink s{reinterpret_cast<uint32_t*>(scratch + ((uint64_t)c * 32u + t) * lane_cap), 0u, lane_cap, 0u};
    if constexpr (CODEC == GD_CODEC_RLEV1)
        enc::rlev1_encode_lane<T>(v, chunk_size / 32u / sizeof(T), s);
    else
        enc::rlev2_encode_lane(v, chunk_size / 256u, s);
    s.flush();
    const bool over = s.n > lane_cap;
    const uint32_t len = over ? 0u : s.n;
    col_len[(uint64_t)c * 32u + t] = over && take ? ~0ull : len;
    if (take) return;
    const uint32_t words = __reduce_add_sync(GD_FULL_MASK, (len + 3u) >> 2);
    const bool bad = __any_sync(GD_FULL_MASK, over);
    if (t == 0) {
        blk_size[c] = ((uint64_t)words * 4u + 127u) & ~127ull;
        put_status(status, c, bad ? (uint32_t)ST_OVERRUN : (uint32_t)ST_OK);
    }
}

// Who encodes a column: threads (all), warps (neither), or threads if it has
// `ends` sampled run ends, else warps.
struct ThreadRule {
    bool all;
    uint32_t ends;
};

}  // namespace encd
}  // namespace gd
