// rlev1_enc.cuh -- RLE v1 lane-stream encoder on a warp (sm_100a).
//
// The writer (rlev1_encode_lane in lane_enc.h, after compression_warp,
// include/rle_v1/encoder.h:607-1018) is greedy.  With d_k the difference of
// values k and k - 1 in the element type, taken as an int64, a position i with
// -128 <= d_{i+1} <= 127 and d_{i+2} == d_{i+1} starts a run: as many values
// as keep that difference, 129 at most.  Any other value is a literal; literals
// up to the next run make groups of 127 at most.  So a warp takes a lane stream
// token by token: the next run's place and length from two bit masks over the
// values, a literal group's bytes from a prefix sum of its varints' lengths,
// 32 values at a time; runs one after the other are taken together, a lane each
// (64 MiB of runs of 8: 0.23 ms, one by one 0.49).  A thread per lane stream, a
// value at a time, took 0.63 ms for 64 MiB of the benchmark's column.
#pragma once
#include "gd_common.cuh"

namespace gd {
namespace encd {

constexpr uint32_t V1_WPB = 4;      // lane streams (warps) per block
constexpr uint32_t V1_FLUSH = 512;  // bytes of output held back at most before a token (which adds 1.3 KB at most)

template <typename T>
struct V1Warp {
    T ring[256];       // values by index mod 256
    uint32_t eq[8];    // bit k mod 256: d_k == d_{k-1}
    uint32_t small[8]; // bit k mod 256: -128 <= d_k <= 127
    alignas(4) uint8_t out[2048];
};

template <typename T>
__device__ __forceinline__ uint32_t v1_varint_len(T v) {
    const uint32_t bits = 64u - (uint32_t)__clzll((long long)(uint64_t)v);
    return bits ? (bits + 6u) / 7u : 1u;
}
template <typename T>
__device__ __forceinline__ void v1_put_varint(T v, uint32_t nb, uint8_t* out) {
#pragma unroll
    for (uint32_t b = 0; b < (sizeof(T) == 4 ? 5u : 10u); ++b)
        if (b < nb) out[b] = (uint8_t)((uint32_t)(v >> (7u * b)) & 0x7fu) | (b + 1u < nb ? 0x80u : 0u);
}

// A warp per lane stream; col_len gets the stream's bytes, all ones if they
// outgrew the slot (lane_sizes_kernel turns that into a status).  skip (or
// null): nothing to do if it is not 0.
template <typename T>
__global__ void __launch_bounds__(V1_WPB * 32) rlev1_encode_kernel(const uint8_t* __restrict__ in, uint64_t n_bytes,
                                                                   uint64_t n_lanes, uint64_t chunk_size, uint32_t wil,
                                                                   uint8_t* __restrict__ scratch, uint32_t lane_cap,
                                                                   uint64_t* __restrict__ col_len,
                                                                   const uint64_t* __restrict__ skip) {
    __shared__ V1Warp<T> smem[V1_WPB];
    const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
    const uint64_t id = (uint64_t)blockIdx.x * V1_WPB + wid;  // 32 * chunk + lane stream
    if (id >= n_lanes || (skip && *skip)) return;      // warp-uniform
    V1Warp<T>& S = smem[wid];
    const uint64_t cb = (id >> 5) * chunk_size;
    const uint64_t avail =
        (n_bytes > cb ? min((unsigned long long)(n_bytes - cb), (unsigned long long)chunk_size) : 0ull) / sizeof(T);
    const T* base = reinterpret_cast<const T*>(in + cb);
    const uint32_t n = (uint32_t)(chunk_size / 32u / sizeof(T)), t = (uint32_t)id & 31u;
    uint32_t* slot = reinterpret_cast<uint32_t*>(scratch + id * lane_cap);
    // value k of the lane is chunk element (k / wil) * 32 * wil + t * wil + k %
    // wil (encoder.h:139-153); elements past the input are zero
    auto fetch = [&](uint32_t k) -> T {
        if (k >= n) return (T)0;
        const uint32_t q = k / wil;
        const uint64_t at = (uint64_t)q * 32u * wil + (uint64_t)t * wil + (k - q * wil);
        return at < avail ? __ldg(base + at) : (T)0;
    };
    uint32_t loaded = 0;      // a multiple of 32, or n rounded up to one
    T ahead = fetch(lane);    // values loaded .. loaded + 31, on their way
    T last = 0, dlast = 0;    // value and difference loaded - 1
    uint32_t on = 0;          // bytes in S.out
    uint32_t written = 0;     // words in the slot
    bool over = false;
    for (uint32_t i = 0; i < n;) {
        while (loaded < n && loaded < i + 129u) {
            const T v = ahead;
            ahead = fetch(loaded + 32u + lane);
            S.ring[(loaded + lane) & 255u] = v;
            const T up = __shfl_up_sync(GD_FULL_MASK, v, 1);
            const T d = v - (lane ? up : last);
            const T dup = __shfl_up_sync(GD_FULL_MASK, d, 1);
            const int64_t sd = (int64_t)d;  // 32-bit differences are taken unsigned, as the writer takes them
            const uint32_t eq = __ballot_sync(GD_FULL_MASK, d == (lane ? dup : dlast));
            const uint32_t sm = __ballot_sync(GD_FULL_MASK, sd >= -128 && sd <= 127);
            if (lane == 0) {
                S.eq[(loaded >> 5) & 7u] = eq;
                S.small[(loaded >> 5) & 7u] = sm;
            }
            last = __shfl_sync(GD_FULL_MASK, v, 31);
            dlast = __shfl_sync(GD_FULL_MASK, d, 31);
            loaded += 32;
        }
        __syncwarp();
        // bit k of E: values i + k .. i + k + 2 have one difference; of the lane's values only
        uint32_t r = 127;  // literals before the next run
        const uint32_t valid = n - i > 2u ? n - i - 2u : 0u;
        uint32_t E[4], P[4];
        {
            uint32_t e0 = S.eq[((i + 2u) >> 5) & 7u], s0 = S.small[((i + 1u) >> 5) & 7u];
#pragma unroll
            for (uint32_t w = 0; w < 4; ++w) {
                const uint32_t e1 = S.eq[(((i + 2u) >> 5) + w + 1u) & 7u];
                const uint32_t s1 = S.small[(((i + 1u) >> 5) + w + 1u) & 7u];
                E[w] = __funnelshift_r(e0, e1, i + 2u);
                if (valid < 32u * w + 32u) E[w] &= valid > 32u * w ? (1u << (valid - 32u * w)) - 1u : 0u;
                P[w] = E[w] & __funnelshift_r(s0, s1, i + 1u);
                e0 = e1;
                s0 = s1;
            }
#pragma unroll
            for (int w = 3; w >= 0; --w)
                if (P[w]) r = min(32u * w + __ffs(P[w]) - 1u, 127u);
        }
        uint8_t* out = S.out + on;
        uint32_t z = 127;  // equal differences from i on
        if (r == 0) {
#pragma unroll
            for (int w = 3; w >= 0; --w)
                if (~E[w]) z = min(32u * w + __ffs(~E[w]) - 1u, 127u);
        }
        if (r == 0 && z < 30u && (P[0] >> (z + 2u) & 1u)) {
            // runs one after the other, as many as the masks show the ends
            // of (their bit 126 is the last that is known): a lane each
            const uint64_t e0 = (uint64_t)E[1] << 32 | E[0], e1 = (uint64_t)E[3] << 32 | E[2];
            const uint64_t p0 = (uint64_t)P[1] << 32 | P[0], p1 = (uint64_t)P[3] << 32 | P[2];
            uint32_t at = 0, k = 0, start = 0, L = 0;
            while (k < 32u && at < 126u && ((at < 64u ? p0 >> at : p1 >> (at - 64u)) & 1u)) {
                const uint64_t x = at == 0u ? e0 : at < 64u ? e0 >> at | e1 << (64u - at) : e1 >> (at - 64u);
                const uint32_t ones = (uint32_t)__ffsll((long long)~x) - 1u;  // all ones: none
                if (ones >= 64u || at + ones > 126u) break;
                if (lane == k) {
                    start = at;
                    L = 2u + ones;
                }
                at += 2u + ones;
                ++k;
            }
            const T v = S.ring[(i + start) & 255u], d = S.ring[(i + start + 1u) & 255u] - v;
            const uint32_t nb = v1_varint_len(v), size = lane < k ? 2u + nb : 0u, inc = warp_incl_scan(size);
            if (lane < k) {
                uint8_t* o = out + inc - size;
                o[0] = (uint8_t)(L - 3u);
                o[1] = (uint8_t)d;
                v1_put_varint(v, nb, o + 2);
            }
            on += __shfl_sync(GD_FULL_MASK, inc, 31);
            i += at;
        } else if (r == 0) {
            const uint32_t L = 2u + z;
            const T v = S.ring[i & 255u], d = S.ring[(i + 1u) & 255u] - v;
            const uint32_t nb = v1_varint_len(v);
            if (lane == 0) {
                out[0] = (uint8_t)(L - 3u);
                out[1] = (uint8_t)d;
            }
            if (lane < nb) out[2 + lane] = (uint8_t)(((uint32_t)(v >> (7u * lane)) & 0x7fu) | (lane + 1u < nb ? 0x80u : 0u));
            on += 2u + nb;
            i += L;
        } else {
            const uint32_t m = min(r, n - i);
            if (lane == 0) out[0] = (uint8_t)(0u - m);
            uint32_t at = 1;
            for (uint32_t k = 0; k < m; k += 32) {
                const T v = S.ring[(i + k + lane) & 255u];
                const uint32_t nb = k + lane < m ? v1_varint_len(v) : 0u;
                const uint32_t inc = warp_incl_scan(nb);
                v1_put_varint(v, nb, out + at + inc - nb);
                at += __shfl_sync(GD_FULL_MASK, inc, 31);
            }
            on += at;
            i += m;
        }
        __syncwarp();
        if (on >= V1_FLUSH || i >= n) {
            // whole words to the slot; at the end also the last, its unused bytes zero
            if (i >= n && (on & 3u) && (on & 3u) + lane < 4u) S.out[on + lane] = 0;
            __syncwarp();
            const uint32_t nw = i >= n ? (on + 3u) >> 2 : on >> 2;
            over = over || 4ull * (written + nw) > lane_cap;
            if (!over)
                for (uint32_t w = lane; w < nw; w += 32)
                    slot[written + w] = reinterpret_cast<const uint32_t*>(S.out)[w];
            if (i >= n) {
                if (lane == 0) col_len[id] = over ? ~0ull : 4ull * written + on;
                break;
            }
            written += nw;
            on &= 3u;
            uint8_t keep = 0;
            if (lane < on) keep = S.out[4u * nw + lane];
            __syncwarp();
            if (lane < on) S.out[lane] = keep;
            __syncwarp();
        }
    }
}

}  // namespace encd
}  // namespace gd
