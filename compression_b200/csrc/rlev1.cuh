// rlev1.cuh -- RLE v1 (ORC-style integer RLE v1) decoder for sm_100a.
//
// Grammar (restated from decoder_warp, include/rle_v1/decoder.h:278-423):
// int8 header h; h < 0: -h literal values, each an unsigned LEB128 varint;
// h >= 0: a run of h+3 values, int8 delta then varint base, v_i = base+i*delta.
// Lane t of a chunk owns elements (i / wil)*32*wil + t*wil + i % wil,
// wil = COMP_COL_LEN / sizeof(T); a lane stream ends once it has produced
// chunk_size/32 bytes (decoder.h:283,291).
//
// The reference pairs a reader warp and a decoder warp per chunk (spin
// queues, one byte fetched per funnel-shift call, one scalar store per
// value).  Here every lane stream gets a whole warp (same block loader as
// RLE v2: 8 adjacent lane streams per block, copied with fully used 32-byte
// row sectors):
//   * runs are closed form: lane i writes base + i*delta;
//   * a header, a run's delta and a base of up to 4 bytes come from two
//     funnel-shifted words (a longer base's other bytes one by one), a base of
//     1 or 2 bytes from the first word alone: the steps from one run to the next
//     are a chain (64 MiB of runs of 8: bases of 1 byte 0.162 ms, 2 0.172, 5
//     0.212; with one path for up to 4 bytes and a longer base read again from
//     its start 0.213, 0.215, 0.295);
//   * a literal group is decoded 32 values at a time: the lanes load a
//     128-byte window and ballot the varint terminators (bytes < 0x80); the
//     lane at the j-th terminator stores its place for lane j (a select of the
//     j-th set bit of the ballots by every lane took most of the step), so
//     every lane knows where its varint starts and ends and decodes it alone
//     (the first 4 bytes by one funnel-shifted word, compacted with masks).
#pragma once
#include "interleave.cuh"

namespace gd {
namespace rlev1 {


// Largest lane stream for nv values: literal varints of up to 10 bytes plus
// one header per 127 values; +128 tail for terminator windows.
__host__ __device__ constexpr uint32_t stream_cap(uint32_t nv, uint32_t eb) {
    return (((eb == 8 ? 10u : 5u) * nv + nv / 127u + 64u + 15u) & ~15u) + 144u;
}

// Shared-memory bytes reserved for a lane stream of at most `n` bytes.
__host__ __device__ constexpr uint32_t lane_cap(uint32_t n) { return ((n + 15u) & ~15u) + 144u; }

// The 7-bit groups of 4 varint bytes.
__device__ __forceinline__ uint32_t low28(uint32_t v) {
    return (v & 0x7fu) | ((v >> 1) & 0x3f80u) | ((v >> 2) & 0x1fc000u) | ((v >> 3) & 0xfe00000u);
}

// Decode one lane stream (sbuf[0..len), readable 144 bytes past len) of nv
// elements of type T with the calling warp.  Lane stream t with wil = values
// per lane slice: element e goes to outv[(e/wil)*32*wil + t*wil + e%wil] if
// that index is below want.  Returns a gd status (same on every lane).
template <typename T>
static __device__ __noinline__ uint32_t lane_warp(const uint8_t* __restrict__ sbuf, uint32_t len, uint32_t nv, uint32_t t,
                                           uint32_t wil, T* __restrict__ outv, uint64_t want) {
    __shared__ uint8_t s_ends[8][32];  // blocks have at most 8 warps
    const uint32_t lane = lane_id();
    uint8_t* ends = s_ends[threadIdx.x >> 5];
    // wil a power of two (COMP_COL_LEN / sizeof(T) always is in the
    // reference's configurations): shifts instead of a division per value
    const bool pow2 = (wil & (wil - 1u)) == 0u;
    const uint32_t wsh = __ffs(wil) - 1u;
    // a chunk holds at most 2^31 bytes, so element indices fit in 32 bits
    const uint32_t want32 = want < 0xffffffffull ? (uint32_t)want : 0xffffffffu;
    const uint32_t tw = t << wsh;
    auto put = [&](uint32_t e, T v) {
        const uint32_t oe = pow2 ? ((e >> wsh) << (wsh + 5u)) + tw + (e & (wil - 1u))
                                 : (e / wil) * 32u * wil + t * wil + (e % wil);
        if (oe < want32) outv[oe] = v;
    };
    uint32_t err = ST_OK, pos = 0, g = 0;
    while (g < nv) {
        // ---- header: every lane parses it (shared-memory broadcast reads),
        // so nothing needs to be shuffled ----
        uint32_t kind = 0, cnt = 0, next = 0, e = ST_OK;
        T base = 0, delta = 0;
        if (pos >= len) {
            e = ST_CORRUPT;
        } else {
            const uint32_t* w = reinterpret_cast<const uint32_t*>(sbuf + (pos & ~3u));
            const uint32_t w1 = w[1], sh8 = 8u * (pos & 3u);
            const uint32_t lo = __funnelshift_r(w[0], w1, sh8);  // the next 4 bytes
            const uint32_t h = lo & 0xffu;
            if (h & 0x80u) {
                kind = 1;
                cnt = 256u - h;
                next = pos + 1;
            } else {
                cnt = h + 3u;
                delta = (T)(int64_t)(int8_t)(lo >> 8);
                const uint32_t v = __funnelshift_r(lo, __funnelshift_r(w1, w[2], sh8), 16);  // the base's first 4
                const uint32_t term = ~v & 0x80808080u;
                // short bases first: a column of runs is a chain of these steps
                if (!(lo & 0x800000u)) {
                    base = (T)(lo >> 16 & 0x7fu);
                    next = pos + 3;
                    if (next > len) e = ST_CORRUPT;
                } else if (!(lo & 0x80000000u)) {
                    base = (T)((lo >> 16 & 0x7fu) | (lo >> 17 & 0x3f80u));
                    next = pos + 4;
                    if (next > len) e = ST_CORRUPT;
                } else if (term) {
                    const bool three = !(v & 0x800000u);  // bytes, or 4
                    base = (T)low28(three ? v & 0xffffffu : v);
                    next = pos + (three ? 5u : 6u);
                    if (next > len) e = ST_CORRUPT;
                } else {
                    uint32_t p = pos + 6, sh = 28, b;
                    uint64_t x = low28(v);
                    do {
                        if (p >= len || sh > 63) {
                            e = ST_CORRUPT;
                            break;
                        }
                        b = sbuf[p++];
                        x |= (uint64_t)(b & 0x7fu) << sh;
                        sh += 7;
                    } while (b & 0x80u);
                    base = (T)x;
                    next = p;
                }
            }
        }
        if (e != ST_OK) {
            err = e;
            break;
        }
        if (g + cnt > nv) {
            err = ST_OVERRUN;
            break;
        }
        if (kind == 0) {  // run: closed form (in T's width: the low bits of base + i*delta)
            for (uint32_t i = lane; i < cnt; i += 32) put(g + i, base + (T)i * delta);
            g += cnt;
            pos = next;
            continue;
        }
        // literal group: cnt varints starting at `next`
        uint32_t p = next, rem = cnt;
        while (rem) {
            uint32_t m[4], nterm = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t bpos = p + 32u * q + lane;
                const bool term = (bpos < len) && !(sbuf[bpos] & 0x80u);
                m[q] = __ballot_sync(GD_FULL_MASK, term);
                const uint32_t rank = nterm + __popc(m[q] & ((1u << lane) - 1u));
                if (term && rank < 32u) ends[rank] = (uint8_t)(32u * q + lane);
                nterm += __popc(m[q]);
            }
            if (nterm == 0) {  // no varint ends within 128 bytes (or the stream ran out)
                err = ST_CORRUPT;
                break;
            }
            const uint32_t take = min(min(rem, nterm), 32u);
            __syncwarp();
            const uint32_t end = lane < take ? ends[lane] : 0u;
            const uint32_t prev = __shfl_up_sync(GD_FULL_MASK, end, 1);  // the previous varint's last byte
            if (lane < take) {
                const uint32_t beg = lane ? prev + 1 : 0;
                const uint32_t a = p + beg, n = end - beg + 1;
                const uint32_t* wp = reinterpret_cast<const uint32_t*>(sbuf + (a & ~3u));
                uint32_t lo = __funnelshift_r(wp[0], wp[1], 8u * (a & 3u));
                if (n < 4) lo &= (1u << (8u * n)) - 1u;
                T v = (T)low28(lo);
                if constexpr (sizeof(T) == 4) {
                    // a 32-bit value takes the varint's first 5 bytes
                    if (n >= 5) v |= (T)sbuf[a + 4] << 28;
                } else {
                    for (uint32_t k = 4; k < n && k < 10; ++k) v |= (T)(sbuf[a + k] & 0x7fu) << (7u * k);
                }
                put(g + lane, v);
            }
            p += __shfl_sync(GD_FULL_MASK, end, take - 1) + 1;
            g += take;
            rem -= take;
        }
        if (err != ST_OK) break;
        pos = p;
    }
    return err;
}

}  // namespace rlev1
}  // namespace gd
