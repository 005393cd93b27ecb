// rlev2_enc.cuh -- RLE v2 lane-stream encoder on a warp (sm_100a).
//
// The writer's state machine (rlev2_encode_lane in lane_enc.h, after
// include/rlev2/encoder.h:538-969) cuts a lane's values into runs and writes
// each run from its values alone, except for one leftover: a run of more than
// 10 equal values is written with the first delta of the last run that was not
// written as a delta run (`stale` below).  So a warp takes a lane stream run by
// run: the run's end from a bit mask of equal neighbours, its encoding from
// warp reductions over at most 128 values (four a lane), its bytes one a lane.
// Short runs of equal values one after the other are taken together, a lane each
// (64 MiB: the benchmark's column 0.298 -> 0.278 ms, runs of 8 0.28 -> 0.15).
// A thread per lane stream, each with 6 KB of run buffers in local memory and
// branching on its own run, took 5.5 ms for 64 MiB of the benchmark's column.
//
// Where a run ends, starting at value i (num_literals == 0):
//   e = values equal to the first, 128 at most.  e >= 3: they are the run.
//   Otherwise it ends before the first three equal neighbours that lie inside
//   the 128 values from i, after 128 values, or with the lane.
#pragma once
#include "gd_common.cuh"
#include "lane_enc.h"

namespace gd {
namespace encd {

constexpr uint32_t V2_WPB = 4;       // lane streams (warps) per block
constexpr uint32_t V2_FLUSH = 512;   // bytes of output held back at most before a run (which adds 1.2 KB at most)

struct V2Warp {
    int64_t ring[256];   // values by index mod 256
    int64_t pk[128];     // deltas or reduced values to pack
    int64_t gp[128];     // gap and patch pairs to pack
    uint32_t eq[8];      // bit k mod 256: value k equals value k + 1
    uint32_t hist[32];   // values per width class
    uint8_t pos[128];    // patched positions
    alignas(4) uint8_t out[2048];
};

// Byte sink over the warp's output buffer, for the serial writer.
struct BufSink {
    uint8_t* p;
    uint32_t n;
    __device__ void put(uint8_t b) { p[n++] = b; }
};

// One run through the serial writer (lane 0), for the values whose arithmetic
// wraps there; returns the bytes written and replaces stale.
static __device__ __noinline__ uint32_t v2_serial_run(const V2Warp& S, uint32_t i, uint32_t m, uint8_t* out,
                                                      int64_t* stale) {
    BufSink o{out, 0};
    enc::V2Info<BufSink> info;
    for (uint32_t k = 0; k < 128; ++k) info.deltas[k] = 0;
    info.deltas[0] = *stale;
    for (uint32_t k = 0; k < m; ++k) info.literals[k] = S.ring[(i + k) & 255u];
    info.num_literals = info.var_runlen = m;
    info.fix_runlen = 0;
    info.delta_bits = 0;
    info.is_fixed_delta = false;
    info.out = &o;
    enc::determine_encoding(info);
    *stale = info.deltas[0];
    return o.n;
}

__device__ __forceinline__ uint32_t v2_bits(uint64_t v) { return 64u - (uint32_t)__clzll((long long)v); }

// Pack count values, value k at src[(first + k) & wrap], `width` bits each,
// first bit highest; returns the bytes (the last one filled with zeros).
__device__ __forceinline__ uint32_t v2_pack(const int64_t* src, uint32_t first, uint32_t wrap, uint32_t count,
                                            uint32_t width, uint8_t* out) {
    const uint32_t lane = lane_id();
    const uint32_t total = (count * width + 7u) >> 3;
    if ((width & 7u) == 0) {
        const uint32_t nb = width >> 3, inv = 65536u / nb + 1u;  // B / nb for B < 1024
        for (uint32_t B = lane; B < total; B += 32) {
            const uint32_t k = (B * inv) >> 16, r = B - k * nb;
            out[B] = reinterpret_cast<const uint8_t*>(src + ((first + k) & wrap))[nb - 1u - r];
        }
    } else {
        for (uint32_t B = lane; B < total; B += 32) {
            uint32_t k = 8u * B / width, off = 8u * B - k * width, need = 8, acc = 0;
            while (need && k < count) {
                const uint32_t take = min(need, width - off);
                const uint64_t v = (uint64_t)src[(first + k) & wrap] >> (width - off - take);
                need -= take;
                acc |= ((uint32_t)v & ((1u << take) - 1u)) << need;
                off = 0;
                ++k;
            }
            out[B] = (uint8_t)acc;
        }
    }
    return total;
}

// Unsigned LEB128 of u; returns its bytes.
__device__ __forceinline__ uint32_t v2_varint(uint64_t u, uint8_t* out) {
    const uint32_t lane = lane_id(), nb = u ? (v2_bits(u) + 6u) / 7u : 1u;
    if (lane < nb) out[lane] = (uint8_t)(((u >> (7u * lane)) & 0x7fu) | (lane + 1u < nb ? 0x80u : 0u));
    return nb;
}
__device__ __forceinline__ uint64_t v2_zigzag(int64_t v) { return ((uint64_t)v << 1) ^ (uint64_t)(v >> 63); }

// Width class holding the value of rank `more` from the widest (percentile_bits
// in lane_enc.h): the highest class c with more than `more` values in classes
// >= c.  cls[r]: class of this lane's r-th value, 32 = none.
__device__ __forceinline__ void v2_hist(const uint32_t (&cls)[4], V2Warp& S, uint32_t& at_least) {
    const uint32_t lane = lane_id();
    S.hist[lane] = 0;
    __syncwarp();
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
        const uint32_t peers = __match_any_sync(GD_FULL_MASK, cls[r]);
        if (cls[r] < 32u && (peers & ((1u << lane) - 1u)) == 0) S.hist[cls[r]] += __popc(peers);
        __syncwarp();
    }
    const uint32_t h = S.hist[31u - lane];                                  // classes from the widest
    at_least = __shfl_sync(GD_FULL_MASK, warp_incl_scan(h), 31 - (int)lane);  // values in classes >= lane
    __syncwarp();
}
__device__ __forceinline__ uint32_t v2_class(uint32_t at_least, uint32_t more) {
    return 31u - (uint32_t)__clz(__ballot_sync(GD_FULL_MASK, at_least > more));
}
__device__ __forceinline__ uint32_t v2_rank(uint32_t m, uint32_t p) { return (m * (100u - p) - 1u) / 100u + 1u; }

// DIRECT run: values i .. i + m of the ring, runlen as written in the header.
__device__ __forceinline__ uint32_t v2_direct(V2Warp& S, uint32_t i, uint32_t m, uint32_t bits, uint32_t vl,
                                              uint8_t* out) {
    const uint32_t nb = enc::w_closest_aligned(enc::w_closest(bits));
    if (lane_id() == 0) {
        out[0] = (uint8_t)(0x40u | ((uint32_t)enc::w_encode(nb) << 1) | ((vl & 0x100u) >> 8));
        out[1] = (uint8_t)vl;
    }
    return 2u + v2_pack(S.ring, i, 255u, m, nb, out + 2);
}

// DELTA run of one delta: base, delta.
__device__ __forceinline__ uint32_t v2_delta_fixed(int64_t base, int64_t delta, uint32_t m, uint8_t* out) {
    const uint32_t len = m - 1u;
    if (lane_id() == 0) {
        out[0] = (uint8_t)(0xC0u | ((len & 0x100u) >> 8));
        out[1] = (uint8_t)len;
    }
    const uint32_t b = v2_varint((uint64_t)base, out + 2);
    return 2u + b + v2_varint(v2_zigzag(delta), out + 2 + b);
}

// A run of m values from value i that are not all equal (or fewer than 3), by
// its values: DIRECT, DELTA or PATCHED_BASE (determine_encoding).
__device__ __forceinline__ uint32_t v2_var_run(V2Warp& S, uint32_t i, uint32_t m, int64_t& stale, uint8_t* out) {
    const uint32_t lane = lane_id();
    int64_t x[4];
    uint64_t all = 0, span = 0;
    const int64_t x0 = S.ring[i & 255u], init = (int64_t)((uint64_t)S.ring[(i + 1u) & 255u] - (uint64_t)x0);
    bool inc = true, dec = true, fixed = true;
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
        const uint32_t k = lane + 32u * r;
        x[r] = 0;
        if (k < m) {
            x[r] = S.ring[(i + k) & 255u];
            all |= (uint64_t)x[r];
            if (k) {
                const int64_t cd = (int64_t)((uint64_t)x[r] - (uint64_t)S.ring[(i + k - 1u) & 255u]);
                inc = inc && cd >= 0;
                dec = dec && cd <= 0;
                fixed = fixed && cd == init;
                const uint64_t ad = cd < 0 ? 0ull - (uint64_t)cd : (uint64_t)cd;
                span |= ad;
                S.pk[k] = (int64_t)ad;
            }
        }
    }
    all = (uint64_t)__reduce_or_sync(GD_FULL_MASK, (uint32_t)(all >> 32)) << 32 |
          __reduce_or_sync(GD_FULL_MASK, (uint32_t)all);
    const uint32_t bits = v2_bits(all);  // of the widest value; a negative one has 64
    __syncwarp();
    if (m <= 3) return v2_direct(S, i, m, bits, m - 1u, out);
    int64_t lmin = 0;
    if ((int64_t)all < 0) {
        // some values are negative: the writer takes DIRECT unless the
        // range wraps (safe_subtract)
        int64_t lo = x0, hi = x0;
#pragma unroll
        for (uint32_t r = 0; r < 4; ++r)
            if (lane + 32u * r < m) {
                lo = x[r] < lo ? x[r] : lo;
                hi = x[r] > hi ? x[r] : hi;
            }
#pragma unroll
        for (int s = 16; s; s >>= 1) {
            const int64_t l2 = __shfl_xor_sync(GD_FULL_MASK, lo, s), h2 = __shfl_xor_sync(GD_FULL_MASK, hi, s);
            lo = l2 < lo ? l2 : lo;
            hi = h2 > hi ? h2 : hi;
        }
        if (!enc::safe_subtract(hi, lo)) {
            stale = init;
            return v2_direct(S, i, m, 64, m - 1u, out);
        }
        uint32_t nb = 0;
        if (lane == 0) nb = v2_serial_run(S, i, m, out, &stale);
        stale = __shfl_sync(GD_FULL_MASK, stale, 0);
        return __shfl_sync(GD_FULL_MASK, nb, 0);
    }
    // no value is negative from here on: no difference wraps
    if (__all_sync(GD_FULL_MASK, fixed)) {
        stale = 0;
        return v2_delta_fixed(x0, init, m, out);
    }
    if (init != 0 && (__all_sync(GD_FULL_MASK, inc) || __all_sync(GD_FULL_MASK, dec))) {
        span = (uint64_t)__reduce_or_sync(GD_FULL_MASK, (uint32_t)(span >> 32)) << 32 |
               __reduce_or_sync(GD_FULL_MASK, (uint32_t)span);
        uint32_t nb = enc::w_closest_aligned(enc::w_closest(v2_bits(span)));
        if (nb == 1) nb = 2;
        const uint32_t len = m - 1u;
        if (lane == 0) {
            out[0] = (uint8_t)(0xC0u | ((uint32_t)enc::w_encode(nb) << 1) | ((len & 0x100u) >> 8));
            out[1] = (uint8_t)len;
        }
        uint32_t b = 2u + v2_varint((uint64_t)x0, out + 2);
        b += v2_varint(v2_zigzag(init), out + b);
        b += v2_pack(S.pk, 2, 127u, m - 2u, nb, out + b);
        stale = 0;
        return b;
    }
    stale = init;
    uint32_t cls[4], ge;
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r)
        cls[r] = lane + 32u * r < m ? enc::w_encode(v2_bits((uint64_t)x[r])) : 32u;
    v2_hist(cls, S, ge);
    const uint32_t b100 = enc::w_decode(v2_class(ge, 0)), b90 = enc::w_decode(v2_class(ge, v2_rank(m, 90)));
    if (b100 - b90 <= 1u) return v2_direct(S, i, m, bits, m - 1u, out);
    // ---- PATCHED_BASE, if the reduced values' widths differ too ----
    {
        uint64_t lo = ~0ull;
#pragma unroll
        for (uint32_t r = 0; r < 4; ++r)
            if (lane + 32u * r < m) lo = (uint64_t)x[r] < lo ? (uint64_t)x[r] : lo;
        const uint32_t h = __reduce_min_sync(GD_FULL_MASK, (uint32_t)(lo >> 32));
        const uint32_t l = __reduce_min_sync(GD_FULL_MASK, (uint32_t)(lo >> 32) == h ? (uint32_t)lo : 0xffffffffu);
        lmin = (int64_t)((uint64_t)h << 32 | l);
    }
    if (enc::w_closest(v2_bits((uint64_t)lmin)) == 64) {  // a base of 9 bytes
        uint32_t nb = 0;
        if (lane == 0) nb = v2_serial_run(S, i, m, out, &stale);
        stale = __shfl_sync(GD_FULL_MASK, stale, 0);
        return __shfl_sync(GD_FULL_MASK, nb, 0);
    }
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r)
        if (lane + 32u * r < m) {
            x[r] -= lmin;
            cls[r] = enc::w_encode(v2_bits((uint64_t)x[r]));
        }
    v2_hist(cls, S, ge);
    uint32_t b95 = enc::w_decode(v2_class(ge, v2_rank(m, 95)));
    const uint32_t top = enc::w_decode(v2_class(ge, 0));
    if (top == b95) return v2_direct(S, i, m, bits, m - 1u, out);
    uint32_t pw = enc::w_closest(top - b95);
    if (pw == 64) {
        pw = 56;
        b95 = 8;
    }
    const int64_t mask = (int64_t)((1ull << b95) - 1ull);
    uint32_t np = 0;
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
        const uint32_t k = lane + 32u * r;
        const bool patch = k < m && x[r] > mask;
        const uint32_t b = __ballot_sync(GD_FULL_MASK, patch);
        if (patch) {
            const uint32_t g = np + __popc(b & ((1u << lane) - 1u));
            S.pos[g] = (uint8_t)k;
            S.gp[g] = x[r] >> b95;
        }
        if (k < m) S.pk[k] = x[r] & mask;
        np += __popc(b);
    }
    __syncwarp();
    uint32_t gap = 0;
    for (uint32_t g = lane; g < np; g += 32) {
        const uint32_t d = S.pos[g] - (g ? S.pos[g - 1u] : 0u);
        gap = max(gap, d);
        S.gp[g] |= (int64_t)((uint64_t)d << pw);
    }
    gap = __reduce_max_sync(GD_FULL_MASK, gap);
    const uint32_t pgw = gap ? enc::w_closest(v2_bits(gap)) : 1u;
    const uint32_t vbytes = enc::w_closest(v2_bits((uint64_t)lmin)) / 8u + 1u;
    if (lane == 0) {
        const uint32_t vl = m - 1u;
        out[0] = (uint8_t)(0x80u | ((uint32_t)enc::w_encode(b95) << 1) | ((vl & 0x100u) >> 8));
        out[1] = (uint8_t)vl;
        out[2] = (uint8_t)(((vbytes - 1u) << 5) | enc::w_encode(pw));
        out[3] = (uint8_t)(((pgw - 1u) << 5) | np);
    }
    if (lane < vbytes) out[4 + lane] = (uint8_t)((uint64_t)lmin >> (8u * (vbytes - 1u - lane)));
    __syncwarp();
    uint32_t b = 4u + vbytes;
    b += v2_pack(S.pk, 0, 127u, m, enc::w_closest(b95), out + b);
    b += v2_pack(S.gp, 0, 127u, np, enc::w_closest(pgw + pw), out + b);
    return b;
}

// A warp per lane stream; col_len gets the stream's bytes, all ones if they
// outgrew the slot (lane_sizes_kernel turns that into a status).  skip (or
// null): nothing to do if it is not 0.
__global__ void __launch_bounds__(V2_WPB * 32) rlev2_encode_kernel(const uint8_t* __restrict__ in, uint64_t n_bytes,
                                                                   uint64_t n_lanes, uint64_t chunk_size,
                                                                   uint32_t read_unit, uint8_t* __restrict__ scratch,
                                                                   uint32_t lane_cap, uint64_t* __restrict__ col_len,
                                                                   const uint64_t* __restrict__ skip) {
    __shared__ V2Warp smem[V2_WPB];
    const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
    const uint64_t id = (uint64_t)blockIdx.x * V2_WPB + wid;  // 32 * chunk + lane stream
    if (id >= n_lanes || (skip && *skip)) return;  // warp-uniform
    V2Warp& S = smem[wid];
    const uint64_t cb = (id >> 5) * chunk_size;
    const uint64_t avail = (n_bytes > cb ? min((unsigned long long)(n_bytes - cb), (unsigned long long)chunk_size) : 0ull) / 8u;
    const int64_t* base = reinterpret_cast<const int64_t*>(in + cb);
    const uint32_t n = (uint32_t)(chunk_size / 256u), t = (uint32_t)id & 31u;
    uint32_t* slot = reinterpret_cast<uint32_t*>(scratch + id * lane_cap);

    uint32_t loaded = 0;   // a multiple of 32, or n rounded up to one
    int64_t last = 0;      // value loaded - 1
    uint32_t on = 0;       // bytes in S.out
    uint32_t written = 0;  // words in the slot
    bool over = false;
    int64_t stale = 0;
    // value k of the lane is chunk value (k / ru) * 32 * ru + t * ru + k % ru
    // (encoder_trans.h:40-108); values past the input are zero
    auto fetch = [&](uint32_t k) -> int64_t {
        if (k >= n) return 0;
        const uint32_t q = k / read_unit;
        const uint64_t at = (uint64_t)q * 32u * read_unit + (uint64_t)t * read_unit + (k - q * read_unit);
        return at < avail ? __ldg(base + at) : 0;
    };
    int64_t ahead = fetch(lane);  // values loaded .. loaded + 31, on their way
    for (uint32_t i = 0; i < n;) {
        while (loaded < n && loaded < i + 128u) {
            const int64_t v = ahead;
            ahead = fetch(loaded + 32u + lane);
            S.ring[(loaded + lane) & 255u] = v;
            const int64_t up = __shfl_down_sync(GD_FULL_MASK, v, 1);
            const uint32_t e = __ballot_sync(GD_FULL_MASK, lane < 31 && up == v);
            if (lane == 0) {
                S.eq[(loaded >> 5) & 7u] = e;
                if (loaded && v == last) S.eq[((loaded >> 5) - 1u) & 7u] |= 0x80000000u;
            }
            last = __shfl_sync(GD_FULL_MASK, v, 31);
            loaded += 32;
        }
        __syncwarp();
        // equal neighbours from value i on, those inside the lane and the next 128 values
        uint32_t E[5], a = S.eq[(i >> 5) & 7u];
        const uint32_t pairs = min(n - 1u - i, 127u);
#pragma unroll
        for (uint32_t w = 0; w < 4; ++w) {
            const uint32_t b = S.eq[((i >> 5) + w + 1u) & 7u];
            E[w] = __funnelshift_r(a, b, i);
            if (pairs < 32u * w + 32u) E[w] &= pairs > 32u * w ? (1u << (pairs - 32u * w)) - 1u : 0u;
            a = b;
        }
        E[4] = 0;
        uint32_t e = 128, j = 128;
#pragma unroll
        for (int w = 3; w >= 0; --w) {
            if (~E[w]) e = 32u * w + __ffs(~E[w]);  // the first unequal pair, counted from 1
            const uint32_t tri = E[w] & __funnelshift_r(E[w], E[w + 1], 1);
            if (tri) j = 32u * w + __ffs(tri) - 1u;
        }
        uint8_t* out = S.out + on;
        if (e >= 3 && e <= 10 && (E[0] >> e & 3u) == 3u) {
            // short runs one after the other, as many as the mask shows the
            // ends of (its bit 126 is the last that is known): a lane each
            const uint64_t lo = (uint64_t)E[1] << 32 | E[0], hi = (uint64_t)E[3] << 32 | E[2];
            uint32_t at = 0, k = 0, start = 0, m = 0;
            while (k < 32u && at < 126u) {
                const uint64_t x = at == 0u ? lo : at < 64u ? lo >> at | hi << (64u - at) : hi >> (at - 64u);
                const uint32_t ones = (uint32_t)__ffsll((long long)~x) - 1u;  // all ones: none
                if (ones - 2u > 7u || at + ones > 126u) break;
                if (lane == k) {
                    start = at;
                    m = ones + 1u;
                }
                at += ones + 1u;
                ++k;
            }
            const int64_t v = S.ring[(i + start) & 255u];
            const uint32_t nb = v < 0 ? 8u : (enc::w_closest(v2_bits((uint64_t)v)) + 7u) / 8u;
            const uint32_t size = lane < k ? 1u + nb : 0u, inc = warp_incl_scan(size);
            if (lane < k) {
                uint8_t* o = out + inc - size;
                o[0] = (uint8_t)(((nb - 1u) << 3) | (m - 3u));
#pragma unroll
                for (uint32_t b = 0; b < 8; ++b)
                    if (b < nb) o[1 + b] = (uint8_t)((uint64_t)v >> (8u * (nb - 1u - b)));
            }
            on += __shfl_sync(GD_FULL_MASK, inc, 31);
            i += at;
        } else if (e >= 3) {
            const int64_t v = S.ring[i & 255u];
            if (e <= 10) {
                const uint32_t nb = v < 0 ? 8u : (enc::w_closest(v2_bits((uint64_t)v)) + 7u) / 8u;
                if (lane == 0) out[0] = (uint8_t)(((nb - 1u) << 3) | (e - 3u));
                if (lane < nb) out[1 + lane] = (uint8_t)((uint64_t)v >> (8u * (nb - 1u - lane)));
                on += 1u + nb;
            } else if (e < 128) {
                on += v2_delta_fixed(v, stale, e, out);
                stale = 0;
            } else {
                // 128 equal values go through the general writer: one delta
                // of 0, or, if negative, DIRECT with a length of 0 - 1
                on += v >= 0 ? v2_delta_fixed(v, 0, 128, out) : v2_direct(S, i, 128, 64, 0xffffu, out);
                stale = 0;
            }
            i += e;
        } else {
            const uint32_t m = min(min(j, 128u), n - i);
            on += v2_var_run(S, i, m, stale, out);
            i += m;
        }
        __syncwarp();
        if (on >= V2_FLUSH || i >= n) {
            // whole words to the slot; at the end also the last, its unused bytes zero
            if (i >= n && lane < 4 && (on & 3u) && (on & 3u) + lane < 4u) S.out[on + lane] = 0;
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

// A warp per chunk: block size from the lane streams' bytes, and the status.
__global__ void __launch_bounds__(128) lane_sizes_kernel(uint32_t n_chunks, uint64_t* __restrict__ col_len,
                                                         uint64_t* __restrict__ blk_size,
                                                         uint32_t* __restrict__ status) {
    const uint32_t c = (blockIdx.x * 128u + threadIdx.x) >> 5, lane = lane_id();
    if (c >= n_chunks) return;  // warp-uniform
    const uint64_t n = col_len[(uint64_t)c * 32u + lane];
    const bool over = n == ~0ull;
    if (over) col_len[(uint64_t)c * 32u + lane] = 0;
    const uint32_t words = __reduce_add_sync(GD_FULL_MASK, over ? 0u : (uint32_t)((n + 3u) >> 2));
    const bool bad = __any_sync(GD_FULL_MASK, over);
    if (lane == 0) {
        blk_size[c] = ((uint64_t)words * 4u + 127u) & ~127ull;
        put_status(status, c, bad ? (uint32_t)ST_OVERRUN : (uint32_t)ST_OK);
    }
}

}  // namespace encd
}  // namespace gd
