// lzss_follow.cuh -- LZSS (32-column interleaved container) decoder for
// sm_100a that keeps a column's whole history in shared memory and takes the
// tokens of a column in parallel.
//
// Same container and statuses as the decoders of lzss.cuh.  A block decodes
// COLS adjacent output columns of a chunk, a warp per column after the walk:
//   stage   -- the columns' words are gathered from the interleaved rows;
//   walk    -- a lane per column follows its flag bytes (a group's size
//              follows from its flag byte alone) and notes where groups start;
//   tokens  -- 32 tokens (four groups) at a time, a lane each: a token's place
//              in its group follows from the flag byte, a warp scan of the
//              lengths gives the output offsets, literals are stored, and the
//              matches whose source lies before the first unfinished one are
//              copied together, 4 bytes a lane and step, until all are done;
//              after 32 literals, whole groups of literals a lane each;
//   rows    -- the block stores its part of every row, 16 bytes a thread.
// The lane-per-column decoders take some 1000 dependent tokens a column and
// read older history back from the output (15 chunks an SM: more history than
// the L2 holds): 1.43 ms for 256 MiB in 64 KiB chunks at 39% of the issue
// slots; this one 1.20 ms at 71%; random bytes, all literals, 1.40 and 0.85
// (a lane per literal throughout: 1.50).  Two forms that placed all tokens of a column
// first and then resolved its bytes 32 or 128 at a time took 1.34 and 1.28 ms:
// their tables left room for three blocks an SM instead of five.
#pragma once
#include "interleave.cuh"

namespace gd {
namespace lzss {

constexpr uint32_t FMAXL = 4096;  // column bytes, at most
// Stream bytes that a column of L bytes can use: L literals, a flag byte per
// 8 tokens and the reserved last one.
__host__ __device__ constexpr uint32_t follow_cap(uint32_t L) { return L + L / 8u + 2u; }
// Words of a column's stream buffer (a group may be read past the end).
__host__ __device__ constexpr uint32_t follow_words(uint32_t L) { return ((follow_cap(L) + 3u) / 4u + 5u + 3u) & ~3u; }
__host__ __device__ constexpr uint32_t follow_groups(uint32_t L) { return (follow_cap(L) / 9u + 4u) & ~3u; }
// Words of a column's output: 4 above a multiple of 32, so that the rows'
// reads of 8 columns fall on different banks.
__host__ __device__ constexpr uint32_t follow_out_words(uint32_t L) { return (L / 4u + 2u + 31u) / 32u * 32u + 4u; }
// stream, output, group starts
__host__ __device__ constexpr uint32_t follow_col_smem(uint32_t L) {
    return 4u * follow_words(L) + 4u * follow_out_words(L) + 2u * follow_groups(L);
}

template <uint32_t COLS>
__global__ void __launch_bounds__(COLS * 32, COLS == 8 ? 8 : 12) decode_follow_kernel(
    const uint8_t* __restrict__ data, const uint64_t* __restrict__ blk_off, const uint64_t* __restrict__ col_len,
    const uint8_t* __restrict__ col_map, uint32_t L, uint8_t* __restrict__ out, uint32_t* __restrict__ status) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ SegTable T;
    __shared__ uint32_t s_len[COLS], s_rank[COLS], s_ng[COLS], s_err;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
    const uint32_t chunk = blockIdx.x / (32u / COLS), c0 = blockIdx.x % (32u / COLS) * COLS;
    const uint32_t words = follow_words(L), owords = follow_out_words(L), groups = follow_groups(L);
    uint32_t* out0 = reinterpret_cast<uint32_t*>(smem);
    uint32_t* buf0 = out0 + COLS * owords;
    uint16_t* gp0 = reinterpret_cast<uint16_t*>(buf0 + COLS * words);  // where groups start
    const uint64_t b0 = blk_off[chunk], b1 = blk_off[chunk + 1];
    const uint8_t* block = data + b0;

    // ---- the chunk's streams ----
    if (wid == 0) {
        uint32_t err = ST_OK;
        const uint64_t len64 = col_len[32ull * chunk + lane];
        const uint32_t len = len64 > 0x3fffffffull ? 0u : (uint32_t)len64;
        const uint32_t q = col_map[32ull * chunk + lane];
        if (len64 > 0x3fffffffull || q >= 32) err = ST_CORRUPT;
        // col_map must be a permutation of the 32 columns
        if (__reduce_or_sync(GD_FULL_MASK, 1u << (q & 31u)) != 0xffffffffu) err = ST_CORRUPT;
        const uint32_t nw = (len + 3u) >> 2;
        const uint32_t tot = __shfl_sync(GD_FULL_MASK, warp_incl_scan(nw), 31);
        if (b1 < b0 || (uint64_t)tot * 4 > b1 - b0) err = ST_CORRUPT;
        if ((reinterpret_cast<uintptr_t>(block) & 3u) != 0) err = ST_CORRUPT;
        err = __reduce_max_sync(GD_FULL_MASK, err);
        seg_build(&T, nw);
        if (q - c0 < COLS) {
            s_len[q - c0] = len;
            s_rank[q - c0] = lane;
        }
        if (lane == 0) s_err = err;
    }
    __syncthreads();
    if (s_err != ST_OK) {
        if (tid == 0 && status) atomicMax(status + chunk, s_err);
        return;
    }
    // ---- stage: warp w the stream of column c0 + w ----
    const uint32_t len = s_len[wid];
    {
        uint32_t* d = buf0 + wid * words;
        const uint32_t nw = min((len + 3u) >> 2, (follow_cap(L) + 3u) >> 2), ltmask = (1u << s_rank[wid]) - 1u;
        uint32_t j = 0;
        for (uint32_t k = lane; k < nw; k += 32) {
            while (j < 31 && T.hi[j] <= k) ++j;
            const uint32_t lo = j ? T.hi[j - 1] : 0u;
            const uint32_t off = T.base[j] + (k - lo) * 4u * (32u - j) + 4u * __popc(T.mask[j] & ltmask);
            const uint32_t sa = (uint32_t)__cvta_generic_to_shared(d + k);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(block + off) : "memory");
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
        if (lane < 5) d[nw + lane] = 0;  // a group read past the end
    }
    __syncthreads();
    // ---- walk: lane c of warp 0 column c0 + c ----
    if (tid < COLS) {
        const uint8_t* s = reinterpret_cast<const uint8_t*>(buf0 + tid * words);
        uint16_t* gp = gp0 + tid * groups;
        const uint32_t n = min(s_len[tid], follow_cap(L));
        uint32_t g = 0;
        for (uint32_t p = 0; p < n; ++g) {
            gp[g] = (uint16_t)p;
            p += 9u + __popc(~(uint32_t)s[p] & 0xffu);
        }
        s_ng[tid] = g;
    }
    __syncthreads();
    // ---- tokens ----
    const uint8_t* s = reinterpret_cast<const uint8_t*>(buf0 + wid * words);
    const uint16_t* gp = gp0 + wid * groups;
    uint8_t* val = reinterpret_cast<uint8_t*>(out0 + wid * owords);
    const uint32_t ng = s_ng[wid], t = lane & 7u;
    uint32_t err = ST_OK, done = 0;  // output bytes
    for (uint32_t g0 = 0; g0 < ng && done < L; g0 += 4) {
        const uint32_t g = g0 + (lane >> 3);
        uint32_t n = 0, off = 0, v = 0, p = len;
        bool lit = true;
        if (g < ng) {
            const uint32_t q = gp[g], f = s[q];
            p = q + 1u + t + __popc(~f & ((1u << t) - 1u));
            lit = (f >> t) & 1u;
            v = s[p] | ((uint32_t)s[p + 1u] << 8);
            off = v >> 5;
            n = lit ? 1u : (v & 31u) + 3u;
        }
        const uint32_t inc = warp_incl_scan(n), o = done + inc - n;
        const bool live = g < ng && o < L;
        const bool corrupt = p + (lit ? 0u : 1u) >= len || (!lit && (off == 0 || off > o));
        const uint32_t badm = __ballot_sync(GD_FULL_MASK, live && (corrupt || o + n > L));
        if (badm) {  // the first bad token ends the column
            err = __shfl_sync(GD_FULL_MASK, corrupt ? (uint32_t)ST_CORRUPT : (uint32_t)ST_OVERRUN, __ffs(badm) - 1);
            break;
        }
        if (live && lit) val[o] = (uint8_t)v;
        const uint32_t src = o - off;
        uint32_t pend = __ballot_sync(GD_FULL_MASK, live && !lit);
        __syncwarp();
        const uint32_t end = done + __shfl_sync(GD_FULL_MASK, inc, 31);
        if (pend == 0) {
            done = end;
            // 32 literals: groups of literals as many as follow, up to 32 at a
            // time, a lane each
            while ((done & 3u) == 0) {
                const uint32_t h = g0 + 4u + lane, at = h < ng ? gp[h] : 0u;
                const bool all = h < ng && s[at] == 0xffu && at + 9u <= len && done + 8u * lane + 8u <= L;
                const uint32_t run = min(__ffs(~__ballot_sync(GD_FULL_MASK, all)) - 1u, 32u);
                if (lane < run) {
                    const uint32_t* w = buf0 + wid * words + ((at + 1u) >> 2);
                    const uint32_t w1 = w[1], sh = 8u * ((at + 1u) & 3u);
                    uint32_t* d = out0 + wid * owords + (done >> 2) + 2u * lane;
                    d[0] = __funnelshift_r(w[0], w1, sh);
                    d[1] = __funnelshift_r(w1, w[2], sh);
                }
                done += 8u * run;
                g0 += run;
                if (run < 32u) break;
            }
            __syncwarp();
            continue;
        }
        do {
            // everything before the first unfinished match is there
            const uint32_t fo = __shfl_sync(GD_FULL_MASK, o, __ffs(pend) - 1);
            const bool ready = ((pend >> lane) & 1u) && src + min(n, off) <= fo;
            if (ready) {
                if (off >= 4u) {
                    for (uint32_t j = 0; j < n; j += 4) {
                        const uint32_t a = src + j;
                        const uint32_t* w = reinterpret_cast<const uint32_t*>(val) + (a >> 2);
                        const uint32_t x = __funnelshift_r(w[0], w[1], 8u * (a & 3u));
                        uint8_t* d = val + o + j;
                        d[0] = (uint8_t)x;
                        if (j + 1 < n) d[1] = (uint8_t)(x >> 8);
                        if (j + 2 < n) d[2] = (uint8_t)(x >> 16);
                        if (j + 3 < n) d[3] = (uint8_t)(x >> 24);
                    }
                } else {
                    for (uint32_t j = 0; j < n; ++j) val[o + j] = val[src + j];
                }
            }
            pend &= ~__ballot_sync(GD_FULL_MASK, ready);
            __syncwarp();
        } while (pend);
        done = end;
    }
    if (err == ST_OK && done < L) err = ST_CORRUPT;
    if (err != ST_OK && lane == 0 && status) atomicMax(status + chunk, err);
    __syncthreads();
    // ---- rows: thread (row, quarter) 4 words ----
    constexpr uint32_t Q = COLS / 4u;
    uint4* dst = reinterpret_cast<uint4*>(out + (uint64_t)chunk * 32u * L + 4u * c0);
    for (uint32_t x = tid; x < L / 4u * Q; x += COLS * 32u) {
        const uint32_t k = x / Q, h = x % Q;
        const uint32_t* w = out0 + 4u * h * owords + k;
        dst[8u * k + h] = make_uint4(w[0], w[owords], w[2u * owords], w[3u * owords]);
    }
}

}  // namespace lzss
}  // namespace gd
