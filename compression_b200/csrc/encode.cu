// encode.cu -- RLE v1 and RLE v2 container encoders for sm_100a.
//
// The writer side of the two interleaved integer containers
// (rle_v1::compress_gpu, include/rle_v1/rlev1.h:25-97;
// rlev2::compress_gpu_transpose, include/rlev2/encoder_trans.h:428-537),
// producing the same bytes as the host encoders (gd_encode.cpp, lane_enc.h).
// Launches on one stream:
//   1. the lane streams, a warp each (rlev1_enc.cuh, rlev2_enc.cuh) or a thread
//      each (rle_thread_enc.cuh), into scratch slots; then a warp per chunk sums
//      the padded word counts into the chunk's block size;
//   2. offsets_kernel: one block turns the block sizes into blk_off;
//   3. interleave_kernel: row k = one word of every lane longer than 4k bytes,
//      in lane order, through the same segment table the decoders read with
//      (interleave.cuh), then the block's pad to 128 bytes zeroed.
// The column is read once and the scratch and the container written once each.
#include "gd_common.cuh"
#include "interleave.cuh"
#include "lane_enc.h"
#include "rle_thread_enc.cuh"
#include "rlev1_enc.cuh"
#include "rlev2_enc.cuh"

namespace gd {
namespace encd {

constexpr int NT = 128;  // threads per block

// blk_off[1..n] hold block sizes on entry and their inclusive prefix sums on
// exit; blk_off[0] = 0.  One block of 1024 threads, each over a contiguous
// range of chunks.
__global__ void __launch_bounds__(1024) offsets_kernel(uint64_t* __restrict__ blk_off, uint32_t n) {
    __shared__ uint64_t tmp[1024 / 32 + 1];
    const uint64_t per = ((uint64_t)n + 1023u) / 1024u;
    const uint64_t b = min((uint64_t)n, threadIdx.x * per), e = min((uint64_t)n, b + per);
    uint64_t sum = 0;
    for (uint64_t i = b; i < e; ++i) sum += blk_off[1 + i];
    uint64_t tot;
    uint64_t acc = block_excl_scan64<1024>(sum, tmp, &tot);
    for (uint64_t i = b; i < e; ++i) {
        acc += blk_off[1 + i];
        blk_off[1 + i] = acc;
    }
    if (threadIdx.x == 0) blk_off[0] = 0;
}

// Block c = slots' words in rows.  Slot t's stream is scratch slot
// col_map[32c + t] of the chunk (LZSS: slots are length ranks) or slot t
// (col_map null).  A block takes the chunk's tiles of 32 rows, every gridDim.y-th
// one: the 32 slots' words are read 128 bytes at a time, turned in shared
// memory, and every row is written by a warp, its words side by side.  (A warp
// per slot, storing one word in every row, wrote a sector per word: 0.124
// against 0.034 ms for 47 MB of RLE v1 streams.)
__global__ void __launch_bounds__(NT) interleave_kernel(const uint8_t* __restrict__ scratch, uint32_t lane_cap,
                                                        const uint64_t* __restrict__ col_len,
                                                        const uint64_t* __restrict__ blk_off, uint32_t n_chunks,
                                                        uint8_t* __restrict__ data,
                                                        const uint8_t* __restrict__ col_map = nullptr) {
    __shared__ SegTable T;
    __shared__ uint32_t s_nw[32];
    __shared__ uint32_t s_tot;
    __shared__ uint32_t s_slot[32];
    __shared__ uint32_t s_tile[32][33];
    const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
    for (uint32_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
        if (wid == 0) {
            const uint32_t nw = (uint32_t)((col_len[(uint64_t)c * 32u + lane] + 3u) >> 2);
            seg_build(&T, nw);
            s_nw[lane] = nw;
            s_slot[lane] = col_map ? (col_map[(uint64_t)c * 32u + lane] & 31u) : lane;
            const uint32_t tot = __reduce_add_sync(GD_FULL_MASK, nw);
            if (lane == 0) s_tot = tot;
        }
        __syncthreads();
        const uint64_t b0 = blk_off[c];
        uint32_t* dst = reinterpret_cast<uint32_t*>(data + b0);
        const uint32_t* src0 = reinterpret_cast<const uint32_t*>(scratch + (uint64_t)c * 32u * lane_cap);
        const uint32_t nw = s_nw[lane], rows = T.hi[31];
        for (uint32_t k0 = 32u * blockIdx.y; k0 < rows; k0 += 32u * gridDim.y) {
#pragma unroll
            for (uint32_t t = wid; t < 32; t += NT / 32)
                s_tile[t][lane] = k0 + lane < s_nw[t] ? src0[(uint64_t)s_slot[t] * (lane_cap / 4u) + k0 + lane] : 0u;
            __syncthreads();
#pragma unroll
            for (uint32_t r = wid; r < 32; r += NT / 32) {
                const uint32_t k = k0 + r;
                const uint32_t act = __ballot_sync(GD_FULL_MASK, nw > k), j = 32u - __popc(act);
                if (nw > k) {
                    const uint32_t lo = j ? T.hi[j - 1] : 0u;
                    const uint32_t off = (T.base[j] >> 2) + (k - lo) * (32u - j);
                    dst[off + __popc(act & ((1u << lane) - 1u))] = s_tile[lane][r];
                }
            }
            __syncthreads();
        }
        const uint32_t bw = (uint32_t)((blk_off[c + 1] - b0) >> 2);
        if (blockIdx.y == 0)
            for (uint32_t w = s_tot + threadIdx.x; w < bw; w += NT) dst[w] = 0;
        __syncthreads();  // T and s_nw are rebuilt for the next chunk
    }
}

// Grid of interleave_kernel: blocks for every chunk, and for every four tiles
// of the longest stream a slot can hold, up to 8 a chunk.
inline dim3 interleave_grid(uint64_t n_chunks, uint64_t lane_cap) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint64_t x = n_chunks < (uint64_t)sms * 16u ? n_chunks : (uint64_t)sms * 16u;
    const uint64_t y = lane_cap / 512u;
    return dim3((uint32_t)x, (uint32_t)(y < 1 ? 1 : y > 8 ? 8 : y));
}

// ---------------------------------------------------------------------------
// LZSS interleaved container (lzss::compress_gpu, include/lzss/lzss_gpu2.h:
// 1915-2127; columns by compress_init_func / compress_func_new :330-707)
// ---------------------------------------------------------------------------
//
// Column q of a chunk is the chunk's bytes [128k + 4q, 128k + 4q + 4) for
// every k; each column is one token stream: a flag byte before every 8
// tokens (bit set = literal byte, clear = 2-byte match v = offset << 5 |
// (length - 3), offsets 1..2047 back into the column, lengths 3..34).  The
// greedy writer takes at every position the oldest of the longest matches in
// the 2048-byte history (find_match, lzss_gpu2.h:70-108), so a position's
// match depends only on the position.  A warp per column:
//   - stages the column in shared memory and counts its positions by a hash of
//     their 3-byte keys, so that each bucket has its place;
//   - takes 32 positions at a time, a lane each: puts them into their buckets
//     (ascending inside each), finds the matches of all 32, a lane per pair of
//     a position and an older one of its bucket (compared 4 bytes at a time;
//     the longest match, then the oldest, is the largest of 16 bits), and then
//     the positions that the greedy walk visits, by doubling its jumps;
//   - where the 32 positions have more than LZ_PAIRS such pairs (long runs, few
//     distinct keys), walks them token by token instead, the candidates 32 at a
//     time from the oldest on, stopping at a 34-byte match;
//   - writes their tokens, a lane each, to a small buffer that leaves in words;
//     the open group's flag byte is rewritten until its 8 tokens are there.
// Bound by issue (66% of the slots at 24 warps per SM, set by shared memory).
// 64 MiB of Markov text with copies (a column: 383 matches, 618 literals,
// 7700 pairs in most, 45,000 in one of a hundred): 2.2 ms, 45,500 warp
// instructions a column, of which the pairs take 17,000 (62 for each 32), the
// windows that go token by token 7000, and the rest of a window about 200.
// Literals queued up to the next position with a match, then its candidates 32
// at a time (6.6 are in a bucket), took 3.2 ms; searching at every token 5.66.
// LZ_PAIRS: 256 2.15, 512 2.17, no limit 3.4 ms (columns of many pairs last
// longest).  320 buckets, for 7 blocks per SM, 2.22 ms; 1024, for 5, 2.40; the
// next pairs fetched ahead 2.18 ms.
// (Finding every position's match with a lane per position was slower still:
// the candidate lists differ in length, and are serial per lane.)

constexpr uint32_t LZ_WPB = 4;      // columns (warps) per block
// hash buckets of 3-byte keys; fewer for columns of up to LZ_SHORT bytes, whose
// time is mostly that of clearing and summing the buckets (4 MiB in 8 KiB chunks:
// zeros 0.102 ms, 512 buckets 0.123, 64 0.101; text 0.098, 0.115, 0.106; 1 MiB of
// text in 512-byte chunks 0.064, 0.159, 0.063)
constexpr uint32_t LZ_NB = 512, LZ_NB_SHORT = 128, LZ_SHORT = 256;
__host__ __device__ constexpr uint32_t lz_buckets(uint32_t L) { return L <= LZ_SHORT ? LZ_NB_SHORT : LZ_NB; }
constexpr uint32_t LZ_HIST = 2048, LZ_MAXM = 34, LZ_MINM = 3;
constexpr uint32_t LZ_OUT = 256;    // output bytes held back: less than 128, and the next 32 tokens' (37 at most)
constexpr uint32_t LZ_PAIRS = 256;  // pairs of 32 positions found at once

__host__ __device__ constexpr uint32_t a16(uint32_t x) { return (x + 15u) & ~15u; }
// column bytes (+64 zero pad) | positions by bucket, also the counts before them | bucket ends | bucket starts (the
// oldest in the history) | a word per lane | output
__host__ __device__ constexpr uint32_t lz_pos_bytes(uint32_t L) {
    return a16(2u * L > 4u * lz_buckets(L) ? 2u * L : 4u * lz_buckets(L));
}
__host__ __device__ constexpr uint32_t lz_warp_smem(uint32_t L) {
    return a16(L + 64u) + lz_pos_bytes(L) + 4u * lz_buckets(L) + 128u + LZ_OUT;
}
// the 4 bytes at p
__device__ __forceinline__ uint32_t lz_word(const uint8_t* d, uint32_t p) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(d) + (p >> 2);
    return __funnelshift_r(w[0], w[1], 8u * (p & 3u));
}
template <uint32_t NB>
__device__ __forceinline__ uint32_t lz_hash(uint32_t word) {
    return (((word & 0xffffffu) * 2654435761u) >> 16) * NB >> 16;
}

template <uint32_t NB>  // lz_buckets of the columns' length
__global__ void __launch_bounds__(LZ_WPB * 32) lzss_column_kernel(const uint8_t* __restrict__ in, uint64_t n_bytes,
                                                                  uint64_t chunk_size, uint32_t n_cols,
                                                                  uint8_t* __restrict__ scratch, uint32_t cap,
                                                                  uint32_t* __restrict__ raw_len, uint32_t wsm) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t lane = lane_id(), wid = threadIdx.x >> 5, lt = (1u << lane) - 1u;
    const uint32_t col = blockIdx.x * LZ_WPB + wid;  // 32 * chunk + column
    if (col >= n_cols) return;                        // warp-uniform
    const uint32_t q = col & 31u;
    const uint32_t L = (uint32_t)(chunk_size / 32u);
    uint8_t* d = smem + wid * wsm;
    uint16_t* pos = reinterpret_cast<uint16_t*>(d + a16(L + 64u));
    uint32_t* cnt = reinterpret_cast<uint32_t*>(pos);
    uint16_t* end = reinterpret_cast<uint16_t*>(reinterpret_cast<uint8_t*>(pos) + lz_pos_bytes(L));
    uint16_t* start = end + NB;
    uint32_t* area = reinterpret_cast<uint32_t*>(start + NB);
    uint8_t* out = reinterpret_cast<uint8_t*>(area + 32);
    const bool aged = L > LZ_HIST;  // candidates can leave the history

    // ---- the column: word k = chunk bytes [128k + 4q, +4); zero past the input ----
    const uint64_t cb = (uint64_t)(col >> 5) * chunk_size;
#pragma unroll 4
    for (uint32_t k = lane; k < L / 4u; k += 32) {
        const uint64_t g = cb + 128ull * k + 4u * q;
        uint32_t w = 0;
        if (g + 4 <= n_bytes) {
            w = __ldg(reinterpret_cast<const uint32_t*>(in + g));
        } else {
            for (uint32_t b = 0; b < 4; ++b)
                if (g + b < n_bytes) w |= (uint32_t)__ldg(in + g + b) << (8u * b);
        }
        reinterpret_cast<uint32_t*>(d)[k] = w;
    }
    for (uint32_t i = L / 4u + lane; i < L / 4u + 16u; i += 32) reinterpret_cast<uint32_t*>(d)[i] = 0;
    for (uint32_t b = lane; b < NB; b += 32) cnt[b] = 0;
    __syncwarp();

    // ---- where each bucket of the positions with a full key (p + 2 < L)
    // starts; not the first, which is never a source ----
    const uint32_t np = L - 2u;
    for (uint32_t p = 1u + lane; p < np; p += 32) atomicAdd(&cnt[lz_hash<NB>(lz_word(d, p))], 1u);
    __syncwarp();
    {
        constexpr uint32_t PER = NB / 32u;
        uint32_t v[PER], sum = 0;
#pragma unroll
        for (uint32_t i = 0; i < PER; ++i) {
            v[i] = cnt[lane * PER + i];
            sum += v[i];
        }
        uint32_t run = warp_incl_scan(sum) - sum;
#pragma unroll
        for (uint32_t i = 0; i < PER; ++i) {
            start[lane * PER + i] = end[lane * PER + i] = (uint16_t)run;
            run += v[i];
        }
    }
    __syncwarp();

    uint32_t* slot = reinterpret_cast<uint32_t*>(scratch + (uint64_t)col * cap);
    uint32_t on = 0, written = 0;              // bytes in out, words in the slot
    uint32_t nt = 0, flag_at = 0, flag = 0;    // tokens in the open group (0: none is), its flag byte's place, and bits
    bool over = false;
    // length of the match of the candidate c with the bytes at p (w, w4: the
    // words at p and p + 4), 0 if there is none
    auto match = [&](uint32_t c, uint32_t p, uint32_t w, uint32_t w4) -> uint32_t {
        const uint32_t* q = reinterpret_cast<const uint32_t*>(d) + (c >> 2);
        const uint32_t a0 = q[0], a1 = q[1], a2 = q[2], sh = 8u * (c & 3u);
        const uint32_t x = __funnelshift_r(a0, a1, sh) ^ w, y = __funnelshift_r(a1, a2, sh) ^ w4;
        uint32_t f = (uint32_t)(x ? __clz(__brev(x)) : 32 + __clz(__brev(y))) >> 3;
        const uint32_t off = p - c, lim = min(off, min(L - p, LZ_MAXM));
        if (off - LZ_MINM >= LZ_HIST - LZ_MINM) return 0;  // too near, or too old
        if (f == 8)
            for (; f < lim; f += 4) {
                const uint32_t z = lz_word(d, c + f) ^ lz_word(d, p + f);
                if (z) {
                    f += (uint32_t)(__ffs(z) - 1) >> 3;
                    break;
                }
            }
        f = min(f, lim);
        return f < LZ_MINM ? 0u : f;
    };
    uint32_t cur = 0;  // the next token's position
    for (uint32_t w0 = 0; w0 < L; w0 += 32) {
        // ---- the next 32 positions into their buckets ----
        const uint32_t p = w0 + lane, w = lz_word(d, p);
        const bool keyed = p >= 1u && p < np;
        const uint32_t h = keyed ? lz_hash<NB>(w) : NB + lane;
        const uint32_t peers = __match_any_sync(GD_FULL_MASK, h);
        uint32_t at = 0, first = 0;
        if (keyed) {
            at = end[h] + __popc(peers & lt);
            pos[at] = (uint16_t)p;
            first = start[h];
        }
        __syncwarp();
        if (aged) {
            // too old for all 32, and those after; the list may reach into these 32 positions
            if (keyed)
                while (first < at && pos[first] + LZ_HIST <= w0) ++first;
            __syncwarp();
        }
        if (keyed && (peers >> lane) == 1u) {  // the last of its bucket here
            end[h] = (uint16_t)(at + 1u);
            if (aged) start[h] = (uint16_t)first;
        }
        __syncwarp();
        if (cur >= w0 + 32u) continue;
        // ---- matches: a lane per (position, older position of its bucket) ----
        const uint32_t n = keyed && p >= cur ? at - first : 0u;
        const uint32_t w4 = lz_word(d, p + 4u);
        const uint32_t inc = warp_incl_scan(n), total = __shfl_sync(GD_FULL_MASK, inc, 31);
        uint32_t len = 1, next = w & 0xffu;  // this position's token: a byte, or a match's two
        uint32_t reach = cur < L ? 1u << (cur - w0) : 0u;  // positions where a token starts
        if (total <= LZ_PAIRS) {
            // a word per list: its position, and where it lies in pos, less the pairs before it
            const uint32_t excl = inc - n, has = __ballot_sync(GD_FULL_MASK, n != 0);
            if (n) area[__popc(has & lt)] = (first - excl) << 5 | lane;
            __syncwarp();
            const uint32_t list = area[lane];
            __syncwarp();
            area[lane] = 0;
            __syncwarp();
            uint32_t before = 0;  // lists that start before the step
            for (uint32_t t = 0; t < total; t += 32) {
                const uint32_t s =
                    __reduce_or_sync(GD_FULL_MASK, n && excl - t < 32u ? 1u << (excl - t) : 0u);  // lists that start here
                const uint32_t mine = __shfl_sync(GD_FULL_MASK, list, (int)(before + __popc(s & (lt << 1 | 1u)) - 1u));
                const uint32_t ow = __shfl_sync(GD_FULL_MASK, w, (int)(mine & 31u));
                const uint32_t ow4 = __shfl_sync(GD_FULL_MASK, w4, (int)(mine & 31u));
                before += __popc(s);
                if (t + lane < total) {
                    const uint32_t at0 = (uint32_t)((int32_t)mine >> 5) + t + lane, o = mine & 31u;
                    const uint32_t c = pos[at0], f = match(c, w0 + o, ow, ow4);
                    if (f) atomicMax(&area[o], (f - LZ_MINM) << 11 | (w0 + o - c));
                }
            }
            __syncwarp();
            const uint32_t v = area[lane];
            if (v) {
                len = (v >> 11) + LZ_MINM;
                next = (v & 0x7ffu) << 5 | v >> 11;
            }
            // the positions that the walk visits: after k rounds, those up to 2^k - 1 tokens on
            uint32_t to = p + len < L ? min(lane + len, 32u) : 32u;
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                reach |= __reduce_or_sync(GD_FULL_MASK, (reach >> lane & 1u) && to < 32u ? 1u << to : 0u);
                const uint32_t on2 = __shfl_sync(GD_FULL_MASK, to, (int)(to & 31u));
                if (to < 32u) to = on2;
            }
        } else {
            for (uint32_t q = cur - w0; q < 32u && w0 + q < L;) {
                const uint32_t qw = __shfl_sync(GD_FULL_MASK, w, q), qw4 = __shfl_sync(GD_FULL_MASK, w4, q);
                const uint32_t qat = __shfl_sync(GD_FULL_MASK, at, q);
                uint32_t best = 0;  // (length - 3) << 11 | offset
                for (uint32_t i = __shfl_sync(GD_FULL_MASK, first, q); i < qat; i += 32) {
                    const uint32_t c = i + lane < qat ? pos[i + lane] : w0 + q;  // itself: no match
                    const uint32_t f = match(c, w0 + q, qw, qw4);
                    best = max(best, __reduce_max_sync(GD_FULL_MASK, f ? (f - LZ_MINM) << 11 | (w0 + q - c) : 0u));
                    if (best >> 11 == LZ_MAXM - LZ_MINM) break;  // later candidates are nearer
                }
                const uint32_t step = best ? (best >> 11) + LZ_MINM : 1u;
                if (lane == q && best) {
                    len = step;
                    next = (best & 0x7ffu) << 5 | best >> 11;
                }
                reach |= 1u << q;
                q += step;
            }
        }
        if (!reach) break;  // the column's end
        // ---- their bytes, and a flag byte before every 8 ----
        const uint32_t k = __popc(reach), last = 31u - __clz(reach);
        cur = w0 + last + __shfl_sync(GD_FULL_MASK, len, last);
        const bool here = reach >> lane & 1u, lit = len == 1u;
        const uint32_t long_ones = __ballot_sync(GD_FULL_MASK, here && !lit);
        const uint32_t rank = __popc(reach & lt), g = nt + rank;
        const uint32_t lits = __reduce_or_sync(GD_FULL_MASK, here && lit ? 1u << rank : 0u);
        const uint64_t flags = (uint64_t)lits << nt | flag;
        const uint32_t place = on + rank + __popc(long_ones & lt) + (g >> 3) + (nt ? 0u : 1u);
        if (here) {
            if ((g & 7u) == 0) out[place - 1u] = (uint8_t)(flags >> g);
            out[place] = (uint8_t)next;
            if (!lit) out[place + 1u] = (uint8_t)(next >> 8);
        }
        if (nt && lane == 0) out[flag_at] = (uint8_t)flags;
        on += k + __popc(long_ones) + ((nt + k + 7u) >> 3) - (nt ? 1u : 0u);
        const uint32_t open = (nt + k) & ~7u;  // the open group's first token
        const uint32_t opener = __ballot_sync(GD_FULL_MASK, here && g == open);
        if (opener) flag_at = __shfl_sync(GD_FULL_MASK, place, __ffs(opener) - 1) - 1u;
        nt = (nt + k) & 7u;
        flag = (uint32_t)(flags >> open) & 0xffu;
        __syncwarp();
        if (on >= LZ_OUT / 2u) {  // whole words, up to the open group
            const uint32_t nw = (nt ? flag_at : on) >> 2;
            over = over || 4u * (written + nw) > cap;
            if (!over)
                for (uint32_t i = lane; i < nw; i += 32) slot[written + i] = reinterpret_cast<const uint32_t*>(out)[i];
            written += nw;
            on -= 4u * nw;
            flag_at -= 4u * nw;
            uint8_t keep = 0;  // 3 bytes and 8 tokens at most
            if (lane < on) keep = out[4u * nw + lane];
            __syncwarp();
            if (lane < on) out[lane] = keep;
            __syncwarp();
        }
    }
    // the end: a reserved flag byte after a full group, zeros to a whole word
    if (nt == 0) {
        if (lane == 0) out[on] = 0;
        ++on;
    }
    if ((on & 3u) && (on & 3u) + lane < 4u) out[on + lane] = 0;
    __syncwarp();
    over = over || 4u * written + ((on + 3u) & ~3u) > cap;
    if (!over)
        for (uint32_t i = lane; i < (on + 3u) >> 2; i += 32) slot[written + i] = reinterpret_cast<const uint32_t*>(out)[i];
    if (lane == 0) raw_len[col] = over ? 0xffffffffu : 4u * written + on;
}

// A warp per chunk: slots are the columns by descending stream length (equal
// lengths: the higher column first, as the reference's stable ascending sort
// read backwards); col_map[32c + slot] = column, col_len in slot order, and
// the chunk's block size into blk_size[c].
__global__ void __launch_bounds__(NT) lzss_rank_kernel(const uint32_t* __restrict__ raw_len, uint32_t n_chunks,
                                                       uint64_t* __restrict__ col_len, uint8_t* __restrict__ col_map,
                                                       uint64_t* __restrict__ blk_size, uint32_t* __restrict__ status) {
    const uint32_t c = (blockIdx.x * NT + threadIdx.x) >> 5;
    const uint32_t q = lane_id();
    if (c >= n_chunks) return;  // warp-uniform
    const uint32_t r0 = raw_len[(uint64_t)c * 32u + q];
    const bool over = r0 == 0xffffffffu;
    const uint32_t len = over ? 0u : r0;
    uint32_t rank = 0;
#pragma unroll 8
    for (uint32_t o = 0; o < 32; ++o) {
        const uint32_t lo = __shfl_sync(GD_FULL_MASK, len, o);
        rank += (lo > len) || (lo == len && o > q);
    }
    col_map[(uint64_t)c * 32u + rank] = (uint8_t)q;
    col_len[(uint64_t)c * 32u + rank] = len;
    const uint32_t words = __reduce_add_sync(GD_FULL_MASK, (len + 3u) >> 2);
    const bool bad = __any_sync(GD_FULL_MASK, over);
    if (q == 0) {
        blk_size[c] = ((uint64_t)words * 4u + 127u) & ~127ull;
        put_status(status, c, bad ? (uint32_t)ST_OVERRUN : (uint32_t)ST_OK);
    }
}

// Longest lane stream the encoders can write for nv values, rounded to 4:
// RLE v1 -- every value a literal varint (5 / 10 bytes) plus a header byte
// per 127 literals; RLE v2 -- at most 10 bytes per value for a one-value
// DIRECT run (2 header bytes + 8), less for every other run.
inline uint64_t rlev1_lane_cap(uint64_t chunk_size, uint32_t eb) {
    const uint64_t ne = chunk_size / 32u / eb;
    return (ne * (eb == 4 ? 5u : 10u) + ne / 64u + 16u + 3u) & ~3ull;
}
// LZSS column of L bytes: all literals, a flag byte per 8 tokens and the
// reserved one after the last group
inline uint64_t lzss_col_cap(uint64_t chunk_size) {
    const uint64_t L = chunk_size / 32u;
    return (L + L / 8u + 8u + 3u) & ~3ull;
}
inline uint64_t rlev2_lane_cap(uint64_t chunk_size) {
    const uint64_t nv = chunk_size / 256u;
    return (nv * 11u + 64u + 3u) & ~3ull;
}

// Lane streams of n values by a thread each where that is the faster: its time
// grows with n and, up to a chip full of them, hardly with their number; the warp
// encoders' grows with the tokens.  Time by threads over time by warps, RLE v1 of
// 4-byte values:
//    n    lanes: 8 K  32 K  128 K  512 K   (runs and literals alternating)
//     8          0.42  0.45   0.41   0.42
//    16          0.88  0.62   0.50   0.47
//    32          1.28  0.97   0.67   0.66
//    64          1.95  1.46   0.99   0.88
//   128          2.39  1.44   1.06   1.14
//   512          4.4   2.2    1.4    1.7
//  1024          8.4   3.4    2.3    2.3
// (8-byte values n = 64 1.66, 1.01, 0.68, 0.70)
// RLE v2 n = 16 1.82, 1.07, 0.89, 0.78, n = 1024 18.8, 7.4, 6.4.  Of runs of 8
// equal values, which are a token each, taken one by one: n = 128 0.94, 0.39, 0.22,
// 0.21, n = 1024 1.85, 0.61, 0.25, 0.22; RLE v2 n = 32 1.33, 0.89, 0.78, 0.58, n =
// 1024 1.75, 0.64, 0.54 (several at a time the warps take half as long).  So short
// lanes go by the sizes, and in columns of over 16,384 lanes (n < 512: as many) a
// sample tells: an end of a run for every 32 values (RLE v2: 14).  It and the
// launch that finds nothing to do take 6 to 8 us, which smaller columns would feel
// (64 MiB in 128 KiB chunks 0.222 ms; there runs of 8 take 0.23 ms by warps, 0.30
// by threads).
inline ThreadRule rlev1_by_thread(uint64_t lanes, uint64_t n, uint32_t elem_bytes) {
    const bool all = n < 16 || (n < 32 && lanes >= 8192) || (n < 64 && lanes >= 32768) || (n < 128 && lanes >= 262144 / elem_bytes) ||
                     (n < 256 && lanes >= 131072);
    return {all, !all && (lanes > 16384 || (n < 512 && lanes >= 16384)) ? SAMPLE : 0u};
}
inline ThreadRule rlev2_by_thread(uint64_t lanes, uint64_t n) {
    const bool all = n < 4 || (n < 8 && lanes >= 8192) || (n < 16 && lanes >= 16384) || (n < 32 && lanes >= 32768);
    return {all, !all && (lanes > 16384 || (n < 512 && lanes >= 16384)) ? SAMPLE * 9u / 4u : 0u};
}

// blk_off from the block sizes, then the container.
inline gd_status_t finish(uint64_t nc, const uint8_t* d_scratch, uint64_t lane_cap, uint8_t* d_data,
                          uint64_t* d_blk_off, const uint64_t* d_col_len, const uint8_t* d_col_map, cudaStream_t s) {
    offsets_kernel<<<1, 1024, 0, s>>>(d_blk_off, (uint32_t)nc);
    interleave_kernel<<<interleave_grid(nc, lane_cap), NT, 0, s>>>(d_scratch, (uint32_t)lane_cap, d_col_len, d_blk_off,
                                                                  (uint32_t)nc, d_data, d_col_map);
    return cudaGetLastError() == cudaSuccess ? GD_OK : GD_ERR_CUDA;
}

}  // namespace encd
}  // namespace gd

using namespace gd::encd;

extern "C" uint64_t gd_rlev1_encode_bound(uint64_t n_bytes, uint64_t chunk_size, uint32_t elem_bytes) {
    if (n_bytes == 0 || chunk_size == 0 || !(elem_bytes == 4 || elem_bytes == 8)) return 0;
    return (n_bytes + chunk_size - 1) / chunk_size * 32u * rlev1_lane_cap(chunk_size, elem_bytes);
}

extern "C" gd_status_t gd_rlev1_encode_device(const uint8_t* d_in, uint64_t n_bytes, uint64_t chunk_size,
                                              uint32_t comp_col_len, uint32_t elem_bytes, uint8_t* d_scratch,
                                              uint8_t* d_data, uint64_t* d_blk_off, uint64_t* d_col_len,
                                              uint32_t* d_status, gd_stream_t stream) {
    if (n_bytes == 0) return GD_OK;
    if (!d_in || !d_scratch || !d_data || !d_blk_off || !d_col_len) return GD_ERR_INVALID_ARG;
    if (!(elem_bytes == 4 || elem_bytes == 8) || n_bytes % elem_bytes) return GD_ERR_INVALID_ARG;
    if (comp_col_len == 0 || comp_col_len % elem_bytes) return GD_ERR_INVALID_ARG;
    if (chunk_size == 0 || chunk_size % (32ull * comp_col_len) || chunk_size > (1ull << 30))
        return GD_ERR_INVALID_ARG;
    if ((reinterpret_cast<uintptr_t>(d_in) % elem_bytes) || (reinterpret_cast<uintptr_t>(d_scratch) & 3u) ||
        (reinterpret_cast<uintptr_t>(d_data) & 3u))
        return GD_ERR_INVALID_ARG;
    if ((n_bytes + chunk_size - 1) / chunk_size > 0xffffffffull) return GD_ERR_UNSUPPORTED;
    // a lane of one value cannot be encoded (the writer starts from two)
    if (chunk_size / 32u / elem_bytes < 2) return GD_ERR_UNSUPPORTED;
    const uint64_t cap = rlev1_lane_cap(chunk_size, elem_bytes);
    const uint32_t wil = comp_col_len / elem_bytes;
    cudaStream_t s = (cudaStream_t)stream;
    const uint64_t nc = (n_bytes + chunk_size - 1) / chunk_size;
    auto go = [&](auto value) {
        using T = decltype(value);
        const ThreadRule by = rlev1_by_thread(nc * 32u, chunk_size / 32u / sizeof(T), sizeof(T));
        uint64_t* runs = by.ends ? d_blk_off : nullptr;  // until the offsets are there
        if (runs)
            sample_runs_kernel<GD_CODEC_RLEV1, T>
                <<<1, 1024, 0, s>>>(reinterpret_cast<const T*>(d_in), n_bytes / sizeof(T), by.ends, runs);
        if (by.all || runs)
            thread_encode_kernel<GD_CODEC_RLEV1, T><<<(uint32_t)((nc + 3) / 4), THREAD_NT, 0, s>>>(
                d_in, n_bytes, (uint32_t)nc, chunk_size, wil, d_scratch, (uint32_t)cap, d_col_len, runs, d_blk_off + 1,
                d_status);
        if (!by.all) {
            rlev1_encode_kernel<T><<<(uint32_t)((nc * 32u + V1_WPB - 1) / V1_WPB), V1_WPB * 32, 0, s>>>(
                d_in, n_bytes, nc * 32u, chunk_size, wil, d_scratch, (uint32_t)cap, d_col_len, runs);
            lane_sizes_kernel<<<(uint32_t)((nc + 3) / 4), 128, 0, s>>>((uint32_t)nc, d_col_len, d_blk_off + 1,
                                                                       d_status);
        }
    };
    if (elem_bytes == 4) go(uint32_t{});
    else go(uint64_t{});
    return finish(nc, d_scratch, cap, d_data, d_blk_off, d_col_len, nullptr, s);
}

extern "C" uint64_t gd_rlev2_encode_bound(uint64_t n_bytes, uint64_t chunk_size) {
    if (n_bytes == 0 || chunk_size == 0) return 0;
    return (n_bytes + chunk_size - 1) / chunk_size * 32u * rlev2_lane_cap(chunk_size);
}

extern "C" gd_status_t gd_rlev2_encode_device(const uint8_t* d_in, uint64_t n_bytes, uint64_t chunk_size,
                                              uint32_t read_unit, uint8_t* d_scratch, uint8_t* d_data,
                                              uint64_t* d_blk_off, uint64_t* d_col_len, uint32_t* d_status,
                                              gd_stream_t stream) {
    if (n_bytes == 0) return GD_OK;
    if (!d_in || !d_scratch || !d_data || !d_blk_off || !d_col_len) return GD_ERR_INVALID_ARG;
    if (read_unit == 0 || n_bytes % 8) return GD_ERR_INVALID_ARG;
    if (chunk_size == 0 || chunk_size % (256ull * read_unit) || chunk_size > (1ull << 30)) return GD_ERR_INVALID_ARG;
    if ((reinterpret_cast<uintptr_t>(d_in) & 7u) || (reinterpret_cast<uintptr_t>(d_scratch) & 3u) ||
        (reinterpret_cast<uintptr_t>(d_data) & 3u))
        return GD_ERR_INVALID_ARG;
    if ((n_bytes + chunk_size - 1) / chunk_size > 0xffffffffull) return GD_ERR_UNSUPPORTED;
    const uint64_t nc = (n_bytes + chunk_size - 1) / chunk_size, cap = rlev2_lane_cap(chunk_size);
    cudaStream_t s = (cudaStream_t)stream;
    const ThreadRule by = rlev2_by_thread(nc * 32u, chunk_size / 256u);
    uint64_t* runs = by.ends ? d_blk_off : nullptr;  // until the offsets are there
    if (runs)
        sample_runs_kernel<GD_CODEC_RLEV2, int64_t>
            <<<1, 1024, 0, s>>>(reinterpret_cast<const int64_t*>(d_in), n_bytes / 8u, by.ends, runs);
    if (by.all || runs)
        thread_encode_kernel<GD_CODEC_RLEV2, int64_t><<<(uint32_t)((nc + 3) / 4), THREAD_NT, 0, s>>>(
            d_in, n_bytes, (uint32_t)nc, chunk_size, read_unit, d_scratch, (uint32_t)cap, d_col_len, runs, d_blk_off + 1,
            d_status);
    if (!by.all) {
        rlev2_encode_kernel<<<(uint32_t)((nc * 32u + V2_WPB - 1) / V2_WPB), V2_WPB * 32, 0, s>>>(
            d_in, n_bytes, nc * 32u, chunk_size, read_unit, d_scratch, (uint32_t)cap, d_col_len, runs);
        lane_sizes_kernel<<<(uint32_t)((nc + 3) / 4), 128, 0, s>>>((uint32_t)nc, d_col_len, d_blk_off + 1, d_status);
    }
    return finish(nc, d_scratch, cap, d_data, d_blk_off, d_col_len, nullptr, s);
}

extern "C" uint64_t gd_lzss_encode_bound(uint64_t n_bytes, uint64_t chunk_size) {
    if (n_bytes == 0 || chunk_size == 0) return 0;
    return (n_bytes + chunk_size - 1) / chunk_size * 32u * (lzss_col_cap(chunk_size) + 4u) + 16u;
}

extern "C" gd_status_t gd_lzss_encode_device(const uint8_t* d_in, uint64_t n_bytes, uint64_t chunk_size,
                                             uint8_t* d_scratch, uint8_t* d_data, uint64_t* d_blk_off,
                                             uint64_t* d_col_len, uint8_t* d_col_map, uint32_t* d_status,
                                             gd_stream_t stream) {
    if (n_bytes == 0) return GD_OK;
    if (!d_in || !d_scratch || !d_data || !d_blk_off || !d_col_len || !d_col_map) return GD_ERR_INVALID_ARG;
    if (chunk_size == 0 || chunk_size % 128u || chunk_size > 128u * 1024u) return GD_ERR_INVALID_ARG;
    if ((reinterpret_cast<uintptr_t>(d_in) & 3u) || (reinterpret_cast<uintptr_t>(d_scratch) & 3u) ||
        (reinterpret_cast<uintptr_t>(d_data) & 3u))
        return GD_ERR_INVALID_ARG;
    const uint64_t nc = (n_bytes + chunk_size - 1) / chunk_size;
    if (nc * 32u > 0xffffffffull) return GD_ERR_UNSUPPORTED;
    const uint64_t cap = lzss_col_cap(chunk_size);
    uint32_t* raw_len = reinterpret_cast<uint32_t*>(d_scratch + nc * 32u * cap);
    const uint32_t L = (uint32_t)(chunk_size / 32u);
    const uint32_t wsm = lz_warp_smem(L);
    cudaStream_t s = (cudaStream_t)stream;
    auto kern = lz_buckets(L) == LZ_NB ? lzss_column_kernel<LZ_NB> : lzss_column_kernel<LZ_NB_SHORT>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LZ_WPB * wsm);
    const uint32_t ncol = (uint32_t)(nc * 32u);
    kern<<<(ncol + LZ_WPB - 1) / LZ_WPB, LZ_WPB * 32, LZ_WPB * wsm, s>>>(
        d_in, n_bytes, chunk_size, ncol, d_scratch, (uint32_t)cap, raw_len, wsm);
    lzss_rank_kernel<<<(uint32_t)((nc + NT / 32 - 1) / (NT / 32)), NT, 0, s>>>(raw_len, (uint32_t)nc, d_col_len,
                                                                              d_col_map, d_blk_off + 1, d_status);
    return finish(nc, d_scratch, cap, d_data, d_blk_off, d_col_len, d_col_map, s);
}

// ---------------------------------------------------------------------------
// Byte-RLE flag container (brle_trans::compress_gpu, include/brle/brle_trans.h:
// 563-660; column streams by compress_func :437-562)
// ---------------------------------------------------------------------------
//
// Same column split, ranking and interleave as the LZSS container; only the
// column stream differs: maximal runs of equal bytes, a run of 3 or more as a
// run item (count byte, value byte; flag bit 0), a shorter one as that many
// literal items (flag bit 1), a flag byte before every 8 items (LSB first)
// and, after the 8th item of a group, the next flag byte reserved (0 if no
// item follows) -- except after the column's last item when that is a run,
// which the reference writes without counting it (brle_trans.h:529-536).  A thread per column: the warp's 32 lanes are one chunk's
// 32 columns, so each step reads 128 contiguous input bytes.  Output bytes
// gather in a word register; a group's flag byte goes into that register when
// its word is still open, else it is stored over the 0 already written.
// Run counts fit the count byte because a column holds at most 252 bytes.

__global__ void __launch_bounds__(NT) brle_trans_column_kernel(const uint8_t* __restrict__ in, uint64_t n_bytes,
                                                               uint64_t chunk_size, uint32_t n_cols,
                                                               uint8_t* __restrict__ scratch, uint32_t cap,
                                                               uint32_t* __restrict__ raw_len) {
    const uint32_t col = blockIdx.x * NT + threadIdx.x;
    if (col >= n_cols) return;
    const uint64_t c = col >> 5;
    const uint32_t q = col & 31u;
    const uint32_t L = (uint32_t)(chunk_size / 32u);
    const uint64_t base = c * chunk_size + 4u * q;
    uint8_t* slot = scratch + (uint64_t)col * cap;
    uint32_t* wslot = reinterpret_cast<uint32_t*>(slot);
    uint32_t pos = 1, hpos = 0, items = 0, flags = 0, wbuf = 0;  // byte 0: the first flag byte
    auto put = [&](uint32_t b) {
        wbuf |= b << (8u * (pos & 3u));
        if ((++pos & 3u) == 0) {
            wslot[(pos >> 2) - 1u] = wbuf;
            wbuf = 0;
        }
    };
    auto set_flag = [&]() {
        if (hpos >= (pos & ~3u))
            wbuf |= flags << (8u * (hpos & 3u));
        else
            slot[hpos] = (uint8_t)flags;
    };
    auto item_done = [&]() {
        if (++items == 8u) {
            set_flag();
            flags = 0;
            items = 0;
            hpos = pos;
            put(0u);
        }
    };
    auto emit = [&](uint32_t v, uint32_t run, bool last) {
        if (run >= 3u) {
            put(run);
            put(v);
            if (!last) item_done();  // the column's last run is written uncounted
        } else {
            for (uint32_t k = 0; k < run; ++k) {
                flags |= 1u << items;
                put(v);
                item_done();
            }
        }
    };
    uint32_t cur = 0, run = 0;
    for (uint32_t k = 0; k < L / 4u; ++k) {
        const uint64_t at = base + 128ull * k;
        uint32_t w = 0;
        if (at + 4u <= n_bytes) {
            w = *reinterpret_cast<const uint32_t*>(in + at);
        } else {
            for (uint32_t b = 0; b < 4u; ++b)
                if (at + b < n_bytes) w |= (uint32_t)in[at + b] << (8u * b);
        }
#pragma unroll
        for (uint32_t b = 0; b < 4u; ++b) {
            const uint32_t x = (w >> (8u * b)) & 0xffu;
            if (run && x == cur) {
                ++run;
            } else {
                if (run) emit(cur, run, false);
                cur = x;
                run = 1;
            }
        }
    }
    if (run) emit(cur, run, true);
    if (items) set_flag();
    if (pos & 3u) wslot[pos >> 2] = wbuf;
    raw_len[col] = pos;
}

extern "C" uint64_t gd_brle_trans_encode_bound(uint64_t n_bytes, uint64_t chunk_size) {
    if (n_bytes == 0 || chunk_size == 0) return 0;
    return (n_bytes + chunk_size - 1) / chunk_size * 32u * (lzss_col_cap(chunk_size) + 4u) + 16u;
}

extern "C" gd_status_t gd_brle_trans_encode_device(const uint8_t* d_in, uint64_t n_bytes, uint64_t chunk_size,
                                                   uint8_t* d_scratch, uint8_t* d_data, uint64_t* d_blk_off,
                                                   uint64_t* d_col_len, uint8_t* d_col_map, uint32_t* d_status,
                                                   gd_stream_t stream) {
    if (n_bytes == 0) return GD_OK;
    if (!d_in || !d_scratch || !d_data || !d_blk_off || !d_col_len || !d_col_map) return GD_ERR_INVALID_ARG;
    if (chunk_size == 0 || chunk_size % 128u || chunk_size / 32u > 252u) return GD_ERR_INVALID_ARG;
    if ((reinterpret_cast<uintptr_t>(d_in) & 3u) || (reinterpret_cast<uintptr_t>(d_scratch) & 3u) ||
        (reinterpret_cast<uintptr_t>(d_data) & 3u))
        return GD_ERR_INVALID_ARG;
    const uint64_t nc = (n_bytes + chunk_size - 1) / chunk_size;
    if (nc * 32u > 0xffffffffull) return GD_ERR_UNSUPPORTED;
    const uint64_t cap = lzss_col_cap(chunk_size);
    uint32_t* raw_len = reinterpret_cast<uint32_t*>(d_scratch + nc * 32u * cap);
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t ncol = (uint32_t)(nc * 32u);
    brle_trans_column_kernel<<<(ncol + NT - 1) / NT, NT, 0, s>>>(d_in, n_bytes, chunk_size, ncol, d_scratch,
                                                                 (uint32_t)cap, raw_len);
    lzss_rank_kernel<<<(uint32_t)((nc + NT / 32 - 1) / (NT / 32)), NT, 0, s>>>(raw_len, (uint32_t)nc, d_col_len,
                                                                              d_col_map, d_blk_off + 1, d_status);
    return finish(nc, d_scratch, cap, d_data, d_blk_off, d_col_len, d_col_map, s);
}
