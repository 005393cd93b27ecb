// encode.cu -- RLE v1 and RLE v2 container encoders for sm_100a.
//
// The writer side of the two interleaved integer containers
// (rle_v1::compress_gpu, include/rle_v1/rlev1.h:25-97;
// rlev2::compress_gpu_transpose, include/rlev2/encoder_trans.h:428-537),
// producing the same bytes as the host encoders (gd_encode.cpp, lane_enc.h).
// Launches on one stream:
//   1. the lane streams, a warp each (rlev1_enc.cuh, rlev2_enc.cuh), into
//      scratch slots; then a warp per chunk sums the padded word counts into
//      the chunk's block size;
//   2. offsets_kernel: one block turns the block sizes into blk_off;
//   3. interleave_kernel: row k = one word of every lane longer than 4k bytes,
//      in lane order, through the same segment table the decoders read with
//      (interleave.cuh), then the block's pad to 128 bytes zeroed.
// The column is read once and the scratch and the container written once each.
#include "gd_common.cuh"
#include "interleave.cuh"
#include "lane_enc.h"
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
//   - stages the column in shared memory and sorts its positions by a hash of
//     their 3-byte keys, ascending inside a bucket;
//   - marks the positions that have a match, a lane per sorted position
//     looking back in its bucket for its key (usually the entry before);
//   - walks the tokens: literals up to the next marked position in one step,
//     and there the bucket's candidates 32 at a time, oldest first (one lane
//     per candidate, compared 4 bytes at a time, the longest with the oldest
//     winning ties), stopping at a 34-byte match;
//   - queues tokens a lane each and writes 32 (four flag groups) together.
// Searching at every token, literals too (64% of the benchmark's), and writing
// each token from one lane took 88 warp instructions a token and 5.66 ms for
// 64 MiB.  (Finding every position's match with a lane per position was 2.4x
// slower still: the candidate lists are long, and serial per lane.)

constexpr uint32_t LZ_WPB = 4;      // columns (warps) per block
constexpr uint32_t LZ_NB = 512;     // hash buckets of 3-byte keys
constexpr uint32_t LZ_HIST = 2048, LZ_MAXM = 34, LZ_MINM = 3;
constexpr uint32_t LZ_OUT = 256;    // output bytes held back: less than 128, and the next 32 tokens

__host__ __device__ constexpr uint32_t a16(uint32_t x) { return (x + 15u) & ~15u; }
// column bytes (+64 zero pad) | positions by bucket, also the counts before them | bucket ends | marks | output |
// oldest candidates by bucket, where the column is longer than the history
__host__ __device__ constexpr uint32_t lz_pos_bytes(uint32_t L) { return a16(2u * L > 4u * LZ_NB ? 2u * L : 4u * LZ_NB); }
__host__ __device__ constexpr uint32_t lz_warp_smem(uint32_t L) {
    return a16(L + 64u) + lz_pos_bytes(L) + a16(2u * LZ_NB) + a16(L / 8u + 8u) + LZ_OUT + (L > LZ_HIST ? a16(2u * LZ_NB) : 0u);
}
// the 4 bytes at p
__device__ __forceinline__ uint32_t lz_word(const uint8_t* d, uint32_t p) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(d) + (p >> 2);
    return __funnelshift_r(w[0], w[1], 8u * (p & 3u));
}
__device__ __forceinline__ uint32_t lz_hash(uint32_t word) { return ((word & 0xffffffu) * 2654435761u) >> 23; }  // 9 bits

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
    uint32_t* mark = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(end) + a16(2u * LZ_NB));
    uint8_t* out = reinterpret_cast<uint8_t*>(mark) + a16(L / 8u + 8u);
    uint16_t* oldest = reinterpret_cast<uint16_t*>(out + LZ_OUT);
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
    for (uint32_t b = lane; b < LZ_NB; b += 32) cnt[b] = 0;
    for (uint32_t i = lane; i < L / 32u + 2u; i += 32) mark[i] = 0;
    __syncwarp();

    // ---- positions with a full key (p + 2 < L), sorted by bucket; not the
    // first, which is never a source ----
    const uint32_t np = L - 2u;
    for (uint32_t p = 1u + lane; p < np; p += 32) atomicAdd(&cnt[lz_hash(lz_word(d, p))], 1u);
    __syncwarp();
    {
        constexpr uint32_t PER = LZ_NB / 32u;
        uint32_t v[PER], sum = 0;
#pragma unroll
        for (uint32_t i = 0; i < PER; ++i) {
            v[i] = cnt[lane * PER + i];
            sum += v[i];
        }
        uint32_t run = warp_incl_scan(sum) - sum;
#pragma unroll
        for (uint32_t i = 0; i < PER; ++i) {  // where each bucket starts; its end once it is filled
            end[lane * PER + i] = (uint16_t)run;
            if (aged) oldest[lane * PER + i] = (uint16_t)run;
            run += v[i];
        }
    }
    __syncwarp();
    for (uint32_t p0 = 1; p0 < np; p0 += 32) {
        const uint32_t p = p0 + lane;
        const uint32_t h = p < np ? lz_hash(lz_word(d, p)) : LZ_NB + lane;
        const uint32_t peers = __match_any_sync(GD_FULL_MASK, h);
        uint32_t at = 0;
        if (p < np) {
            at = end[h] + __popc(peers & lt);
            pos[at] = (uint16_t)p;
        }
        __syncwarp();
        if (p < np && (peers >> lane) == 1u) end[h] = (uint16_t)(at + 1u);  // the last of its bucket here
        __syncwarp();
    }
    // ---- mark the positions with a match: the same key 3 or more bytes back,
    // inside the history ----
    for (uint32_t x = lane; x + 1u < np; x += 32) {
        const uint32_t p = pos[x], w = lz_word(d, p), h = lz_hash(w);
        const uint32_t first = h ? end[h - 1u] : 0u, lo = p < LZ_HIST ? 0u : p - LZ_HIST + 1u;
        for (uint32_t y = x; y > first;) {
            const uint32_t c = pos[--y];
            if (c < lo) break;
            if (c + LZ_MINM <= p && ((lz_word(d, c) ^ w) & 0xffffffu) == 0) {
                atomicOr(&mark[p >> 5], 1u << (p & 31u));
                break;
            }
        }
    }
    __syncwarp();

    // ---- greedy token walk (warp-uniform) ----
    uint32_t* slot = reinterpret_cast<uint32_t*>(scratch + (uint64_t)col * cap);
    uint32_t tok = 0, nt = 0;        // token `lane` of the queue (literal: 1 << 16 | byte), tokens queued
    uint32_t on = 0, written = 0;    // bytes in out, words in the slot
    bool over = false;
    // write the queue's tokens, a flag byte before every 8; last: the stream
    // ends, with a reserved flag byte if its last group is full
    auto emit = [&](bool last) {
        const uint32_t lits = __ballot_sync(GD_FULL_MASK, lane < nt && (tok >> 16) != 0);
        const uint32_t size = lane < nt ? ((tok >> 16) ? 1u : 2u) + ((lane & 7u) == 0 ? 1u : 0u) : 0u;
        const uint32_t inc = warp_incl_scan(size);
        uint32_t at = on + inc - size;
        if (size) {
            if ((lane & 7u) == 0) out[at++] = (uint8_t)(lits >> lane);
            out[at] = (uint8_t)tok;
            if (!(tok >> 16)) out[at + 1] = (uint8_t)(tok >> 8);
        }
        on += __shfl_sync(GD_FULL_MASK, inc, 31);
        if (last) {
            if ((nt & 7u) == 0) {
                if (lane == 0) out[on] = 0;
                ++on;
            }
            if ((on & 3u) && (on & 3u) + lane < 4u) out[on + lane] = 0;
        }
        nt = 0;
        __syncwarp();
        if (on < LZ_OUT / 2u && !last) return;
        const uint32_t nw = last ? (on + 3u) >> 2 : on >> 2;
        over = over || 4u * (written + nw) > cap;
        if (!over)
            for (uint32_t w = lane; w < nw; w += 32) slot[written + w] = reinterpret_cast<const uint32_t*>(out)[w];
        if (last) return;
        written += nw;
        on &= 3u;
        uint8_t keep = 0;
        if (lane < on) keep = out[4u * nw + lane];
        __syncwarp();
        if (lane < on) out[lane] = keep;
        __syncwarp();
    };
    for (uint32_t cur = 0; cur < L;) {
        // literals up to the next marked position
        uint32_t m = mark[cur >> 5] >> (cur & 31u);
        uint32_t lit = m ? (uint32_t)__ffs(m) - 1u : min(32u - (cur & 31u), L - cur);
        while (lit) {
            const uint32_t k = min(lit, 32u - nt);
            if (lane - nt < k) tok = 0x10000u | d[cur + lane - nt];
            nt += k;
            cur += k;
            lit -= k;
            if (nt == 32) emit(false);
        }
        if (!m) continue;
        // the longest match here
        const uint32_t w = lz_word(d, cur), b = lz_hash(w), bend = end[b];
        uint32_t idx = b ? end[b - 1u] : 0u;
        if (aged) {
            idx = oldest[b];
            const uint32_t lo = cur < LZ_HIST ? 0u : cur - LZ_HIST + 1u;
            while (idx < bend && pos[idx] < lo) ++idx;
            __syncwarp();
            if (lane == 0) oldest[b] = (uint16_t)idx;
        }
        const uint32_t most = min(L - cur, LZ_MAXM), w4 = lz_word(d, cur + 4u);
        uint32_t best_len = 0, best_pos = 0;
        for (uint32_t base = idx; base < bend; base += 32) {
            const uint32_t p = base + lane < bend ? pos[base + lane] : 0xffffu;
            const bool valid = p + LZ_MINM <= cur;
            uint32_t f = 0;
            if (valid) {
                const uint32_t x = lz_word(d, p) ^ w;
                if ((x & 0xffffffu) == 0) {
                    const uint32_t lim = min(cur - p, most);
                    f = 3;
                    if (x == 0) {
                        const uint32_t y4 = lz_word(d, p + 4u) ^ w4;
                        f = y4 ? 4u + ((uint32_t)(__ffs(y4) - 1) >> 3) : 8u;
                        if (!y4)
                            for (; f < lim; f += 4) {
                                const uint32_t y = lz_word(d, p + f) ^ lz_word(d, cur + f);
                                if (y) {
                                    f += (uint32_t)(__ffs(y) - 1) >> 3;
                                    break;
                                }
                            }
                        f = min(f, lim);
                    }
                }
            }
            const uint32_t best = __reduce_max_sync(GD_FULL_MASK, f ? (f << 6) | (63u - lane) : 0u);
            const uint32_t from = __shfl_sync(GD_FULL_MASK, p, 63 - (int)(best & 63u));
            if ((best >> 6) > best_len) {
                best_len = best >> 6;
                best_pos = from;
            }
            if (best_len >= LZ_MAXM || __any_sync(GD_FULL_MASK, !valid)) break;
        }
        if (lane == nt) tok = ((cur - best_pos) << 5) | (best_len - LZ_MINM);
        ++nt;
        cur += best_len;
        if (nt == 32) emit(false);
    }
    emit(true);
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
    auto kern = elem_bytes == 4 ? rlev1_encode_kernel<uint32_t> : rlev1_encode_kernel<uint64_t>;
    kern<<<(uint32_t)((nc * 32u + V1_WPB - 1) / V1_WPB), V1_WPB * 32, 0, s>>>(d_in, n_bytes, nc * 32u, chunk_size, wil,
                                                                              d_scratch, (uint32_t)cap, d_col_len);
    lane_sizes_kernel<<<(uint32_t)((nc + 3) / 4), 128, 0, s>>>((uint32_t)nc, d_col_len, d_blk_off + 1, d_status);
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
    rlev2_encode_kernel<<<(uint32_t)((nc * 32u + V2_WPB - 1) / V2_WPB), V2_WPB * 32, 0, s>>>(
        d_in, n_bytes, nc * 32u, chunk_size, read_unit, d_scratch, (uint32_t)cap, d_col_len);
    lane_sizes_kernel<<<(uint32_t)((nc + 3) / 4), 128, 0, s>>>((uint32_t)nc, d_col_len, d_blk_off + 1, d_status);
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
    cudaFuncSetAttribute(lzss_column_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LZ_WPB * wsm);
    const uint32_t ncol = (uint32_t)(nc * 32u);
    lzss_column_kernel<<<(ncol + LZ_WPB - 1) / LZ_WPB, LZ_WPB * 32, LZ_WPB * wsm, s>>>(
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
