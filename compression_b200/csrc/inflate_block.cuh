// inflate_block.cuh -- Deflate / zlib / gzip inflate of one stream by a whole
// thread block (sm_100a), used by the plain kernels (inflate.cu) and the
// batched decoder (batch.cu).
//
// Replaces the reference's deflate::inflate / inflate_shared
// (include/zlib/zlib.h:832-962).  The time of a set of streams is mostly that
// of its longest one, and a stream decoded by one lane and copied one command
// at a time takes about 500 cycles a symbol, however idle the chip: each of
// those steps is a chain of dependent instructions.  Here both halves are
// spread over the block, in phases:
//
//   decode  -- the next NT * KSEG bits of a Huffman block are cut into a
//              segment per thread.  Every thread decodes its segment from its
//              first bit (only thread 0 knows that a symbol starts there) and
//              notes where it leaves the segment; threads whose start differs
//              from the previous thread's exit decode again from that exit,
//              until no start changes.  Huffman codes fall back into step: a
//              repeated pass ends at the first of four check points that it
//              reaches at the same bit as before.  Each pass settles one
//              thread more at least; a thread keeps the paths that it has
//              decoded, so that codes of (nearly) one length, which keep their
//              phase, are decoded once in each phase (random 7-bit values, 512
//              streams of 128 KiB: 10.2 ms, 43.6 decoding on every pass).  The
//              segments are as many as the step has room for: their symbols
//              are counted in the step before.  A prefix sum of the symbol
//              counts places a last pass that writes the symbols, one word
//              each, to shared memory.
//   place   -- a thread per symbol: a prefix sum of the lengths gives every
//              symbol its output position, literals are stored, and copies are
//              listed.
//   copy    -- 8 lanes per listed copy write the bytes whose source lies
//              before this placement's output, and for every other byte the
//              position that it copies; then a thread per byte follows those
//              positions to a byte that is there.  Deflate takes the nearest
//              match, so most copies read what one of the last few wrote (the
//              benchmark's streams: a median distance of 470 bytes, and chains
//              of 13 copies in 500 symbols): copying them in order, or in
//              rounds of those whose sources are done, is a chain of hundreds
//              of instructions each, where a followed position is one
//              shared-memory read.
// The newest WIN bytes of output stay in shared memory; most sources lie
// there, farther ones are read from the output.  The output leaves the window
// in 16-byte stores.
// Every read is bounded by the stream's compressed size and every write by its
// output size; malformed input yields GD_ERR_CORRUPT / GD_ERR_OVERRUN.
#pragma once
#include "gd_common.cuh"

namespace gd {
namespace inflb {

constexpr uint32_t LBITS = 10, DBITS = 8;  // primary lookup bits
// Bits per segment: 8 above a multiple of 64, so that threads that sit at the
// same place in their segments read 32 different shared-memory banks (256
// bits would put eight threads of a warp on each of four banks).
// Fewer where the rest of the stream does not fill the block's threads: a
// short stream's time is that of a few threads' chains (16,384 streams of 1 KiB
// of text 1.43 ms at 264 bits, 1.20 at 72).
constexpr uint32_t KSEG = 264, KSEG_MID = 136, KSEG_LOW = 72;

// Code-length code order (RFC 1951 3.2.7).
__device__ __constant__ uint8_t CLEN_ORDER[19] = {16, 17, 18, 0, 8, 7, 9, 6, 10, 5, 11, 4, 12, 3, 13, 2, 14, 1, 15};

// A canonical Huffman code: primary table, and for codes longer than the
// table's index the canonical limits.
template <uint32_t BITS, uint32_t NS>
struct Code {
    uint32_t lut[1u << BITS];  // make_entry; 0 = longer than BITS, E_NONE = no such code
    uint16_t sym[NS];          // symbols by (length, symbol)
    uint16_t lim[16];          // codes of length <= L lie below lim[L] (15 bits, first bit highest)
    int16_t delta[16];         // sym index of a code of length L = (code >> (15 - L)) + delta[L]
};

// Batch words: a literal is S_LIT | byte, a copy (distance - 1) << 9 | length.
constexpr uint32_t S_LIT = 0x80000000u;

// Shared state of a stream.  NW warps; the newest WIN output bytes (a power of
// two); NC symbols per decode step; TMAX output bytes placed at once, at most
// half the window less 160: what is farther back than the rest of the window
// is then already in the output.
template <int NW, uint32_t WIN_, uint32_t NC_, uint32_t TMAX_>
struct alignas(16) Smem {
    static constexpr uint32_t NT = 32u * NW, WIN = WIN_, NC = NC_;
    static constexpr uint32_t IN_BYTES = (NT * KSEG / 8u + 64u) & ~15u;  // a step's bits, and what a symbol at its end reads
    static constexpr uint32_t NSUB = 4u * NT;                            // symbols placed at once
    static constexpr uint32_t TMAX = TMAX_;
    static constexpr uint32_t BIG = 512;
    uint8_t win[WIN];
    union {
        uint32_t in[IN_BYTES / 4u];         // decode: the step's input
        uint16_t from[(TMAX + 15u) & ~7u];  // copy: the place that each byte copies; its own: the byte is there
    };
    uint32_t sym[NC];
    union {
        uint32_t cp[4][NT];  // decode: check points, bit of the segment | symbols << 16
        struct {
            uint16_t o[NSUB], e[NSUB], d[NSUB];  // copies: places of start and end, distance - 1
            uint16_t big[TMAX / BIG + 1];        // those of BIG bytes and more
        } c;
    };
    Code<LBITS, 288> lit;
    Code<DBITS, 32> dist;
    uint32_t exits[NT];
    uint32_t red[NW + 1];       // scans
    uint32_t evw[NW];
    uint32_t use_n, use_bit, use_ev;      // of the last thread taken from a step
    uint32_t take, take_T, take_c, bad, n_big;  // of a placement
    alignas(4) uint8_t lens[320];  // code lengths of a block
};

// Lookup-table entries carry what the decoder needs next:
//   bits 0-3 code length, 4-7 extra bits, 8-23 value, 24-31 kind.
// Table kinds: TK_PLAIN (code-length code: value = symbol; bits 0-3 count the
// bits of a repeat too, 4-7 the code's alone), TK_LIT
// (literal/length: E_LIT value = byte, E_LEN value = length base, E_EOB,
// E_BAD), TK_DIST (E_DIST value = distance base, E_BAD).  No entry of a real
// code is 0.
enum : uint32_t { TK_PLAIN = 0, TK_LIT = 1, TK_DIST = 2 };
enum : uint32_t { E_LIT = 0, E_LEN = 1, E_EOB = 2, E_DIST = 3, E_BAD = 4 };
constexpr uint32_t E_NONE = (E_BAD << 24) | 1u;  // no such code: a speculative thread moves on by one bit

// The length and distance bases and extra bits of RFC 1951 3.2.5 follow from
// the symbol: after the first 8 lengths (4 distances) every 4 (2) symbols
// share a number of extra bits, one more than the group before.
__device__ __forceinline__ uint32_t make_entry(uint32_t tk, uint32_t sym, uint32_t L) {
    uint32_t kind = E_LIT, value = sym, extra = 0;
    if (tk == TK_LIT && sym >= 256) {
        const uint32_t s = sym - 257u;
        if (sym == 256) {
            kind = E_EOB;
        } else if (sym > 285) {
            kind = E_BAD;
        } else {
            kind = E_LEN;
            extra = s < 8u || s == 28u ? 0u : (s >> 2) - 1u;
            value = s == 28u ? 258u : s < 8u ? s + 3u : ((4u + (s & 3u)) << extra) + 3u;
        }
    } else if (tk == TK_PLAIN) {
        extra = L;
        L += sym == 16u ? 2u : sym == 17u ? 3u : sym == 18u ? 7u : 0u;
    } else if (tk == TK_DIST) {
        kind = sym > 29 ? E_BAD : E_DIST;
        extra = sym < 4u ? 0u : ((sym >> 1) - 1u) & 15u;
        value = sym < 4u ? sym + 1u : ((2u + (sym & 1u)) << extra) + 1u;
    }
    return L | (extra << 4) | (value << 8) | (kind << 24);
}

// Entry of a code that the primary table does not hold (lo: the stream's next
// bits, first bit lowest), from the canonical limits; E_NONE if there is none.
template <uint32_t BITS, uint32_t NS>
__device__ __forceinline__ uint32_t long_code(const Code<BITS, NS>& h, uint32_t lo, uint32_t tk) {
    const uint32_t c = __brev(lo) >> 17;  // the next 15 bits, first bit highest
    uint32_t L = BITS + 1;
#pragma unroll
    for (uint32_t i = BITS + 1; i < 16; ++i) L += c >= h.lim[i] ? 1u : 0u;
    if (L > 15) return E_NONE;
    return make_entry(tk, h.sym[(int32_t)(c >> (15 - L)) + h.delta[L]], L);
}

// Build `h` from code lengths lens[0..n) for table kind tk: the warps count
// the lengths of 32 symbols each (tab: 16 words for every 32 symbols), warp 0
// finds the canonical limits, the warps sort their symbols by length (stable),
// then every table index finds its own code.  Returns false (on every thread)
// for an over-subscribed code.  Called by the whole block (NW warps).
template <int NW, uint32_t BITS, uint32_t NS>
static __device__ bool build_code(Code<BITS, NS>& h, const uint8_t* lens, uint32_t n, uint32_t* tab, uint32_t tk) {
    const uint32_t lane = lane_id(), wid = threadIdx.x >> 5, groups = (n + 31u) / 32u;
    for (uint32_t i = threadIdx.x; i < 16u * groups; i += 32u * NW) tab[i] = 0;
    __syncthreads();
    for (uint32_t g = wid; g < groups; g += NW) {
        const uint32_t i = 32u * g + lane, L = i < n ? lens[i] : 0u;
        const uint32_t peers = __match_any_sync(GD_FULL_MASK, L);
        if ((peers & ((1u << lane) - 1u)) == 0) tab[16u * g + L] = __popc(peers);
    }
    __syncthreads();
    bool ok = true;
    if (wid == 0) {
        // lane L: codes of length L, and where the next length's start
        const bool length = lane >= 1u && lane < 16u;
        uint32_t k = 0;
        for (uint32_t g = 0; g < groups; ++g) k += length ? tab[16u * g + lane] : 0u;
        const uint32_t share = length ? k << (15u - lane) : 0u, lim = warp_incl_scan(share);
        uint32_t idx = warp_incl_scan(k) - k;
        if (length) {
            ok = lim <= 32768u;
            h.lim[lane] = (uint16_t)min(lim, 32768u);
            h.delta[lane] = (int16_t)((int32_t)idx - (int32_t)((lim - share) >> (15u - lane)));
            for (uint32_t g = 0; g < groups; ++g) {
                const uint32_t c = tab[16u * g + lane];
                tab[16u * g + lane] = idx;
                idx += c;
            }
        }
    }
    if (__syncthreads_or(!ok)) return false;
    for (uint32_t g = wid; g < groups; g += NW) {
        const uint32_t i = 32u * g + lane, L = i < n ? lens[i] : 0u;
        const uint32_t peers = __match_any_sync(GD_FULL_MASK, L);
        if (L) h.sym[tab[16u * g + L] + __popc(peers & ((1u << lane) - 1u))] = (uint16_t)i;
    }
    __syncthreads();
    uint32_t lim[BITS + 1];
#pragma unroll
    for (uint32_t l = 1; l <= BITS; ++l) lim[l] = h.lim[l];
    const uint32_t end = h.lim[15];
    for (uint32_t x = threadIdx.x; x < (1u << BITS); x += blockDim.x) {
        // deflate sends codes first bit highest into a lowest-first stream
        const uint32_t c = (__brev(x) >> (32u - BITS)) << (15u - BITS);
        uint32_t L = 1;
#pragma unroll
        for (uint32_t l = 1; l <= BITS; ++l) L += c >= lim[l] ? 1u : 0u;
        uint32_t e = c < end ? 0u : E_NONE;
        if (L <= BITS) e = make_entry(tk, h.sym[(int32_t)(c >> (15u - L)) + h.delta[L]], L);
        h.lut[x] = e;
    }
    __syncthreads();
    return true;
}

// One symbol at bit `pos` of the staged input.  Returns its kind (E_LIT,
// E_LEN, E_EOB, E_BAD) and moves pos past it; word: its batch word.
template <class SmemT>
__device__ __forceinline__ uint32_t symbol_at(const SmemT& S, uint32_t& pos, uint32_t& word) {
    const uint32_t* w = S.in + (pos >> 5);
    const uint32_t a1 = w[1], lo = __funnelshift_r(w[0], a1, pos);
    uint32_t e = S.lit.lut[lo & ((1u << LBITS) - 1u)];
    if (e == 0) e = long_code(S.lit, lo, TK_LIT);
    uint32_t adv = e & 15u;
    word = S_LIT | ((e >> 8) & 0xffu);
    uint32_t kind = e >> 24;
    if (kind == E_LEN) {
        const uint32_t ex = (e >> 4) & 15u;
        const uint32_t len = ((e >> 8) & 0xffffu) + ((lo >> adv) & ((1u << ex) - 1u));
        adv += ex;  // at most 15 + 5
        const uint32_t lo2 = __funnelshift_r(lo, __funnelshift_r(a1, w[2], pos), adv);
        uint32_t ed = S.dist.lut[lo2 & ((1u << DBITS) - 1u)];
        if (ed == 0) ed = long_code(S.dist, lo2, TK_DIST);
        const uint32_t Ld = ed & 15u, exd = (ed >> 4) & 15u;
        const uint32_t dist = ((ed >> 8) & 0xffffu) + ((lo2 >> Ld) & ((1u << exd) - 1u));
        adv += Ld + exd;
        word = ((dist - 1u) << 9) | len;
        if ((ed >> 24) != E_DIST) kind = E_BAD;
    }
    pos += adv;
    return kind;
}

// Exclusive sum of v over the block (NW warps); *total gets the sum.
template <int NW>
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* red, uint32_t* total) {
    const uint32_t inc = warp_incl_scan(v), wid = threadIdx.x >> 5;
    if (lane_id() == 31) red[wid] = inc;
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        const uint32_t x = red[w];
        before += (uint32_t)w < wid ? x : 0u;
        all += x;
    }
    *total = all;
    return before + inc - v;
}

// The output side of a stream.  Positions count from the 16-byte-aligned
// address below dst, so that window words and 16-byte vectors line up with the
// output's.  They are taken modulo 2^32 (a stream of 2^32 - 1 bytes may end
// beyond it), so they are told apart by their differences, and the output is
// addressed from `flushed`.  Bytes from there on are in the window only.
template <class SmemT>
struct Writer {
    static constexpr uint32_t NT = SmemT::NT, WIN = SmemT::WIN, M = WIN - 1, NW = NT / 32;
    static_assert((WIN & (WIN - 1)) == 0 && 2 * SmemT::TMAX + 274 <= WIN, "window");
    static_assert(SmemT::TMAX >= 258 && SmemT::TMAX % 8 == 0, "a placement holds a symbol");
    SmemT& S;
    uint8_t* at;       // where position `flushed` goes
    uint32_t base;     // position of dst
    uint32_t flushed;

    __device__ __forceinline__ Writer(SmemT& s, uint8_t* dst) : S(s) {
        base = (uint32_t)(reinterpret_cast<uintptr_t>(dst) & 15u);
        at = dst;
        flushed = base;
    }
    __device__ __forceinline__ void advance(uint32_t n) {
        at += n;
        flushed += n;
    }
    // Write the whole vectors before `to` out; last: also the bytes after them.
    __device__ __forceinline__ void flush(uint32_t to, bool last) {
        const uint32_t tid = threadIdx.x;
        if (flushed & 15u) {  // the stream's first vector, shared with what precedes dst
            const uint32_t v = 16u - (flushed & 15u), m = min(to - flushed, v);
            if (!last && m < v) return;
            if (tid < m) at[tid] = S.win[(flushed + tid) & M];
            advance(m);
        }
        const uint32_t n = to - flushed;
        for (uint32_t k = 16u * tid; k + 16u <= n; k += 16u * NT)
            *reinterpret_cast<uint4*>(at + k) = *reinterpret_cast<const uint4*>(S.win + ((flushed + k) & M));
        advance(n & ~15u);
        if (last && tid < (n & 15u)) at[tid] = S.win[(flushed + tid) & M];
    }
    // m stored bytes from s to position p.  Whole vectors go straight to the
    // output and the window, four in flight a thread.
    __device__ __forceinline__ void stored(const uint8_t* __restrict__ s, uint32_t m, uint32_t p) {
        const uint32_t tid = threadIdx.x;
        // whole vectors of the output: [v0, v1) of the m bytes
        const uint32_t v0 = min(m, (0u - p) & 15u), r = (p + m) & 15u, v1 = m >= v0 + r ? m - r : v0;
        if (tid < v0) S.win[(p + tid) & M] = s[tid];
        __syncthreads();
        flush(p + v0, false);
        // a block of nearly WIN bytes or more also writes the window's place
        // of the vector that flush reads
        __syncthreads();
        const uint8_t* sv = s + v0;
        const uint32_t sh = (uint32_t)(reinterpret_cast<uintptr_t>(sv) & 3u) * 8u;
        const uint32_t* sw = reinterpret_cast<const uint32_t*>(sv - (sh >> 3));
        const uint32_t n = v1 - v0;
#pragma unroll 4
        for (uint32_t k = 16u * tid; k < n; k += 16u * NT) {
            const uint32_t* q = sw + (k >> 2);
            uint32_t w[5];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = __ldg(q + i);
            w[4] = sh ? __ldg(q + 4) : 0u;
            const uint4 x = make_uint4(__funnelshift_r(w[0], w[1], sh), __funnelshift_r(w[1], w[2], sh),
                                       __funnelshift_r(w[2], w[3], sh), __funnelshift_r(w[3], w[4], sh));
            *reinterpret_cast<uint4*>(at + k) = x;
            if (k + WIN >= n) *reinterpret_cast<uint4*>(S.win + ((p + v0 + k) & M)) = x;  // the newest WIN bytes
        }
        advance(n);
        __syncthreads();  // the tail's window bytes may replace ones the loop stored
        if (v1 + tid < m) S.win[(p + v1 + tid) & M] = s[v1 + tid];
        __syncthreads();
    }
    // Bytes [o, e) after position q0 (a multiple of 4) from d bytes before them
    // (e - o <= d) with W lanes, the caller being lane `sub`.  word(x): the
    // aligned source word at position x.
    template <class Word>
    __device__ __forceinline__ void copy_words(uint32_t q0, uint32_t o, uint32_t e, uint32_t d, uint32_t sub, uint32_t W,
                                               Word word) {
        const uint32_t o4 = (o + 3u) & ~3u, e4 = e & ~3u;
        // up to 3 bytes before the first whole word and after the last: lanes 0-3 and 4-7
        const uint32_t x = sub < 4u ? o + sub : max(e4, o4) + sub - 4u;
        const bool edge = sub < 4u ? x < min(o4, e) : sub < 8u && x < e;
        uint32_t v = 0;
        if (edge) v = word((q0 + x - d) & ~3u) >> (8u * ((x - d) & 3u));
        const uint32_t sh = ((0u - d) & 3u) * 8u;
        for (uint32_t q = o4 + 4u * sub; q < e4; q += 8u * W) {
            const uint32_t s0 = (q0 + q - d) & ~3u, s1 = s0 + 4u * W;
            const bool two = q + 4u * W < e4;
            const uint32_t a0 = word(s0), b0 = word(s0 + 4u);
            uint32_t a1 = 0, b1 = 0;
            if (two) {
                a1 = word(s1);
                b1 = word(s1 + 4u);
            }
            *reinterpret_cast<uint32_t*>(S.win + ((q0 + q) & M)) = __funnelshift_r(a0, b0, sh);
            if (two) *reinterpret_cast<uint32_t*>(S.win + ((q0 + q + 4u * W) & M)) = __funnelshift_r(a1, b1, sh);
        }
        if (edge) S.win[(q0 + x) & M] = (uint8_t)v;
    }
    // from[k] = k - d for k in [lo, hi), by W lanes or threads
    __device__ __forceinline__ void fill(uint32_t lo, uint32_t hi, uint32_t d, uint32_t sub, uint32_t W) {
        const uint32_t lo4 = (lo + 3u) & ~3u, hi4 = hi & ~3u;
        const uint32_t x = sub < 4u ? lo + sub : max(hi4, lo4) + sub - 4u;
        if (sub < 4u ? x < min(lo4, hi) : sub < 8u && x < hi) S.from[x] = (uint16_t)(x - d);
        for (uint32_t k = lo4 + 4u * sub; k < hi4; k += 4u * W) {
            const uint32_t v = ((k - d) & 0xffffu) * 0x10001u + 0x10000u;  // k >= d: no carry between the halves
            *reinterpret_cast<uint2*>(S.from + k) = make_uint2(v, v + 0x20002u);
        }
    }
    // Listed copy c by W lanes or threads, the caller being number `sub`: the
    // bytes with a source before the placement, and the places that the others
    // copy (an overlapping copy repeats the d bytes before it).  The placement
    // starts at place z of position q0.
    __device__ __forceinline__ void copy(uint32_t c, uint32_t sub, uint32_t W, uint32_t q0, uint32_t z, uint32_t T) {
        const uint32_t o = S.c.o[c], e = S.c.e[c], d = S.c.d[c] + 1u, in0 = max(o, d + z);
        if (o < in0) {
            const uint32_t x = min(e, in0);
            if (d + T <= WIN + o - z) {
                copy_words(q0, o, x, d, sub, W,
                           [&](uint32_t q) { return *reinterpret_cast<const uint32_t*>(S.win + (q & M)); });
            } else {
                // the placement's later bytes may have taken the source's
                // place in the window: read the output
                copy_words(q0, o, x, d, sub, W, [&](uint32_t q) {
                    return *reinterpret_cast<const uint32_t*>(at + (int32_t)(q - flushed));
                });
            }
        }
        if (in0 < e) {
            if (e - o <= d) {
                fill(in0, e, d, sub, W);
            } else {
                for (uint32_t k = in0 + sub; k < e; k += W) {
                    // place o - d + m, or, where that lies before the
                    // placement, the copy's own first such byte
                    const uint32_t m = (k - o) % d;
                    S.from[k] = (uint16_t)(o + m >= d + z ? o + m - d : o + m);
                }
            }
        }
    }
    // Symbols S.sym[0..n) at output byte opos, which moves past them; olen:
    // the output's size.  Returns a status (the same on every thread).
    __device__ __forceinline__ uint32_t symbols(uint32_t n, uint32_t& opos, uint32_t olen) {
        const uint32_t tid = threadIdx.x, wid = tid >> 5, lane = tid & 31u;
        for (uint32_t g = 0; g < n;) {
            // places count from the 8-byte-aligned position q0, so that their
            // words line up with the window's
            const uint32_t p = opos + base, z = p & 7u, q0 = p - z, room = olen - opos;
            // ---- place: four symbols a thread ----
            // consecutive copies of one distance are one longer copy (a match
            // of more than 258 bytes, a run): a shorter chain of rounds
            const uint32_t m = min(n - g, SmemT::NSUB), j0 = 4u * tid;
            uint32_t e[6];
#pragma unroll
            for (uint32_t i = 0; i < 6; ++i) {
                const uint32_t j = j0 + i - 1u;  // e[0], e[5]: the neighbours'
                e[i] = j < m ? S.sym[g + j] : S_LIT;
            }
            uint32_t off[4], run[4], sum = 0;
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                const uint32_t x = e[i + 1];
                const bool copy = !(x & S_LIT);
                off[i] = sum & 0xfffffu;
                if (copy && (e[i] >> 9) != (x >> 9)) sum += 1u << 20;
                run[i] = sum >> 20;  // copies listed up to this symbol
                sum += copy ? x & 511u : j0 + i < m ? 1u : 0u;
            }
            if (tid == 0) S.take = 0xffffffffu, S.bad = 0xffffffffu, S.n_big = 0;
            uint32_t total;
            const uint32_t ex = block_scan<NW>(sum, S.red, &total);
            const uint32_t xo = ex & 0xfffffu, xr = ex >> 20;
            // every byte is there but those that copy() points elsewhere
            for (uint32_t k = 8u * tid; k < z + min(total & 0xfffffu, SmemT::TMAX); k += 8u * NT) {
                const uint32_t v = k * 0x10001u + 0x10000u;
                *reinterpret_cast<uint4*>(S.from + k) = make_uint4(v, v + 0x20002u, v + 0x40004u, v + 0x60006u);
            }
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                const uint32_t x = e[i + 1], y = e[i + 2], j = j0 + i;
                const bool lit = (x & S_LIT) != 0;
                const uint32_t len = lit ? (j < m ? 1u : 0u) : (x & 511u);
                const uint32_t o = xo + off[i], c = xr + run[i] - 1u;
                const bool start = !lit && (e[i] >> 9) != (x >> 9);
                if (o + len > SmemT::TMAX) {
                    if (o <= SmemT::TMAX) {  // the first symbol of the next placement
                        S.take = j;
                        S.take_T = o;
                        S.take_c = start ? c : c + 1u;
                    }
                } else if (len) {
                    if (!lit && (x >> 9) >= o && (x >> 9) - o >= opos)
                        atomicMin(&S.bad, 16u * j + ST_CORRUPT);
                    else if (o + len > room)
                        atomicMin(&S.bad, 16u * j + ST_OVERRUN);
                    else if (lit)
                        S.win[(p + o) & M] = (uint8_t)x;
                    if (start) {
                        S.c.o[c] = (uint16_t)(z + o);
                        S.c.d[c] = (uint16_t)(x >> 9);
                    }
                    if (!lit && ((y >> 9) != (x >> 9) || o + len + (y & 511u) > SmemT::TMAX))
                        S.c.e[c] = (uint16_t)(z + o + len);
                }
            }
            __syncthreads();
            if (S.bad != 0xffffffffu) return S.bad & 15u;
            uint32_t take = S.take, T = total & 0xfffffu, nc = total >> 20;
            if (take == 0xffffffffu) {
                take = m;
            } else {
                T = S.take_T;
                nc = S.take_c;
            }
            // ---- copy ----
            for (uint32_t c = 4u * wid + (lane >> 3); c < nc; c += 4u * NW) {
                if ((uint32_t)(S.c.e[c] - S.c.o[c]) < SmemT::BIG)
                    copy(c, lane & 7u, 8, q0, z, T);
                else if ((lane & 7u) == 0)
                    S.c.big[atomicAdd(&S.n_big, 1u)] = (uint16_t)c;
            }
            __syncthreads();
            if (const uint32_t nb = S.n_big) {
                for (uint32_t i = 0; i < nb; ++i) copy(S.c.big[i], tid, NT, q0, z, T);
                __syncthreads();
            }
            // ---- follow the places, lowest first (a byte done shortens the chains through it) ----
            for (uint32_t k = 4u * tid; k < z + T; k += 4u * NT) {
                const uint2 v = *reinterpret_cast<const uint2*>(S.from + k);
                const uint32_t self = k * 0x10001u + 0x10000u;
                if (v.x == self && v.y == self + 0x20002u) continue;
                uint32_t f0 = v.x & 0xffffu, f1 = v.x >> 16, f2 = v.y & 0xffffu, f3 = v.y >> 16;
                for (;;) {
                    const uint32_t r0 = S.from[f0], r1 = S.from[f1], r2 = S.from[f2], r3 = S.from[f3];
                    const bool more = r0 != f0 || r1 != f1 || r2 != f2 || r3 != f3;
                    f0 = r0;
                    f1 = r1;
                    f2 = r2;
                    f3 = r3;
                    if (!more) break;
                }
                *reinterpret_cast<uint2*>(S.from + k) = make_uint2(f0 | (f1 << 16), f2 | (f3 << 16));
                // bytes of other words are read, this word alone is written;
                // a byte that is there keeps its value
                const uint32_t b0 = S.win[(q0 + f0) & M], b1 = S.win[(q0 + f1) & M], b2 = S.win[(q0 + f2) & M],
                               b3 = S.win[(q0 + f3) & M];
                *reinterpret_cast<uint32_t*>(S.win + ((q0 + k) & M)) = b0 | (b1 << 8) | (b2 << 16) | (b3 << 24);
            }
            __syncthreads();
            opos += T;
            g += take;
            flush(opos + base, false);
        }
        return ST_OK;
    }
};

// Inflate one stream with the calling block (NT threads; every thread must
// call).  src: clen compressed bytes (the 16-byte-aligned span around them
// must be readable); dst: room for olen bytes; hdr: 0 raw deflate, 1 zlib, 2
// gzip.  Returns a gd status (same on every thread); *written = bytes output.
template <class SmemT>
static __device__ __forceinline__ uint32_t stream_block(const uint8_t* __restrict__ src, uint32_t clen, uint8_t* dst,
                                                        uint32_t olen, int zlib_hdr, SmemT& S, uint32_t* written) {
    constexpr uint32_t NT = SmemT::NT, NC = SmemT::NC, NW = NT / 32;
    // Paths of a segment that are kept while a step looks for its threads'
    // starts, in S.sym, which holds no symbols yet: a path's first bit of the
    // segment, symbols << 6, bits beyond the segment << 15, the first special
    // one's index << 21 and kind << 29.
    constexpr uint32_t KEEP = NC / NT;
    // one thread's segment always fits (a symbol has at least one bit)
    static_assert(NC >= KSEG, "a step holds a segment");
    const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
    uint32_t err = ST_OK;
    // the 16-byte-aligned view of the stream: it starts at view byte sh
    const uint32_t sh = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 15u);
    const uint8_t* src_al = src - sh;
    const uint64_t span = (uint64_t)clen + sh;  // bytes of the view we may use
    const uint64_t bend = span * 8u;
    uint64_t bp = (uint64_t)sh * 8u;  // next bit of the view
    uint32_t opos = 0;                // output bytes so far

    if (zlib_hdr == 1) {
        // zlib (RFC 1950): CMF, FLG; no preset dictionary
        if (clen < 2) {
            err = ST_CORRUPT;
        } else {
            const uint32_t cmf = src[0], flg = src[1];
            if ((cmf & 15u) != 8u || ((cmf << 8) | flg) % 31u != 0 || (flg & 32u)) err = ST_CORRUPT;
            bp += 16;
        }
    } else if (zlib_hdr == 2) {
        // gzip (RFC 1952) member header, of 8 KiB at most; the 8-byte trailer is not read
        auto at = [&](uint32_t i) -> uint32_t { return i < clen && sh + i < 8192u ? src[i] : 0x100u; };
        uint32_t p = 10;
        if (at(0) != 0x1fu || at(1) != 0x8bu || at(2) != 8u || clen < 18) err = ST_CORRUPT;
        const uint32_t flg = at(3);
        if (err == ST_OK && (flg & 4u)) p += 2 + (at(p) | (at(p + 1) << 8));  // FEXTRA
        for (uint32_t f = 8; f <= 16; f += 8)                                // FNAME, FCOMMENT
            if (err == ST_OK && (flg & f)) {
                uint32_t b;
                while (p < clen && (b = at(p)) != 0) {
                    if (b > 0xffu) {
                        err = ST_CORRUPT;
                        break;
                    }
                    ++p;
                }
                ++p;
            }
        if (err == ST_OK && (flg & 2u)) p += 2;  // FHCRC
        if (err == ST_OK && p + 8 > clen) err = ST_CORRUPT;
        bp += (uint64_t)p * 8u;
    }
    // bit 0 of S.in is bit b0 of the view
    uint64_t b0 = 0;
    auto stage = [&]() {
        const uint64_t from = (bp >> 3) & ~15ull;
        const uint32_t n = (uint32_t)min((unsigned long long)(span - from), (unsigned long long)SmemT::IN_BYTES);
        __syncthreads();  // the last readers of S.in
        for (uint32_t i = 16u * tid; i < n; i += 16u * NT) {
            // whole 16-byte words; the ragged end byte by byte
            if (i + 16u <= n) {
                *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(S.in) + i) =
                    __ldg(reinterpret_cast<const uint4*>(src_al + from + i));
            } else {
                for (uint32_t k = i; k < n; ++k) reinterpret_cast<uint8_t*>(S.in)[k] = src_al[from + k];
            }
        }
        b0 = from * 8u;
        __syncthreads();
    };
    // n <= 25 bits at bp (the same on every thread); false at the end of the input
    auto get_bits = [&](uint32_t n, uint32_t& v) -> bool {
        if (bp + n > bend) return false;
        const uint32_t q = (uint32_t)(bp - b0);
        v = __funnelshift_r(S.in[q >> 5], S.in[(q >> 5) + 1], q) & ((1u << n) - 1u);
        bp += n;
        return true;
    };

    Writer<SmemT> wr(S, dst);
    uint32_t bfinal = 0;
    uint32_t lim = NT, kseg = KSEG;  // threads that decode a step's segments, and their bits
    while (err == ST_OK && !bfinal) {
        // ---- block header (every thread reads the same bits) ----
        stage();
        uint32_t btype = 0;
        if (!get_bits(1, bfinal) || !get_bits(2, btype) || btype == 3) {
            err = ST_CORRUPT;
            break;
        }
        if (btype == 0) {
            // stored block: to a byte boundary, LEN / NLEN
            bp = (bp + 7u) & ~7ull;
            uint32_t ln, nln;
            if (!get_bits(16, ln) || !get_bits(16, nln) || (ln ^ 0xffffu) != nln) {
                err = ST_CORRUPT;
                break;
            }
            if (ln > olen - opos) {
                err = ST_OVERRUN;
                break;
            }
            if (bp + 8ull * ln > bend) {
                err = ST_CORRUPT;
                break;
            }
            if (ln) wr.stored(src + ((bp >> 3) - sh), ln, opos + wr.base);
            bp += 8ull * ln;
            opos += ln;
            continue;
        }
        uint32_t nlen = 288, ndist = 30;
        if (btype == 1) {
            for (uint32_t i = tid; i < 318; i += NT)
                S.lens[i] = i < 144 ? 8 : i < 256 ? 9 : i < 280 ? 7 : i < 288 ? 8 : 5;
        } else {
            // dynamic: code-length code, then literal/length + distance lengths
            uint32_t hlit, hdist, hclen;
            if (!get_bits(5, hlit) || !get_bits(5, hdist) || !get_bits(4, hclen)) {
                err = ST_CORRUPT;
                break;
            }
            nlen = hlit + 257;
            ndist = hdist + 1;
            const uint32_t ncl = hclen + 4;
            if (nlen > 286 || ndist > 30 || bp + 3u * ncl > bend) {
                err = ST_CORRUPT;
                break;
            }
            if (tid < 19) S.lens[tid] = 0;
            __syncthreads();
            if (tid < ncl) {
                const uint32_t q = (uint32_t)(bp - b0) + 3u * tid;
                S.lens[CLEN_ORDER[tid]] = (uint8_t)(__funnelshift_r(S.in[q >> 5], S.in[(q >> 5) + 1], q) & 7u);
            }
            bp += 3u * ncl;
            __syncthreads();
            if (!build_code<NW>(S.dist, S.lens, 19, S.sym, TK_PLAIN)) {
                err = ST_CORRUPT;
                break;
            }
            // warp 0 reads the lengths, 32 codes at a time: every lane
            // follows the chain (a table lookup and a shift of the next 32 to
            // 64 bits, which stay in a register), lane k keeps code k, and the
            // repeats are then expanded together
            const uint32_t tot = nlen + ndist;
            if (wid == 0) {
                const uint32_t avail = (uint32_t)min((unsigned long long)(bend - b0), 0x40000000ull);
                uint32_t q = (uint32_t)(bp - b0), i = 0, prev = 0, bad = 0;
                uint32_t wi = (q >> 5) + 2u, have = 64u - (q & 31u), next = S.in[wi];
                uint64_t buf = (((uint64_t)S.in[wi - 1u] << 32) | S.in[wi - 2u]) >> (q & 31u);
                for (uint32_t k = lane; k < 80; k += 32) reinterpret_cast<uint32_t*>(S.lens)[k] = 0;
                __syncwarp();
                while (i < tot && !bad) {
                    uint32_t e = 0, lo = 0, qe = 0;
                    for (uint32_t k = 0; k < 32; ++k) {
                        const uint32_t x = (uint32_t)buf, ek = S.dist.lut[x & ((1u << DBITS) - 1u)], adv = ek & 15u;
                        buf >>= adv;
                        q += adv;
                        have -= adv;
                        if (have < 32u) {
                            buf |= (uint64_t)next << have;
                            have += 32u;
                            next = S.in[++wi];
                        }
                        if (k == lane) {
                            e = ek;
                            lo = x;
                            qe = q;
                        }
                    }
                    const uint32_t sym = (e >> 8) & 0xffu, L = (e >> 4) & 15u;
                    const uint32_t rep = sym < 16u ? 1u : (sym == 18u ? 11u : 3u) + ((lo >> L) & ((1u << ((e & 15u) - L)) - 1u));
                    const uint32_t end = i + warp_incl_scan(rep);
                    const uint32_t valm = __ballot_sync(GD_FULL_MASK, sym != 16u) & (GD_FULL_MASK >> (31u - lane));
                    const uint32_t last = __shfl_sync(GD_FULL_MASK, sym < 16u ? sym : 0u, valm ? 31 - __clz(valm) : 0);
                    const uint32_t v = valm ? last : prev;
                    // codes up to the first that reaches the total
                    const uint32_t m = __ballot_sync(GD_FULL_MASK, end >= tot);
                    const uint32_t fin = m ? (uint32_t)__ffs(m) - 1u : 31u;
                    const bool mine = lane <= fin;
                    bad = __any_sync(GD_FULL_MASK, mine && ((e >> 24) == E_BAD || qe > avail || end > tot ||
                                                            (sym == 16u && end == rep)));
                    if (mine && !bad && v)  // six at most: longer repeats are of 0
                        for (uint32_t k = end - rep; k < end; ++k) S.lens[k] = (uint8_t)v;
                    i = __shfl_sync(GD_FULL_MASK, end, fin);
                    prev = __shfl_sync(GD_FULL_MASK, v, fin);
                    if (m) q = __shfl_sync(GD_FULL_MASK, qe, fin);
                }
                if (lane == 0) {
                    S.use_ev = bad;
                    S.use_bit = q;
                }
            }
            __syncthreads();
            if (S.use_ev) {
                err = ST_CORRUPT;
                break;
            }
            bp = b0 + S.use_bit;
        }
        __syncthreads();
        if (S.lens[256] == 0 ||  // no end-of-block code
            !build_code<NW>(S.lit, S.lens, nlen, S.sym, TK_LIT) ||
            !build_code<NW>(S.dist, S.lens + nlen, ndist, S.sym, TK_DIST)) {
            err = ST_CORRUPT;
            break;
        }

        // ---- the block's symbols, a step of NT segments at a time ----
        for (bool in_block = true; in_block && err == ST_OK;) {
            if (bp >= bend) {
                err = ST_CORRUPT;  // no end-of-block symbol
                break;
            }
            stage();
            // positions below count bits from b0
            const uint32_t p0 = (uint32_t)(bp - b0);
            const uint32_t avail = (uint32_t)min((unsigned long long)(bend - b0), 0x40000000ull);
            if (avail - p0 <= NT * KSEG_MID && kseg != KSEG_LOW) {
                kseg = avail - p0 <= NT * KSEG_LOW ? KSEG_LOW : KSEG_MID;
                lim = NT;
            }
            const uint32_t seg = p0 + tid * kseg;
            uint32_t s = min(seg, avail), pos = s;  // where this thread starts, and leaves its segment
            uint32_t n = 0;                         // symbols
            uint32_t ev = 0, evn = 0, evs = 0;      // first special one (E_EOB / E_BAD): index, start
            bool run = tid < lim, cps = false;      // cps: S.cp is of the path that pos, n and ev are of
            uint32_t kept = 0;                      // paths kept in S.sym
            // the path from s, if it is one of those kept
            auto recall = [&]() -> bool {
                for (uint32_t j = 0; j < min(kept, KEEP); ++j) {
                    const uint32_t k = S.sym[j * NT + tid];
                    if ((k & 63u) != s - seg) continue;
                    n = (k >> 6) & 511u;
                    pos = seg + kseg + ((k >> 15) & 63u);
                    evn = (k >> 21) & 511u;
                    ev = k >> 30 << 1;
                    cps = false;
                    return true;
                }
                return false;
            };
            for (bool first = true;; first = false) {
                const bool known = run && kept > 1u && recall();
                if (run && !known) {
                    const uint32_t xpos = pos, xn = n, xev = ev, xevn = evn, xevs = evs;
                    pos = s;
                    n = ev = 0;
                    for (uint32_t q = 0; q < 4; ++q) {
                        const uint32_t to = min(seg + (q + 1) * (kseg / 4u), avail);
                        uint32_t at = pos;
                        while (pos < to) {
                            uint32_t word;
                            at = pos;
                            const uint32_t kind = symbol_at(S, pos, word);
                            if (kind > E_LEN && ev == 0) {
                                ev = kind;
                                evn = n;
                                evs = at;
                            }
                            ++n;
                        }
                        if (pos > avail) {  // the input ends inside the last symbol
                            if (ev == 0 || evs == at) {
                                ev = E_BAD;
                                evn = n - 1u;
                                evs = at;
                            }
                            pos = avail;
                        }
                        const uint32_t here = (pos - seg) & 0xffffu;
                        if (cps && ev == 0) {
                            const uint32_t c = S.cp[q][tid];
                            if ((c & 0xffffu) == here && !(xev && xevs < pos)) {
                                // as before from here on
                                const uint32_t dn = n - (c >> 16);
                                for (; q < 4; ++q) S.cp[q][tid] += dn << 16;
                                n = xn + dn;
                                pos = xpos;
                                ev = xev;
                                evn = xevn + dn;
                                evs = xevs;
                                break;
                            }
                        }
                        S.cp[q][tid] = here | (n << 16);
                    }
                    cps = true;
                    if (s - seg < 64u && pos >= seg + kseg) {
                        S.sym[(kept % KEEP) * NT + tid] =
                            (s - seg) | (n << 6) | ((pos - seg - kseg) << 15) | (ev ? evn << 21 | ev << 29 : 0u);
                        ++kept;
                    }
                }
                if (__any_sync(GD_FULL_MASK, known) && __all_sync(GD_FULL_MASK, known == run)) {
                    // nothing new in this warp: on through the paths it knows
                    // (sooner, fewer threads would have a new start to decode)
                    for (bool moved = true; __any_sync(GD_FULL_MASK, moved);) {
                        const uint32_t from = s, ns = __shfl_up_sync(GD_FULL_MASK, pos, 1);
                        moved = false;
                        if (lane && tid < lim && ns != s) {
                            s = ns;
                            moved = recall();
                            if (!moved) s = from;
                        }
                    }
                }
                S.exits[tid] = pos;
                if (first && wid == 0) {
                    const uint32_t sum = __reduce_add_sync(GD_FULL_MASK, n);
                    if (lane == 0) S.take = sum;
                }
                __syncthreads();
                // the first step's guess, from the first 32 segments
                if (first && lim == NT) lim = min(36u * NC / max(S.take, 1u) + 4u, NT);
                const uint32_t ns = tid ? S.exits[tid - 1] : s;
                run = tid < lim && ns != s;
                s = ns;
                if (!__syncthreads_or(run)) break;
            }
            // threads up to the first special symbol, as many as the step holds
            if (ev) n = evn;
            if (tid >= lim) n = ev = 0;
            uint32_t total;
            const uint32_t inc = block_scan<NW>(n, S.red, &total) + n;
            const uint32_t evm = __ballot_sync(GD_FULL_MASK, ev != 0);
            const uint32_t fitm = __ballot_sync(GD_FULL_MASK, inc <= NC);  // inc ascends
            if (lane == 0) {
                S.evw[wid] = evm;
                S.exits[wid] = __popc(fitm);
            }
            __syncthreads();
            uint32_t use = 0, evt = NT;
#pragma unroll
            for (uint32_t w = 0; w < NW; ++w) {
                use += S.exits[w];
                const uint32_t m = S.evw[w];
                if (m && evt == NT) evt = 32u * w + __ffs(m) - 1u;
            }
            use = min(use, lim);
            // what did not fit was decoded for nothing: an eighth more than
            // fits is enough
            if (use == lim) lim = min(2u * lim, NT);
            else if (use <= evt) lim = min(use + use / 8u + 4u, NT);
            use = min(use, evt + 1u);
            if (tid < use) {
                uint32_t q = s;
                for (uint32_t at = inc - n; at < inc; ++at) {
                    uint32_t word;
                    symbol_at(S, q, word);
                    S.sym[at] = word;
                }
                if (tid == use - 1) {
                    uint32_t word;
                    if (ev) symbol_at(S, q, word);
                    S.use_n = inc;
                    S.use_bit = q;
                    S.use_ev = ev;
                }
            }
            __syncthreads();
            const uint32_t tot = S.use_n, uev = S.use_ev;
            bp = b0 + S.use_bit;
            err = wr.symbols(tot, opos, olen);
            if (err == ST_OK && uev == E_BAD) err = ST_CORRUPT;
            in_block = uev == 0;
        }
    }
    __syncthreads();
    if (err == ST_OK) wr.flush(opos + wr.base, true);
    __syncthreads();  // S may be used for another stream
    *written = opos;
    return err;
}

}  // namespace inflb
}  // namespace gd
