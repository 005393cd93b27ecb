// One stream through the block inflate decoder (inflate_block.cuh).
#include "cuda_runtime.h"

#include "inflate_block.cuh"

using namespace gd::inflb;

template <class S>
static int go(const uint8_t* src, uint32_t clen, uint8_t* dst, uint32_t olen, int hdr, uint32_t kind, uint32_t* written) {
    static S smem;
    memset((void*)&smem, 0xA5, sizeof smem);
    uint32_t err = 0;
    const bool ok = simt::run(S::NT, 0, 1, simt::schedule(S::NT, kind), [&] {
        uint32_t w = 0;
        const uint32_t e = stream_block(src, clen, dst, olen, hdr, smem, &w);
        if (threadIdx.x == 0) {
            err = e;
            *written = w;
        }
    });
    return ok ? (int)err : -1;
}

// A status, or -1 if the block hangs.  shape: 1 - 4 as GD_TUNE_INFLATE_VARIANT,
// 5 the batch decoder's blocks of four warps.
extern "C" int inflate(int shape, const uint8_t* src, uint32_t clen, uint8_t* dst, uint32_t olen, int hdr, uint32_t kind,
                       uint32_t* written) {
    switch (shape) {
        case 1: return go<Smem<16, 65536, 8192, 32608>>(src, clen, dst, olen, hdr, kind, written);
        case 2: return go<Smem<8, 32768, 4096, 16224>>(src, clen, dst, olen, hdr, kind, written);
        case 3: return go<Smem<8, 32768, 2048, 8032>>(src, clen, dst, olen, hdr, kind, written);
        case 4: return go<Smem<8, 16384, 2048, 8032>>(src, clen, dst, olen, hdr, kind, written);
        default: return go<Smem<4, 16384, 2048, 8032>>(src, clen, dst, olen, hdr, kind, written);
    }
}

extern "C" uint64_t barriers() { return simt::barriers; }

// A Writer at position `start` puts n bytes, byte i of them src[i], to dst:
// through the window, or as stored bytes.
extern "C" int write_at(uint32_t start, const uint8_t* src, uint32_t n, uint8_t* dst, int stored, uint32_t kind) {
    using S = Smem<8, 16384, 2048, 8032>;
    static S smem;
    const bool ok = simt::run(S::NT, 0, 1, simt::schedule(S::NT, kind), [&] {
        Writer<S> w(smem, dst);
        w.flushed = start;
        if (stored) {
            w.stored(src, n, start);
        } else {
            for (uint32_t i = threadIdx.x; i < n; i += S::NT) smem.win[(start + i) % S::WIN] = src[i];
            __syncthreads();
        }
        w.flush(start + n, true);
    });
    return ok ? 0 : 1;
}
