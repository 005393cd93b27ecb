// cuda_runtime.h -- stand-in for CUDA's header that runs one thread block of
// the library's device code on the host, under a schedule that the test picks.
// Test tooling only: put this directory before CUDA's on the include path.
//
// Every CUDA thread is a fiber of one host thread.  A fiber runs until it waits
// (a block barrier, a warp collective, which all 32 lanes must reach) or calls
// an atomic; then the runnable fiber of the highest priority goes on.  So a
// thread of low priority is as late as the code allows: what it reads after a
// barrier, everybody else has had the time to change up to the next one.  If no
// fiber can run, the kernel would hang: run() returns false.
#pragma once
#undef _FORTIFY_SOURCE  // its longjmp takes a switch of stacks for an error
#include <setjmp.h>
#include <ucontext.h>

#include <algorithm>
#include <bit>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <random>
#include <type_traits>
#include <vector>

#define __host__
#define __device__
#define __global__
#define __constant__
#define __forceinline__ inline
#define __noinline__
#define __launch_bounds__(...)
#define __align__(n) __attribute__((aligned(n)))
#define __shared__ thread_local  // one host thread: shared by the fibers, and `extern` may stand before it

struct uint2 {
    uint32_t x, y;
};
struct alignas(16) uint4 {
    uint32_t x, y, z, w;
};
inline uint2 make_uint2(uint32_t x, uint32_t y) { return {x, y}; }
inline uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }

struct simt_dim {
    uint32_t x = 0, y = 0, z = 0;
};
inline simt_dim threadIdx, blockIdx, blockDim, gridDim;

namespace simt {

enum State : uint8_t { RUN, AT_BLOCK, AT_WARP, DONE };
struct Fiber {
    ucontext_t ctx;      // to start
    jmp_buf at;          // to go on
    bool begun = false;
    State state = RUN;
};
struct Warp {
    uint64_t in[32], out[32];
    uint32_t at = 0;     // lanes that wait,
    int op = 0;          // at this collective
};
struct Block {
    std::vector<Fiber> f;
    std::vector<Warp> w;
    std::function<void()> body;
    ucontext_t end;
    jmp_buf main;
    uint32_t cur = 0, live = 0, at = 0;   // the fiber that runs; those not done; those at the block barrier
    uint32_t or_in = 0, or_out = 0, sum_in = 0, sum_out = 0;
    bool diverged = false;
    std::vector<uint32_t> by, rank;       // fibers by priority, and a fiber's place there
    std::vector<uint64_t> ready;          // bit of a place: its fiber can run
    void set(uint32_t t, State s) {
        f[t].state = s;
        const uint64_t bit = 1ull << (rank[t] & 63u);
        if (s == RUN) ready[rank[t] >> 6] |= bit;
        else ready[rank[t] >> 6] &= ~bit;
    }
};
inline Block* B = nullptr;
inline uint64_t barriers = 0;  // block barriers opened so far

inline void leave() {
    if (!_setjmp(B->f[B->cur].at)) _longjmp(B->main, 1);
}

// The block barrier opens when every fiber that is not done is there.
inline void check_block() {
    if (!B->live || B->at < B->live) return;
    B->or_out = B->or_in;
    ++barriers;
    B->sum_out = B->sum_in;
    B->or_in = B->sum_in = B->at = 0;
    for (uint32_t t = 0; t < B->f.size(); ++t)
        if (B->f[t].state == AT_BLOCK) B->set(t, RUN);
}
inline void entry() {
    B->body();
    B->set(B->cur, DONE);
    --B->live;
    check_block();
    leave();
}

// Runs body as block `block` of `grid` with nt threads; prio[t]: priority of
// thread t.  False if the block hangs, or lanes of a warp meet at different
// collectives.
inline bool run(uint32_t nt, uint32_t block, uint32_t grid, const std::vector<uint32_t>& prio, std::function<void()> body) {
    Block blk;
    B = &blk;
    blk.body = std::move(body);
    blk.f = std::vector<Fiber>(nt);
    blk.w.resize(nt / 32);
    blockIdx = {block, 0, 0};
    gridDim = {grid, 1, 1};
    blockDim = {nt, 1, 1};
    constexpr size_t STACK = 64 << 10;
    static std::vector<std::unique_ptr<char[]>> stacks;  // kept for the next block
    while (stacks.size() < nt) stacks.emplace_back(new char[STACK]);
    for (uint32_t t = 0; t < nt; ++t) {
        Fiber& f = blk.f[t];
        getcontext(&f.ctx);
        f.ctx.uc_stack.ss_sp = stacks[t].get();
        f.ctx.uc_stack.ss_size = STACK;
        f.ctx.uc_link = &blk.end;
        makecontext(&f.ctx, entry, 0);
    }
    blk.by.resize(nt);
    blk.rank.resize(nt);
    blk.ready.assign((nt + 63) / 64, 0);
    blk.live = nt;
    for (uint32_t t = 0; t < nt; ++t) blk.by[t] = t;
    std::stable_sort(blk.by.begin(), blk.by.end(), [&](uint32_t a, uint32_t b) { return prio[a] > prio[b]; });
    for (uint32_t r = 0; r < nt; ++r) blk.rank[blk.by[r]] = r;
    for (uint32_t t = 0; t < nt; ++t) blk.set(t, RUN);
    bool ok = true;
    for (;;) {
        uint32_t k = 0;
        while (k < blk.ready.size() && !blk.ready[k]) ++k;
        if (k < blk.ready.size()) {
            blk.cur = blk.by[64 * k + std::countr_zero(blk.ready[k])];
            threadIdx = {blk.cur, 0, 0};
            Fiber& f = blk.f[blk.cur];
            if (!_setjmp(blk.main)) {
                if (f.begun) _longjmp(f.at, 1);
                f.begun = true;
                setcontext(&f.ctx);
            }
            continue;
        }
        for (auto& f : blk.f) ok = ok && f.state == DONE;
        break;
    }
    ok = ok && !blk.diverged;
    B = nullptr;
    return ok;
}

// Priorities.  0: the threads in order; 1: the last one first; 2: lane 0 of
// every warp last; 3: warp 0 first; 4: warp 0 last; 100 and more: the warps in
// a random order, their lanes in order; else all threads in a random order.
inline std::vector<uint32_t> schedule(uint32_t nt, uint32_t kind) {
    std::vector<uint32_t> p(nt), of_warp(nt / 32);
    std::mt19937 g(kind);
    for (auto& x : of_warp) x = g() >> 6;
    for (uint32_t t = 0; t < nt; ++t) {
        const uint32_t w = t / 32, l = t % 32, late = 31 - l;
        p[t] = kind == 0     ? nt - t
               : kind == 1   ? t
               : kind == 2   ? (l ? 1000 + nt - t : w)
               : kind == 3   ? (w ? 0 : nt) + 32 * (nt / 32 - w) + late
               : kind == 4   ? (w ? nt : 0) + 32 * (nt / 32 - w) + late
               : kind >= 100 ? 32 * of_warp[w] + late
                             : g();
    }
    return p;
}

template <typename T>
inline T warp_op(int op, T v, const std::function<uint64_t(const uint64_t*, uint32_t)>& f) {
    const uint32_t t = B->cur, l = t % 32;
    uint64_t x = 0;
    static_assert(sizeof(T) <= 8);
    memcpy(&x, &v, sizeof v);
    B->w[t / 32].in[l] = x;
    Warp& w = B->w[t / 32];
    B->set(t, AT_WARP);
    if (w.at++ && op != w.op) B->diverged = true;
    w.op = op;
    if (w.at == 32) {
        w.at = 0;
        memcpy(w.out, w.in, sizeof w.out);
        for (uint32_t i = 0; i < 32; ++i) B->set(t - l + i, RUN);
    }
    leave();
    x = f(B->w[t / 32].out, l);
    T r;
    memcpy(&r, &x, sizeof r);
    return r;
}
inline uint32_t block_op(uint32_t v) {
    B->or_in |= v;
    B->sum_in += v;
    B->set(B->cur, AT_BLOCK);
    ++B->at;
    check_block();
    leave();
    return B->or_out;
}
template <typename F>
inline uint32_t fold(int op, uint32_t v, F g) {
    return warp_op<uint32_t>(op, v, [&](const uint64_t* a, uint32_t) {
        uint32_t r = (uint32_t)a[0];
        for (int i = 1; i < 32; ++i) r = g(r, (uint32_t)a[i]);
        return (uint64_t)r;
    });
}
}  // namespace simt

inline void __syncthreads() { simt::block_op(0); }
inline int __syncthreads_or(int p) { return simt::block_op(p != 0) != 0; }
inline int __syncthreads_count(int p) {
    simt::block_op(p != 0);
    return simt::B->sum_out;
}
inline void __syncwarp() {
    simt::warp_op<uint32_t>(1, 0, [](const uint64_t*, uint32_t) { return 0; });
}
template <typename T>
inline T __shfl_sync(uint32_t, T v, int s) {
    return simt::warp_op<T>(2, v, [&](const uint64_t* a, uint32_t) { return a[s & 31]; });
}
template <typename T>
inline T __shfl_up_sync(uint32_t, T v, uint32_t d) {
    return simt::warp_op<T>(3, v, [&](const uint64_t* a, uint32_t l) { return a[l >= d ? l - d : l]; });
}
template <typename T>
inline T __shfl_down_sync(uint32_t, T v, uint32_t d) {
    return simt::warp_op<T>(4, v, [&](const uint64_t* a, uint32_t l) { return a[l + d < 32 ? l + d : l]; });
}
template <typename T>
inline T __shfl_xor_sync(uint32_t, T v, int m) {
    return simt::warp_op<T>(5, v, [&](const uint64_t* a, uint32_t l) { return a[l ^ m]; });
}
inline uint32_t __ballot_sync(uint32_t, int p) {
    return simt::warp_op<uint32_t>(6, p != 0, [](const uint64_t* a, uint32_t) {
        uint64_t r = 0;
        for (int i = 0; i < 32; ++i) r |= (a[i] & 1u) << i;
        return r;
    });
}
inline int __any_sync(uint32_t m, int p) { return __ballot_sync(m, p) != 0; }
inline int __all_sync(uint32_t m, int p) { return __ballot_sync(m, p) == 0xffffffffu; }
template <typename T>
inline uint32_t __match_any_sync(uint32_t, T v) {
    return (uint32_t)simt::warp_op<uint64_t>(7, (uint64_t)v, [](const uint64_t* a, uint32_t l) {
        uint64_t r = 0;
        for (int i = 0; i < 32; ++i) r |= (uint64_t)(a[i] == a[l]) << i;
        return r;
    });
}
inline uint32_t __reduce_add_sync(uint32_t, uint32_t v) { return simt::fold(8, v, [](uint32_t a, uint32_t b) { return a + b; }); }
inline uint32_t __reduce_or_sync(uint32_t, uint32_t v) { return simt::fold(9, v, [](uint32_t a, uint32_t b) { return a | b; }); }
inline uint32_t __reduce_max_sync(uint32_t, uint32_t v) { return simt::fold(10, v, [](uint32_t a, uint32_t b) { return std::max(a, b); }); }
inline uint32_t __reduce_min_sync(uint32_t, uint32_t v) { return simt::fold(11, v, [](uint32_t a, uint32_t b) { return std::min(a, b); }); }

template <typename T, typename F>
inline T simt_atomic(T* p, F f) {
    const T old = *p;
    *p = f(old);
    if (simt::B) simt::leave();  // other threads may run
    return old;
}
template <typename T>
inline T atomicAdd(T* p, T v) { return simt_atomic(p, [&](T o) { return (T)(o + v); }); }
template <typename T>
inline T atomicMin(T* p, T v) { return simt_atomic(p, [&](T o) { return std::min(o, v); }); }
template <typename T>
inline T atomicMax(T* p, T v) { return simt_atomic(p, [&](T o) { return std::max(o, v); }); }
template <typename T>
inline T __ldg(const T* p) { return *p; }

inline int __popc(uint32_t x) { return std::popcount(x); }
inline int __ffs(uint32_t x) { return x ? std::countr_zero(x) + 1 : 0; }
inline int __ffsll(long long x) { return x ? std::countr_zero((uint64_t)x) + 1 : 0; }
inline int __clz(uint32_t x) { return std::countl_zero(x); }
inline int __clzll(long long x) { return std::countl_zero((uint64_t)x); }
inline uint32_t __brev(uint32_t x) {
    uint32_t r = 0;
    for (int i = 0; i < 32; ++i) r |= ((x >> i) & 1u) << (31 - i);
    return r;
}
// shifts of the 64-bit hi:lo by s modulo 32
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) { return (uint32_t)((((uint64_t)hi << 32) | lo) >> (s & 31)); }
template <typename A, typename C>
inline std::common_type_t<A, C> min(A a, C b) { return a < b ? a : b; }
template <typename A, typename C>
inline std::common_type_t<A, C> max(A a, C b) { return a < b ? b : a; }
