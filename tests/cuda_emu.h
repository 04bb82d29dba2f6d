// Runs kernels of csrc/ on the CPU, one schedule at a time: every thread of a
// block is a fiber, every block an OS thread, and one fiber runs at any moment.
// A fiber runs until it waits (block barrier, warp exchange, __nanosleep), so
// the order in which warps and blocks get through a kernel is what the test
// asks for, and a result that depends on it is a race.  Compiled by g++ with the
// kernel's source included after this file.
#pragma once
#include <cuda_runtime.h>
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

#undef __shared__
#undef __global__
#undef __device__
#undef __host__
#undef __constant__
#undef __forceinline__
#undef __launch_bounds__
#undef __noinline__
#define __shared__ static thread_local
#define __global__ static
#define __device__
#define __host__
#define __constant__ const
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __noinline__

namespace emu {

enum Wait { RUN, BLOCK_BARRIER, WARP_BARRIER, SLEEP, DONE };

struct Fiber {
    ucontext_t ctx;
    std::vector<char> stack;
    uint3 tid;
    Wait wait = RUN;
};

// the token that lets one block run at a time: block b keeps it for turns[b]
// waits, then the next block that has not finished gets it
struct Token {
    std::mutex m;
    std::condition_variable cv;
    std::vector<int> turns;
    std::vector<char> done;
    int owner = 0, used = 0;
    void next() {
        used = 0;
        for (size_t k = 0; k < done.size(); ++k) {
            owner = (owner + 1) % (int)done.size();
            if (!done[owner]) break;
        }
        cv.notify_all();
    }
    void acquire(int b) {
        std::unique_lock<std::mutex> l(m);
        cv.wait(l, [&] { return owner == b; });
    }
    void yield(int b) {
        std::unique_lock<std::mutex> l(m);
        if (++used >= turns[b]) next();
        cv.wait(l, [&] { return owner == b; });
    }
    void finish(int b) {
        std::unique_lock<std::mutex> l(m);
        done[b] = 1;
        next();
    }
};

struct Block {
    int id = 0;
    uint3 bid;
    dim3 bdim, gdim;
    std::vector<Fiber> fibers;
    Fiber* cur = nullptr;
    ucontext_t main;
    std::function<void()> body;
    std::vector<unsigned long long> slot;  // warp exchange, one a thread
    int votes = 0, voted = 0;
    Token* token = nullptr;
};
inline thread_local Block* blk = nullptr;

inline void wait(Wait w) {
    Fiber* f = blk->cur;
    f->wait = w;
    swapcontext(&f->ctx, &blk->main);
}
inline void entry() {
    blk->body();
    blk->cur->wait = DONE;
    swapcontext(&blk->cur->ctx, &blk->main);
}

// order: the warps of the block in the order in which they get to run
inline void run_block(Block& b, const std::vector<int>& order) {
    blk = &b;
    const int n = (int)b.bdim.x;
    b.fibers = std::vector<Fiber>(n);
    b.slot.assign(n, 0);
    for (int t = 0; t < n; ++t) {
        Fiber& f = b.fibers[t];
        f.stack.resize(256 << 10);
        f.tid = {(unsigned)t, 0, 0};
        getcontext(&f.ctx);
        f.ctx.uc_stack.ss_sp = f.stack.data();
        f.ctx.uc_stack.ss_size = f.stack.size();
        makecontext(&f.ctx, entry, 0);
    }
    for (;;) {
        // every warp as far as it comes before the next one gets its turn
        bool moved = false, alive = false, slept = false;
        for (int w : order) {
            Fiber* l = &b.fibers[32 * w];
            for (bool again = true; again;) {
                again = false;
                for (int k = 0; k < 32; ++k)
                    if (l[k].wait == RUN) {
                        b.cur = &l[k];
                        swapcontext(&b.main, &l[k].ctx);
                        moved = true;
                    }
                int at = 0;
                for (int k = 0; k < 32; ++k) at += l[k].wait == WARP_BARRIER;
                if (at == 32) {
                    for (int k = 0; k < 32; ++k) l[k].wait = RUN;
                    again = true;
                }
            }
        }
        for (Fiber& f : b.fibers) {
            alive = alive || f.wait != DONE;
            if (f.wait == SLEEP) f.wait = RUN, slept = true;
        }
        if (!alive) break;
        bool barrier = true;
        for (const Fiber& f : b.fibers) barrier = barrier && (f.wait == BLOCK_BARRIER || f.wait == DONE);
        if (barrier) {
            for (Fiber& f : b.fibers)
                if (f.wait == BLOCK_BARRIER) f.wait = RUN;
        } else if (!moved) {
            fprintf(stderr, "block %d cannot go on\n", b.id);
            abort();
        }
        if (b.token && (barrier || slept)) b.token->yield(b.id);
    }
}

// one block after the other
inline void launch(unsigned grid, unsigned block, const std::vector<int>& order, const std::function<void()>& body) {
    for (unsigned k = 0; k < grid; ++k) {
        Block b;
        b.bid = {k, 0, 0}, b.bdim = dim3(block), b.gdim = dim3(grid), b.body = body;
        run_block(b, order);
    }
}
// all blocks resident, block b for turns[b] waits at a time
inline void launch_resident(unsigned block, const std::vector<int>& turns, const std::function<void()>& body) {
    Token tk;
    tk.turns = turns;
    tk.done.assign(turns.size(), 0);
    std::vector<int> order;
    for (int w = 0; w < (int)block / 32; ++w) order.push_back(w);
    std::vector<std::thread> th;
    for (int k = 0; k < (int)turns.size(); ++k)
        th.emplace_back([&, k] {
            Block b;
            b.id = k, b.bid = {(unsigned)k, 0, 0}, b.bdim = dim3(block), b.gdim = dim3((unsigned)turns.size());
            b.body = body, b.token = &tk;
            tk.acquire(k);
            run_block(b, order);
            tk.finish(k);
        });
    for (std::thread& t : th) t.join();
}

template <class T>
T shfl_down(T v, int off) {
    const int t = (int)blk->cur->tid.x, lane = t & 31;
    memcpy(&blk->slot[t], &v, sizeof(T));
    wait(WARP_BARRIER);
    T r = v;
    if (lane + off < 32) memcpy(&r, &blk->slot[t + off], sizeof(T));
    wait(WARP_BARRIER);
    return r;
}
inline unsigned ballot(bool p) {
    const int t = (int)blk->cur->tid.x, w = t & ~31;
    blk->slot[t] = p;
    wait(WARP_BARRIER);
    unsigned r = 0;
    for (int k = 0; k < 32; ++k) r |= (unsigned)(blk->slot[w + k] != 0) << k;
    wait(WARP_BARRIER);
    return r;
}
inline int block_or(int p) {
    blk->votes |= p != 0;
    wait(BLOCK_BARRIER);
    const int r = blk->votes;
    wait(BLOCK_BARRIER);
    blk->votes = 0;
    wait(BLOCK_BARRIER);
    return r;
}

}  // namespace emu

#define threadIdx (emu::blk->cur->tid)
#define blockIdx (emu::blk->bid)
#define blockDim (emu::blk->bdim)
#define gridDim (emu::blk->gdim)

using std::max;
using std::min;
inline void __syncthreads() { emu::wait(emu::BLOCK_BARRIER); }
inline int __syncthreads_or(int p) { return emu::block_or(p); }
inline void __syncwarp() { emu::wait(emu::WARP_BARRIER); }
inline void __nanosleep(unsigned) { emu::wait(emu::SLEEP); }
inline void __threadfence() {}
template <class T>
T __shfl_down_sync(unsigned, T v, int off) {
    return emu::shfl_down(v, off);
}
inline unsigned __ballot_sync(unsigned, int p) { return emu::ballot(p != 0); }
inline int __any_sync(unsigned, int p) { return emu::ballot(p != 0) != 0; }
inline int __all_sync(unsigned, int p) { return emu::ballot(p != 0) == ~0u; }
inline unsigned __reduce_add_sync(unsigned, unsigned v) {
    for (int o = 16; o > 0; o >>= 1) v += emu::shfl_down(v, o);
    return v;
}
inline int __reduce_add_sync(unsigned m, int v) { return (int)__reduce_add_sync(m, (unsigned)v); }
template <class T, class U>
T atomicAdd(T* p, U v) {
    const T o = *p;
    *p = o + (T)v;
    return o;
}
template <class T>
T atomicExch(T* p, T v) {
    std::swap(*p, v);
    return v;
}
template <class T>
T atomicMax(T* p, T v) {
    const T o = *p;
    *p = max(o, v);
    return o;
}
template <class T>
T __ldg(const T* p) {
    return *p;
}
template <class T>
T __ldcg(const T* p) {
    return *p;
}
inline int __popc(unsigned x) { return __builtin_popcount(x); }
inline int __ffs(int x) { return __builtin_ffs(x); }
inline int __clz(int x) { return x ? __builtin_clz((unsigned)x) : 32; }
inline unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned s) {
    return (unsigned)(((((unsigned long long)hi << 32) | lo) << (s & 31)) >> 32);
}
inline unsigned __funnelshift_r(unsigned lo, unsigned hi, unsigned s) {
    return (unsigned)((((unsigned long long)hi << 32) | lo) >> (s & 31));
}
inline long long emu_bits(double x) {
    long long b;
    memcpy(&b, &x, 8);
    return b;
}
inline int __double2hiint(double x) { return (int)(emu_bits(x) >> 32); }
inline int __double2loint(double x) { return (int)emu_bits(x); }
inline double __longlong_as_double(long long b) {
    double x;
    memcpy(&x, &b, 8);
    return x;
}
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
inline float emu_rsqrtf(float x) { return 1.0f / sqrtf(x); }
#define rsqrtf emu_rsqrtf
