// Runs device functions of csrc/*.cuh on the CPU: every CUDA thread of one
// block is a fiber that runs until it meets a barrier or a warp collective,
// and the fibers are resumed in an order that the caller picks.  An order that
// runs some threads as far ahead of the others as the barriers allow shows
// what the barriers do not order.  Barriers are counted over all live threads
// of the block (warp collectives over all 32 lanes); a round in which nothing
// moves is reported as a deadlock.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <ucontext.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <type_traits>
#include <vector>

namespace emu {

struct Fiber {
    ucontext_t ctx;
    std::vector<char> stack;
    bool done = false;
};

inline std::vector<Fiber> fibers;
inline ucontext_t scheduler;
inline uint32_t cur, threads;
inline bool moved;   // some thread went past a barrier, or ended, in this round
inline std::function<void()> body;

inline void yield() { swapcontext(&fibers[cur].ctx, &scheduler); }

// A barrier of `n` threads that also collects one value a thread; every
// thread sees all of a round's values.
struct Meeting {
    uint32_t n = 0, arrived = 0;
    uint64_t round = 0;
    std::vector<uint64_t> in, out;
    const std::vector<uint64_t>& meet(uint32_t rank, uint64_t v) {
        if (in.empty()) in.resize(n);
        in[rank] = v;
        const uint64_t r = round;
        if (++arrived == n) {
            out = in;
            arrived = 0;
            ++round;
            moved = true;
        } else {
            while (round == r) yield();
        }
        return out;
    }
};

inline Meeting block;
inline std::vector<Meeting> warps;

inline const std::vector<uint64_t>& warp_meet(uint64_t v) { return warps[cur / 32].meet(cur % 32, v); }

inline void entry() {
    body();
    fibers[cur].done = true;
    moved = true;
    yield();
}

// Runs `f` as one block of `n` threads, resumed in the order given.  False
// when the threads wait for one another for good.
inline bool run_block(uint32_t n, const std::vector<uint32_t>& order, std::function<void()> f) {
    threads = n;
    body = std::move(f);
    fibers = std::vector<Fiber>(n);
    block = Meeting{};
    block.n = n;
    warps.assign(n / 32, Meeting{});
    for (Meeting& w : warps) w.n = 32;
    for (Fiber& t : fibers) {
        t.stack.resize(64 << 10);
        getcontext(&t.ctx);
        t.ctx.uc_stack.ss_sp = t.stack.data();
        t.ctx.uc_stack.ss_size = t.stack.size();
        t.ctx.uc_link = nullptr;
        makecontext(&t.ctx, entry, 0);
    }
    for (uint32_t left = n; left;) {
        moved = false;
        for (uint32_t k : order) {
            if (fibers[k].done) continue;
            cur = k;
            swapcontext(&scheduler, &fibers[k].ctx);
            if (fibers[k].done) --left;
        }
        if (!moved) return false;
    }
    return true;
}

struct Index {
    struct X {
        operator uint32_t() const { return cur; }
    } x;
};
struct Size {
    struct X {
        operator uint32_t() const { return threads; }
    } x;
};
struct One {
    uint32_t x;
};
inline Index thread_idx;
inline Size block_dim;
inline One block_idx{0}, grid_dim{1};

}  // namespace emu

using std::max;
using std::min;

inline void __syncthreads() { emu::block.meet(emu::cur, 0); }
inline int __syncthreads_or(int p) {
    int r = 0;
    for (uint64_t v : emu::block.meet(emu::cur, p != 0)) r |= static_cast<int>(v);
    return r;
}
inline void __syncwarp(uint32_t = 0xFFFFFFFFu) { emu::warp_meet(0); }
inline uint32_t __ballot_sync(uint32_t, int p) {
    uint32_t r = 0, lane = 0;
    for (uint64_t v : emu::warp_meet(p != 0)) r |= static_cast<uint32_t>(v) << lane++;
    return r;
}
inline int __any_sync(uint32_t m, int p) { return __ballot_sync(m, p) != 0; }
template <typename T>
T __shfl_sync(uint32_t, T v, int src) {
    return static_cast<T>(emu::warp_meet(v)[src]);
}
template <typename T>
T __shfl_down_sync(uint32_t, T v, int d) {
    const uint32_t lane = emu::cur % 32, src = lane + d < 32 ? lane + d : lane;
    return static_cast<T>(emu::warp_meet(v)[src]);
}
inline void __threadfence() {}
template <typename T>
T __ldg(const T* p) {
    return *p;
}
template <typename T>
T __ldcg(const T* p) {
    return *p;
}
template <typename T>
T atomicAdd(T* p, std::common_type_t<T> v) {
    const T o = *p;
    *p += v;
    return o;
}
template <typename T>
T atomicOr(T* p, std::common_type_t<T> v) {
    const T o = *p;
    *p |= v;
    return o;
}
template <typename T>
T atomicMin(T* p, std::common_type_t<T> v) {
    const T o = *p;
    if (v < o) *p = v;
    return o;
}
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) {
    return static_cast<uint32_t>(((static_cast<uint64_t>(hi) << 32) | lo) >> (s & 31));
}
inline int __popc(uint32_t v) { return __builtin_popcount(v); }
inline int __ffs(uint32_t v) { return __builtin_ffs(static_cast<int>(v)); }
inline int __clz(uint32_t v) { return v ? __builtin_clz(v) : 32; }

// Only named by functions that are not run here.
inline size_t __cvta_generic_to_shared(const void*) { return 0; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __ddiv_rn(double a, double b) { return a / b; }

#include "gsc_kernels.cuh"   // (launch configurations have members of the names below)

#define __noinline__ __attribute__((noinline))
#define threadIdx emu::thread_idx
#define blockDim emu::block_dim
#define blockIdx emu::block_idx
#define gridDim emu::grid_dim
