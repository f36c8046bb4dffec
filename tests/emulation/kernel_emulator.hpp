// Runs the source of a CUDA kernel on the CPU: every thread of a launch is a fiber with its own stack, and a
// scheduler picks who runs next, so that a test can choose interleavings a GPU rarely shows. Include it
// before the kernel's headers.
//
//  * A warp collective (vote, shuffle, __syncwarp ...) returns when all 32 lanes have come to the same
//    source line; lanes of a warp at different collectives, a thread that ends while its warp still
//    works, and a launch in which nobody can go on are failures.
//  * __syncthreads waits for all threads of the block.
//  * Order::Lockstep: a warp picked at random runs from one collective to the next, lane after lane (a
//    converged warp). Order::Skewed: any lane may run next, and may stop at any arithmetic operation,
//    atomic or byte-sum between two collectives (independent thread scheduling).
//  * A block can start late: after `start[block]` scheduling decisions.
#pragma once

#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <random>
#include <vector>

struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
struct uint4 { unsigned x, y, z, w; };
inline float2 make_float2(float x, float y) { return {x, y}; }
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
inline uint4 make_uint4(unsigned x, unsigned y, unsigned z, unsigned w) { return {x, y, z, w}; }

namespace emu {

struct Dim { unsigned x = 0, y = 0, z = 0; };
enum class Order { Lockstep, Skewed };
enum class State { Ready, Warp, Block, Done };

struct Fiber {
    ucontext_t ctx;
    std::unique_ptr<char[]> stack;
    Dim thread, block;
    int warp, lane;  // warp: of the launch
    State state = State::Ready;
    int site = 0;       // the collective it waits at
    uint64_t value = 0; // what it brings
};

struct Launch {
    std::vector<Fiber> fibers;
    int threads, warps_per_block;
    std::vector<uint64_t> shared;      // of every block, while it does not run
    size_t shared_words = 0;
    uint64_t (*given)[32] = nullptr;   // of every warp: the last collective's values
    std::vector<uint64_t> values;
    std::mt19937_64 rng;
    Order order;
};
inline Launch *g = nullptr;
inline Fiber *self = nullptr;
inline ucontext_t scheduler;
inline uint64_t *shared_memory = nullptr;  // the array the kernel's `extern __shared__` names
inline const char *failure = nullptr;

inline void pause() { swapcontext(&self->ctx, &scheduler); }
// a place where an independently scheduled lane may stop
inline void may_stop() {
    if (g && g->order == Order::Skewed && g->rng() % 48 == 0) pause();
}
inline const uint64_t *collective(int site, uint64_t value) {
    self->state = State::Warp;
    self->site = site;
    self->value = value;
    pause();
    return g->values.data() + 32 * static_cast<size_t>(self->warp);
}
inline uint32_t ballot(int site, bool p) {
    const uint64_t *v = collective(site, p);
    uint32_t m = 0u;
    for (int i = 0; i < 32; ++i) m |= (v[i] ? 1u : 0u) << i;
    return m;
}
inline uint32_t shfl(int site, uint32_t v, int from) { return static_cast<uint32_t>(collective(site, v)[from & 31]); }
inline uint32_t sum(int site, uint32_t v) {
    const uint64_t *all = collective(site, v);
    uint32_t s = 0u;
    for (int i = 0; i < 32; ++i) s += static_cast<uint32_t>(all[i]);
    return s;
}
inline void sync_block() {
    self->state = State::Block;
    pause();
}

inline const std::function<void()> *body = nullptr;
inline void enter() {
    (*body)();
    self->state = State::Done;
    pause();
}

// Runs `kernel` on `blocks` x `threads` threads with `words` 64-bit words of shared memory per block at
// `memory`. Returns NULL, or what went wrong.
inline const char *run(int blocks, int threads, size_t words, uint64_t *memory, Order order, uint64_t seed,
                       const std::vector<uint64_t> &start, const std::function<void()> &kernel, Dim &threadIdx_, Dim &blockIdx_) {
    const auto owner = std::make_unique<Launch>();
    Launch &l = *owner;
    l.threads = threads;
    l.warps_per_block = threads / 32;
    l.order = order;
    l.rng.seed(seed);
    l.shared.assign(words * static_cast<size_t>(blocks), 0xA5A5A5A5A5A5A5A5ull);
    l.shared_words = words;
    l.values.assign(static_cast<size_t>(blocks) * threads, 0);
    l.fibers = std::vector<Fiber>(static_cast<size_t>(blocks) * threads);
    g = &l;
    body = &kernel;
    failure = nullptr;
    const size_t stack = 64 * 1024;
    for (size_t i = 0; i < l.fibers.size(); ++i) {
        Fiber &f = l.fibers[i];
        f.stack = std::make_unique<char[]>(stack);
        f.block.x = static_cast<unsigned>(i / threads);
        f.thread.x = static_cast<unsigned>(i % threads);
        f.warp = static_cast<int>(i / 32);
        f.lane = static_cast<int>(i % 32);
        getcontext(&f.ctx);
        f.ctx.uc_stack.ss_sp = f.stack.get();
        f.ctx.uc_stack.ss_size = stack;
        f.ctx.uc_link = nullptr;
        makecontext(&f.ctx, enter, 0);
    }
    int resident = -1;  // the block whose shared memory is in place
    const int warps = blocks * l.warps_per_block;
    std::vector<int> waiting(static_cast<size_t>(blocks), 0);
    const auto step = [&](Fiber &f) {
        const int b = static_cast<int>(f.block.x);
        if (b != resident) {
            if (resident >= 0) std::memcpy(l.shared.data() + words * resident, memory, words * 8);
            std::memcpy(memory, l.shared.data() + words * b, words * 8);
            resident = b;
        }
        self = &f;
        threadIdx_ = f.thread;
        blockIdx_ = f.block;
        swapcontext(&scheduler, &f.ctx);
        if (f.state == State::Block && ++waiting[b] == threads) {
            waiting[b] = 0;
            for (int i = 0; i < threads; ++i) l.fibers[static_cast<size_t>(b) * threads + i].state = State::Ready;
        }
    };
    std::vector<int> candidates;
    for (uint64_t tick = 0;; ++tick) {
        if (tick > 40000000ull) return "the launch does not end";
        candidates.clear();
        bool all_done = true, later = false;
        for (int w = 0; w < warps; ++w) {
            bool ready = false;
            for (int i = 0; i < 32; ++i) {
                const State s = l.fibers[static_cast<size_t>(w) * 32 + i].state;
                all_done = all_done && s == State::Done;
                ready = ready || s == State::Ready;
            }
            const size_t b = static_cast<size_t>(w / l.warps_per_block);
            if (ready && b < start.size() && tick < start[b]) later = true;
            else if (ready) candidates.push_back(w);
        }
        if (all_done) break;
        if (candidates.empty()) {
            if (later) continue;
            return "a barrier that not all of its threads come to";
        }
        const int w = candidates[l.rng() % candidates.size()];
        Fiber *const lanes = l.fibers.data() + static_cast<size_t>(w) * 32;
        if (order == Order::Lockstep) {
            for (int i = 0; i < 32; ++i)
                if (lanes[i].state == State::Ready) step(lanes[i]);
        } else {
            for (int turns = 0; turns < 64; ++turns) {
                Fiber &f = lanes[l.rng() % 32];
                if (f.state == State::Ready) step(f);
            }
        }
        int at = 0, ended = 0, site = 0;
        for (int i = 0; i < 32; ++i) {
            if (lanes[i].state == State::Done) ++ended;
            if (lanes[i].state != State::Warp) continue;
            if (at++ && lanes[i].site != site) return "the lanes of a warp wait at different collectives";
            site = lanes[i].site;
        }
        if (at && ended) return "a lane has ended while others of its warp wait for it";
        if (at == 32) {
            for (int i = 0; i < 32; ++i) {
                l.values[static_cast<size_t>(w) * 32 + i] = lanes[i].value;
                lanes[i].state = State::Ready;
            }
        }
    }
    g = nullptr;
    return nullptr;
}

}  // namespace emu

inline emu::Dim threadIdx, blockIdx, blockDim, gridDim;

#define __host__
#define __device__
#define __global__
#define __shared__
#define __grid_constant__
#define __restrict__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#define __align__(n) __attribute__((aligned(n)))
#define __launch_bounds__(...)

// collectives: the site is the source line
#define __ballot_sync(mask, p) emu::ballot(__LINE__, (p))
#define __any_sync(mask, p) (emu::ballot(__LINE__, (p)) != 0u)
#define __all_sync(mask, p) (emu::ballot(__LINE__, (p)) == 0xffffffffu)
#define __shfl_sync(mask, v, from) emu::shfl(__LINE__, (v), (from))
#define __reduce_add_sync(mask, v) emu::sum(__LINE__, (v))
#define __shfl_down_sync(mask, v, n) (v)  // only in kernels that no test runs here
#define __syncwarp() ((void)emu::collective(__LINE__, 0))
#define __syncthreads() emu::sync_block()

// arithmetic, each a place to stop
inline float __fmul_rn(float a, float b) { return emu::may_stop(), a * b; }
inline float __fadd_rn(float a, float b) { return emu::may_stop(), a + b; }
inline float __fsub_rn(float a, float b) { return emu::may_stop(), a - b; }
inline float __fmaf_rn(float a, float b, float c) { return emu::may_stop(), std::fma(a, b, c); }
inline float2 __fmul2_rn(float2 a, float2 b) { return {__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)}; }
inline float2 __ffma2_rn(float2 a, float2 b, float2 c) { return {__fmaf_rn(a.x, b.x, c.x), __fmaf_rn(a.y, b.y, c.y)}; }
template <class T> T emu_add(T *p, T v) {
    emu::may_stop();
    const T old = *p;
    *p = old + v;
    return old;
}
inline uint32_t atomicAdd(uint32_t *p, uint32_t v) { return emu_add(p, v); }
inline unsigned long long atomicAdd(unsigned long long *p, unsigned long long v) { return emu_add(p, v); }
inline int atomicExch(int *p, int v) { return std::swap(*p, v), v; }
inline int atomicCAS(int *p, int expected, int v) {
    const int old = *p;
    if (old == expected) *p = v;
    return old;
}
inline unsigned __dp4a(unsigned a, unsigned b, unsigned c) {
    emu::may_stop();
    for (int i = 0; i < 4; ++i) c += ((a >> (8 * i)) & 0xFFu) * ((b >> (8 * i)) & 0xFFu);
    return c;
}
inline int __popc(unsigned x) { return __builtin_popcount(x); }
inline int __ffs(int x) { return __builtin_ffs(x); }
inline unsigned umin(unsigned a, unsigned b) { return std::min(a, b); }
using std::max;
using std::min;
inline float __uint_as_float(unsigned x) {
    float f;
    std::memcpy(&f, &x, 4);
    return f;
}
inline unsigned __funnelshift_r(unsigned lo, unsigned hi, unsigned n) {
    return static_cast<unsigned>(((static_cast<uint64_t>(hi) << 32) | lo) >> (n & 31));
}
// as the GPU converts: what is no number or negative is 0 (in 64 bits, no number is 2^63), too large the largest
inline unsigned __float2uint_rz(float x) { return !(x > 0.0f) ? 0u : x >= 4294967296.0f ? 0xFFFFFFFFu : static_cast<unsigned>(x); }
inline unsigned long long __float2ull_rn(float x) {
    if (x != x) return 1ull << 63;
    return x <= 0.0f ? 0ull : x >= 18446744073709551616.0f ? ~0ull : static_cast<unsigned long long>(std::nearbyint(static_cast<double>(x)));
}
template <class T> T __ldg(const T *p) { return *p; }
inline void __sincosf(float, float *, float *) { std::abort(); }  // the fast forms are not emulated
