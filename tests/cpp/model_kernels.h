// model_kernels.h - what share.cuh uses of CUDA and of kernels.h, for the host
// (share_model.cpp): a fiber per one-lane warp, every memory operation a step
// after which another fiber may run.
#pragma once
#include <ucontext.h>

#include <algorithm>
#include <cstdint>
#include <functional>
#include <memory>
#include <random>
#include <vector>

#define __device__
#define __forceinline__ inline
#define __noinline__

struct ulonglong2 { unsigned long long x, y; };
struct uint2 { uint32_t x, y; };
inline uint2 make_uint2(uint32_t x, uint32_t y) { return {x, y}; }
using std::max;
using std::min;

namespace model {
struct Dim { uint32_t x; };
struct Fiber {
    ucontext_t ctx;
    std::vector<char> stack;
    std::function<void()> body;
    Dim thread, block, block_dim, grid_dim;
    uint32_t start = 0;
    bool ended = false;
};
inline Fiber* now;
inline ucontext_t home;
inline std::vector<std::unique_ptr<Fiber>> pool;

inline void step() { swapcontext(&now->ctx, &home); }
inline void enter() {
    now->body();
    now->ended = true;
    swapcontext(&now->ctx, &home);
}
inline Fiber* spawn(std::function<void()> body, uint32_t block, uint32_t warp, uint32_t blocks, uint32_t warps, uint32_t start) {
    pool.emplace_back(new Fiber);
    Fiber* f = pool.back().get();
    f->body = std::move(body);
    f->thread = {32 * warp};
    f->block = {block};
    f->block_dim = {32 * warps};
    f->grid_dim = {blocks};
    f->start = start;
    f->stack.resize(64 * 1024);
    getcontext(&f->ctx);
    f->ctx.uc_stack.ss_sp = f->stack.data();
    f->ctx.uc_stack.ss_size = f->stack.size();
    f->ctx.uc_link = nullptr;
    makecontext(&f->ctx, (void (*)()) enter, 0);
    return f;
}
// Runs the fibers to their end, a random one a few steps at a time; false when they do not end.
inline bool run(const std::vector<Fiber*>& fibers, std::mt19937& rng) {
    uint64_t t = 0;
    bool ended = false;
    for (; t < 20000000 && !ended;) {
        Fiber* f = fibers[rng() % fibers.size()];
        const uint32_t burst = rng() % 4 ? 1 : 1 + rng() % 12;
        for (uint32_t k = 0; k < burst && !f->ended && t >= f->start; ++k) {
            now = f;
            swapcontext(&home, &f->ctx);
        }
        ++t;
        ended = std::all_of(fibers.begin(), fibers.end(), [](Fiber* x) { return x->ended; });
    }
    pool.clear();
    return ended;
}
// A pointer whose every use is a step (the places that read or write volatile words).
template <class T>
struct Step {
    T* p;
    Step(T* q) : p(q) {}
    Step(const T* q) : p(const_cast<T*>(q)) {}
    T& operator*() const {
        step();
        return *p;
    }
};
template <class T>
T add(T* p, T v) {
    step();
    const T old = *p;
    *p += v;
    return old;
}
}  // namespace model

#define threadIdx (model::now->thread)
#define blockIdx (model::now->block)
#define blockDim (model::now->block_dim)
#define gridDim (model::now->grid_dim)

inline uint32_t atomicAdd(uint32_t* p, uint32_t v) { return model::add(p, v); }
inline unsigned long long atomicAdd(unsigned long long* p, unsigned long long v) { return model::add(p, v); }
inline uint32_t atomicSub(uint32_t* p, uint32_t v) { return model::add(p, (uint32_t) -v); }
inline uint32_t atomicOr(uint32_t* p, uint32_t v) {
    model::step();
    const uint32_t old = *p;
    *p |= v;
    return old;
}
inline unsigned long long atomicAnd(unsigned long long* p, unsigned long long v) {
    model::step();
    const unsigned long long old = *p;
    *p &= v;
    return old;
}
inline unsigned long long atomicExch(unsigned long long* p, unsigned long long v) {
    model::step();
    std::swap(*p, v);
    return v;
}
inline unsigned long long atomicCAS(unsigned long long* p, unsigned long long was, unsigned long long v) {
    model::step();
    const unsigned long long old = *p;
    if (old == was) *p = v;
    return old;
}
inline void __threadfence() {}
inline void __syncwarp() {}
inline void __nanosleep(uint32_t) {}
template <class T>
T __shfl_sync(uint32_t, T v, int) { return v; }
inline uint32_t __ballot_sync(uint32_t, bool p) { return p ? 1u : 0u; }
inline int __popc(uint32_t v) { return __builtin_popcount(v); }

// The shared word of a block that says whether it counts as live; its reads are steps.
struct LiveWord {
    uint32_t v = 0;
    operator uint32_t() const {
        model::step();
        return v;
    }
    LiveWord& operator=(uint32_t x) {
        v = x;
        return *this;
    }
};
// share_start's barrier keeps its clearing of that word before its setting, both by one thread here.
inline void __syncthreads() {}

namespace rtcd {
constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kErrLookback = 1u << 1;
struct TaskQueue {
    unsigned long long* queue;
    uint32_t* live;
    uint32_t* over;
    uint32_t* err;
    ulonglong2* slot;
    uint32_t slots;
    uint32_t most_waiting;
};
}  // namespace rtcd
