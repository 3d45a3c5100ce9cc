// share_model.cpp - the work sharing of csrc/share.cuh on the host: its own
// code, run by fibers that stand for one-lane warps, one memory operation at a
// time in random order, with blocks that start late.  Prints a line per kind of
// fault found; exit status 0 when there is none.
//
// share_model <schedules> <seed>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "share.cuh"  // beside a kernels.h that provides what follows (model_kernels.h)

using namespace rtcd;

namespace {

constexpr uint32_t kBlocks = 3, kWarps = 2;
constexpr uint32_t kSlots = 64;

struct Launch {
    TaskQueue q{};
    uint32_t live = 0, over = 0, work = 0;
    std::vector<uint32_t> sizes;               // nodes of each item's binary tree (node k: 2k, 2k + 1)
    std::vector<std::vector<uint32_t>> done;   // expansions of each node
    LiveWord s_live[kBlocks];
    bool stale = false;
};

// One warp of the query kernel: items in turn, then tasks; nodes offered while two wait.
void warp_loop(Launch& L, uint32_t block, uint32_t warp) {
    const uint32_t warps = kBlocks * kWarps, n = (uint32_t) L.sizes.size();
    share_start(L.q, &L.s_live[block]);
    uint32_t first = block * kWarps + warp;
    bool listed = true;
    while (true) {
        uint2 task = make_uint2(0u, 1u);
        if (listed) {
            const uint32_t it = first != kNone ? first : warps + atomicAdd(&L.work, 1u);
            first = kNone;
            if (it < n) {
                task.x = it;
            } else {
                listed = false;
                share_wait_live(&L.s_live[block]);
            }
        }
        if (!listed) {
            task = take_task(L.q);
            if (task.x == kNone) break;
            if (task.x >= n || task.y >= L.done[task.x].size()) {
                L.stale = true;
                continue;
            }
        }
        unsigned long long queue = share_look(L.q, &L.s_live[block]);
        uint32_t fr[64];
        int sp = 1;
        fr[0] = task.y;
        while (sp > 0) {
            if (sp == 2) {
                if (waiting(queue) > 0) sp = offer_tasks(L.q, 1, task.x, nullptr, 0xFFFFFFFFu, fr, sp);
                queue = share_look(L.q, &L.s_live[block]);
                if (sp == 0) break;
            }
            const uint32_t k = fr[--sp];
            ++L.done[task.x][k];
            for (uint32_t c = 2 * k; c < 2 * k + 2; ++c)
                if (c < L.done[task.x].size()) fr[sp++] = c;
            model::step();
        }
    }
}

}  // namespace

int main(int argc, char** argv) {
    const int schedules = std::atoi(argv[1]);
    std::mt19937 rng((uint32_t) std::atoi(argv[2]));
    auto below = [&](uint32_t n) { return (uint32_t) (rng() % n); };
    uint32_t lost = 0, twice = 0, stale = 0, left = 0, errors = 0, hung = 0;
    for (int s = 0; s < schedules; ++s) {
        // tickets run on from launch to launch, over the wrap of their 31 bits too
        unsigned long long word = s & 1 ? 0x7FFFFFFA7FFFFFFAull : 0ull;
        std::vector<ulonglong2> slots(kSlots, ulonglong2{~0ull, ~0ull});
        uint32_t err = 0;
        for (int l = 0; l < 3; ++l) {
            Launch L;
            L.q.queue = &word;
            L.q.live = &L.live;
            L.q.over = &L.over;
            L.q.err = &err;
            L.q.slot = slots.data();
            L.q.slots = kSlots;
            L.q.most_waiting = 1 + below(kBlocks * kWarps);
            const uint32_t items = below(6);
            for (uint32_t i = 0; i < items; ++i) {
                L.sizes.push_back(1 + below(below(3) ? 6 : 150));
                L.done.emplace_back(L.sizes.back() + 1, 0u);
            }
            std::vector<model::Fiber*> fibers;
            for (uint32_t b = 0; b < kBlocks; ++b) {
                const uint32_t at = b ? below(120) : 0;  // the block's start
                for (uint32_t w = 0; w < kWarps; ++w)
                    fibers.push_back(model::spawn([&L, b, w] { warp_loop(L, b, w); }, b, w, kBlocks, kWarps, at));
            }
            if (!model::run(fibers, rng)) ++hung;
            for (uint32_t i = 0; i < items; ++i)
                for (uint32_t k = 1; k <= L.sizes[i]; ++k) {
                    lost += L.done[i][k] == 0;
                    twice += L.done[i][k] > 1;
                }
            stale += L.stale;
            left += waiting(word) < 0;
            errors += err != 0;
            err = 0;
        }
    }
    if (lost) std::printf("nodes lost: %u\n", lost);
    if (twice) std::printf("nodes expanded twice: %u\n", twice);
    if (stale) std::printf("launches that took an earlier one's task: %u\n", stale);
    if (left) std::printf("launches that left a task: %u\n", left);
    if (errors) std::printf("error bits: %u\n", errors);
    if (hung) std::printf("launches that did not end: %u\n", hung);
    return lost || twice || stale || left || errors || hung;
}
