// share.cuh - work sharing between the warps of a persistent launch.
//
// A warp that finds its launch's list empty takes a ticket and waits on that
// ticket's slot.  A busy warp that sees more tickets taken than tasks offered
// hands entries of its frontier (task: two words, the owner's and a tree node)
// to the waiting warps, one each.  The warp whose ticket makes every live warp a
// waiting one ends all of them.  Live are the warps of the blocks that have
// started: blocks still waiting for room beside another launch's are not waited
// for, and work through their own first entries after the end.  A warp that
// finds enough others waiting leaves.  A waiting warp gives up after a bounded
// time; what is offered to a ticket that was given up stays with the warp that
// offered it.
//
// Offers follow a sight of the queue that is a step old, so a task may go to a
// ticket that nobody has taken yet, before the end or after it.  No warp leaves
// while more tasks are offered than tickets taken: the last one to have offered
// looks after its offers, takes such a ticket and finds the task there.  So every
// task runs, whatever the counts of live and waiting warps said meanwhile, and a
// launch leaves no task behind for the next one.
#pragma once
#include "kernels.h"

namespace rtcd {

constexpr uint32_t kShareTagShift = 27;  // an entry's tag above its node (wide.cuh)
constexpr int kSharePolls = 1 << 16;  // polls of a word before a wait gives up

// A slot is two 64-bit words, each with the ticket (plus one) it was written
// for in its high half, so a reader knows from each word alone whether it is
// the one it looks for and no fence orders them.  Second word: the node.  First
// word: the owner's word, or the state of the ticket.  Whoever comes first, the
// ticket's warp (kWaiting) or the one that serves or ends the ticket, replaces
// the first word once the slot's last ticket is done with it (free), the other
// replaces the first one's; each with a compare-and-swap.  Tickets run on from
// launch to launch, so slots are never cleared between them.
//
// The queue word is read, added to and swapped as 64 bits: tickets taken in bits
// 0 to 30, tasks offered in bits 32 to 62, both modulo 2^31.  Bit 31 takes the
// carry of the first; whoever caused it clears it.
constexpr uint32_t kTaken = 0xFFFFFFFFu, kGivenUp = 0xFFFFFFFEu, kWaiting = 0xFFFFFFFDu;
__device__ __forceinline__ unsigned long long slot_word(uint32_t t, uint32_t v) {
    return ((unsigned long long) (t + 1) << 32) | v;
}
__device__ __forceinline__ bool slot_free(unsigned long long w) { return (uint32_t) w >= kGivenUp; }
__device__ __forceinline__ unsigned long long look(const unsigned long long* p) {
    return *(const volatile unsigned long long*) p;
}

constexpr uint32_t kTicketMask = 0x7FFFFFFFu;
__device__ __forceinline__ uint32_t taken(unsigned long long q) { return (uint32_t) q & kTicketMask; }
__device__ __forceinline__ uint32_t offered(unsigned long long q) { return (uint32_t) (q >> 32) & kTicketMask; }
// Tickets taken beyond the tasks offered: warps waiting for work.
__device__ __forceinline__ int waiting(unsigned long long q) { return (int) ((taken(q) - offered(q)) << 1) >> 1; }

// Puts v into the slot of ticket t: false when its warp gave up.
__device__ __forceinline__ bool serve(const TaskQueue& Q, uint32_t t, uint32_t v, uint32_t node) {
    ulonglong2* slot = Q.slot + (t & (Q.slots - 1));
    unsigned long long w = look(&slot->x);
    for (int polls = 0; polls < kSharePolls; ++polls) {
        if (w == slot_word(t, kGivenUp)) return false;
        if (w == slot_word(t, kWaiting) || slot_free(w)) {  // else the last ticket's warp is reading its task
            *(volatile unsigned long long*) &slot->y = slot_word(t, node);
            const unsigned long long was = atomicCAS(&slot->x, w, slot_word(t, v));
            if (was == w) return true;
            w = was;
        } else {
            w = look(&slot->x);
        }
    }
    return false;
}

// Ends the launch when every live warp waits (one lane calls): every ticket taken
// counts as served, and the waiting warps see Q.over.
__device__ __forceinline__ void end_if_all_wait(const TaskQueue& Q) {
    __threadfence();  // this warp's ticket, or its leaving, before what it sees of the others
    for (int tries = 0; tries < 64; ++tries) {
        const unsigned long long q = look(Q.queue);
        const int waits = waiting(q);
        if (waits < 0 || waits < (int) *(volatile uint32_t*) Q.live) return;
        if (atomicCAS(Q.queue, q, ((unsigned long long) taken(q) << 32) | taken(q)) == q) {
            *(volatile uint32_t*) Q.over = 1u;
            return;
        }
    }
}

// A warp's leaving (one lane calls).  The last one checks that no task stays behind.
__device__ __forceinline__ void leave_launch(const TaskQueue& Q) {
    if (atomicSub(Q.live, 1u) == 1u && waiting(look(Q.queue)) < 0) atomicOr(Q.err, kErrLookback);
}

// A task for an idle warp (all lanes call): (owner's word, node); (kNone, 0) when
// it is to leave: the launch is over, or enough warps wait already
// (Q.most_waiting), and no task waits for a ticket.  Out of line, like everything
// a warp does seldom: its registers would weigh on the traversal loops.
static __device__ __noinline__ uint2 take_task(const TaskQueue Q) {
    uint2 task = make_uint2(kNone, 0u);
    const int lane = threadIdx.x & 31;
    uint32_t t = 0, leave = 0;
    if (lane == 0) {
        const int waits = waiting(look(Q.queue));
        leave = waits >= (int) Q.most_waiting || (waits >= 0 && *(volatile uint32_t*) Q.over);
        if (leave) {
            leave_launch(Q);
        } else {
            t = taken(atomicAdd(Q.queue, 1ull));
            if (t == kTicketMask) atomicAnd(Q.queue, ~(1ull << 31));
        }
        end_if_all_wait(Q);
    }
    leave = __shfl_sync(0xffffffffu, leave, 0);
    if (leave) return task;
    uint32_t got = 0;
    if (lane == 0) {
        ulonglong2* slot = Q.slot + (t & (Q.slots - 1));
        const unsigned long long wait = slot_word(t, kWaiting);
        uint32_t nap = 100;
        unsigned long long w = 0;
        for (int polls = 0;; ++polls) {
            w = look(&slot->x);
            if ((uint32_t) (w >> 32) == t + 1 && w != wait) break;  // served
            const bool gives_up = polls >= kSharePolls || *(volatile uint32_t*) Q.over;
            const unsigned long long given = slot_word(t, kGivenUp);
            if (w == wait || slot_free(w)) {
                if (gives_up) {  // unless a task arrives just now
                    if (atomicCAS(&slot->x, w, given) != w) continue;
                    w = given;
                    leave_launch(Q);
                    break;
                }
                if (w != wait) {  // first here
                    atomicCAS(&slot->x, w, wait);
                    continue;
                }
            } else if (polls < 2 * kSharePolls) {
                continue;  // the slot's last warp is reading its task
            } else {  // or never did: a task put here later would be lost
                atomicOr(Q.err, kErrLookback);
                w = given;
                break;
            }
            __nanosleep(nap);
            nap = min(2 * nap, 800u);
        }
        if ((uint32_t) w < kWaiting) {
            task.x = (uint32_t) w;
            // written before the first word, so it is here or on its way
            for (int polls = 0; polls < kSharePolls; ++polls) {
                w = look(&slot->y);
                if ((uint32_t) (w >> 32) == t + 1) break;
            }
            if ((uint32_t) (w >> 32) != t + 1) atomicOr(Q.err, kErrLookback);
            else got = 1;
            task.y = (uint32_t) w;
            atomicExch(&slot->x, slot_word(t, kTaken));
        }
    }
    task.x = __shfl_sync(0xffffffffu, task.x, 0);
    task.y = __shfl_sync(0xffffffffu, task.y, 0);
    if (!__shfl_sync(0xffffffffu, got, 0)) task.x = kNone;
    return task;
}

// Hands up to `most` (at most 32) of the oldest of the entries fr[0, sp) to waiting
// warps, or to the next ones that will be idle.  An entry's node is its low bits
// (mask); its owner's word, below kWaiting, is owners[its tag] (the bits above
// the mask), or `owner` for every entry when owners is NULL.  Returns the new sp.
static __device__ __noinline__ int offer_tasks(const TaskQueue Q, int most, uint32_t owner, const uint32_t* owners, uint32_t mask,
                                        uint32_t* fr, int sp) {
    const int lane = threadIdx.x & 31;
    // every warp may offer once on one sight of the same waiting warps, and all of it fits the slots
    const int give = min(min(most, 32), (int) (Q.slots / (gridDim.x * (blockDim.x / 32))));
    uint32_t t0 = 0;
    if (lane == 0) t0 = offered(atomicAdd(Q.queue, (unsigned long long) give << 32));
    t0 = __shfl_sync(0xffffffffu, t0, 0);
    uint32_t entry = 0;
    bool kept = false;
    if (lane < give) {
        entry = fr[lane];
        kept = !serve(Q, (t0 + lane) & kTicketMask, owners ? owners[entry >> kShareTagShift] : owner, entry & mask);
    }
    const uint32_t mkept = __ballot_sync(0xffffffffu, kept);
    const int back = __popc(mkept);
    // the entries kept, then the rest moved down
    for (int i = 0; i < sp - give; i += 32) {
        const bool on = i + lane < sp - give;
        const uint32_t v = on ? fr[give + i + lane] : 0u;
        __syncwarp();
        if (on) fr[back + i + lane] = v;
        __syncwarp();
    }
    if (kept) fr[__popc(mkept & ((1u << lane) - 1u))] = entry;
    __syncwarp();
    return sp - (give - back);
}

// The block counts as live before a warp of it can be idle (all threads call, at
// the start; s_live: a shared word).
__device__ __forceinline__ void share_start(const TaskQueue& Q, volatile uint32_t* s_live) {
    if (threadIdx.x == 0) *s_live = 0;
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(Q.live, blockDim.x / 32) != kNone) *s_live = 1;  // set once it has returned
}
__device__ __forceinline__ void share_wait_live(const volatile uint32_t* s_live) {
    for (int polls = 0; !*s_live && polls < kSharePolls; ++polls) {}
}
// A sight of the queue (one lane calls): no waiting warps until the block counts as live.
__device__ __forceinline__ unsigned long long share_look(const TaskQueue& Q, const volatile uint32_t* s_live) {
    return *s_live ? look(Q.queue) : 0ull;
}

}  // namespace rtcd
