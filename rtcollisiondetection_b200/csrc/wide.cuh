// wide.cuh - a warp's descent of a 4-wide tree (the scene's or a link's) through
// a shared LIFO frontier, generic in the node-box test.
#pragma once
#include "rtcd_internal.cuh"

namespace rtcd {

constexpr int kWideBatch = 2;  // child records a lane loads before testing them

// BATCH rounds of a warp's descent: in each, every lane tests one child record
// (a, b) - (lo.x, lo.y, lo.z, hi.x), (hi.y, hi.z, bits(ref), 0); ref kNone in an
// empty slot or a lane without a record; overlapping internal children are
// pushed on the frontier fr[0, sp), leaves appended to cb[nc, ...), both with
// the lane's tag.  Returns false, with the error flag set, if the frontier
// would overflow (which frontier_reserve's rule excludes).
template <int BATCH, class Test>
__device__ __forceinline__ bool record_rounds(const float4* a, const float4* b, uint32_t tag, uint32_t* fr, int& sp,
                                              uint32_t* cb, int& nc, Test& test, int cap, uint32_t* err,
                                              uint32_t& n_node) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    bool h[BATCH];
#pragma unroll
    for (int r = 0; r < BATCH; ++r) {
        h[r] = false;
        const uint32_t ref = __float_as_uint(b[r].z);
        Box bx;
        bx.lo[0] = a[r].x; bx.lo[1] = a[r].y; bx.lo[2] = a[r].z;
        bx.hi[0] = a[r].w; bx.hi[1] = b[r].x; bx.hi[2] = b[r].y;
        if (ref != kNone) {
            ++n_node;
            h[r] = test(bx);
        }
    }
#pragma unroll
    for (int r = 0; r < BATCH; ++r) {
        const uint32_t ref = __float_as_uint(b[r].z);
        const bool push = h[r] && !(ref & kLeaf), emit = h[r] && (ref & kLeaf);
        const uint32_t mp = __ballot_sync(0xffffffffu, push), me = __ballot_sync(0xffffffffu, emit);
        if (sp + __popc(mp) > cap) {
            if (lane == 0) atomicOr(err, kErrStack);
            return false;
        }
        if (push) fr[sp + __popc(mp & lt)] = tag | ref;
        if (emit) cb[nc + __popc(me & lt)] = tag | (ref & ~kLeaf);
        sp += __popc(mp);
        nc += __popc(me);
    }
    return true;
}

// One step of a warp's descent of a 4-wide tree through a shared LIFO frontier
// fr[0, sp): pops up to 32 nodes (as many as frontier_reserve's rule allows) and
// spreads their children over the lanes (4 lanes per node when at most 8 are
// waiting, 2 when at most 16, else one lane tests all four children of its
// node, so a step costs about one box test per lane); at most 32 * kWide leaves
// are appended per step.  Entries may carry a tag (TAGGED: the top kTagBits
// bits; a pair's candidate), which the test is bound to before its boxes and
// which the children inherit.
constexpr int kTagBits = 5;
constexpr uint32_t kTagShift = 32 - kTagBits;
constexpr uint32_t kTagRef = (1u << kTagShift) - 1u;  // the reference below the tag

template <bool TAGGED, class Test>
__device__ __forceinline__ bool frontier_step(const float4* __restrict__ wn, uint32_t* fr, int& sp, uint32_t* cb, int& nc,
                                              Test& test, int cap, int reserve, uint32_t* err, uint32_t& n_node) {
    const int lane = threadIdx.x & 31;
    const int lg = sp <= 8 ? 2 : (sp <= 16 ? 1 : 0), g = 1 << lg;
    const int take = min(min(sp, 32 >> lg), max(1, (cap - reserve - sp) / (kWide - 1)));
    sp -= take;
    const int j = lane >> lg;
    const uint32_t entry = j < take ? fr[sp + j] : 0u;
    const uint32_t node = TAGGED ? entry & kTagRef : entry;
    const uint32_t tag = TAGGED ? entry & ~kTagRef : 0u;
    const bool on = j < take && test.wants(tag >> kTagShift);  // an entry nobody wants any more is dropped
    __syncwarp();
    const int rounds = kWide >> lg;
    const float4* rec = wn + 2ull * (kWide * (size_t) node + (lane & (g - 1)));
    if (on) test.bind(tag >> kTagShift);
    bool ok = true;
    // two records at a time: with all four the kernel outgrows the instruction cache (stalls on
    // instruction fetch were 5.3 of 13 cycles per issue), one leaves the loads' latency exposed
#pragma unroll 1
    for (int r0 = 0; r0 < rounds; r0 += kWideBatch) {
        float4 a[kWideBatch], b[kWideBatch];
#pragma unroll
        for (int r = 0; r < kWideBatch; ++r) {
            b[r] = make_float4(0.f, 0.f, __uint_as_float(kNone), 0.f);
            if (on && r0 + r < rounds) {
                a[r] = __ldg(rec + 2 * (r0 + r) * g);
                b[r] = __ldg(rec + 2 * (r0 + r) * g + 1);
            }
        }
        ok = record_rounds<kWideBatch>(a, b, tag, fr, sp, cb, nc, test, cap, err, n_node);
        if (!ok) break;
    }
    __syncwarp();
    return ok;
}

// The first step of such a descent: the tree's top cut (at most kWideCut child
// records that cover every root-leaf path), one record per lane and round.
template <class Test>
__device__ __forceinline__ bool frontier_cut(const float4* __restrict__ cut, uint32_t n_cut, uint32_t* fr, int& sp,
                                             uint32_t* cb, int& nc, Test& test, int cap, uint32_t* err,
                                             uint32_t& n_node) {
    const int lane = threadIdx.x & 31;
    bool ok = true;
    test.bind(0u);
#pragma unroll 1
    for (uint32_t i = lane; i - lane < n_cut; i += 32) {
        float4 a, b = make_float4(0.f, 0.f, __uint_as_float(kNone), 0.f);
        if (i < n_cut) {
            a = __ldg(cut + 2ull * i);
            b = __ldg(cut + 2ull * i + 1);
        }
        if (!record_rounds<1>(&a, &b, 0u, fr, sp, cb, nc, test, cap, err, n_node)) {
            ok = false;
            break;
        }
    }
    __syncwarp();
    return ok;
}

}  // namespace rtcd
