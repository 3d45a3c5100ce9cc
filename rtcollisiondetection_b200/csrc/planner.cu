// planner.cu - the planner-side caller of the detectors: roadmap samples,
// nearest-neighbour edges and batched straight-line edge checks.
//
// The reference's planner tooling samples the configuration space with a
// Halton sequence (RTCD/Planner/sampler/sampler.h:11-82), links every sample
// to its K weighted nearest neighbours on the GPU (RTCD/Planner/KNN/
// knnCUDA.cu: all-pairs weighted squared distances, self and masked points
// excluded, a partial insertion sort, square roots), and turns each edge
// into a straight line of evenly spaced configurations that it checks as a
// trajectory (RTCD/Utils/Test/poseUtils.h:115-141).  Here the neighbour search
// is one kernel, a lane per query (k_knn), and an edge check interpolates the
// edges on the device and runs the detector over them in one call.
#include <algorithm>
#include <cfloat>
#include <vector>

#include "../../include/rtcd.h"
#include "kernels.h"

namespace rtcd {

// Squared axis weights, a kernel parameter (unused axes zero).
struct KnnWeights {
    float w2[kKnnMaxDim];
};

constexpr int kKnnBuf = 8;    // points a lane lets wait before the warp inserts them
constexpr int kKnnStep = 4;   // reference points per inner step

// Two FP32 operations in one instruction, each half rounded as the scalar one.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The smaller of two, NaN when either is.
__device__ __forceinline__ float min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// Shared memory of one warp: the lanes' ordered lists [k][32], their waiting
// points [kKnnBuf][32] and the warp's 32 reference points [dim + 1][32].
__host__ __device__ constexpr size_t knn_warp_bytes(uint32_t k, uint32_t dim) {
    return 256ull * k + 128ull * kKnnBuf + 128ull * (dim + 1);
}

// A block answers 32 queries, one per lane; its warps share the queries and
// split the reference points.  A warp stages 32 points at a time in shared
// memory and every lane reads each of them (a broadcast).
//
// A point r is passed over when a lower bound of its distance is above the
// lane's bound: with N(x) = sum w2 x^2 the squared distance is N(q) + N(r) -
// 2 sum w2 q r, one multiply-add per axis instead of the three operations of
// w2 (r - q)^2, and both N are shrunk by kKnnSlack(dim), which covers every
// rounding of either form (relative to N(q) + N(r), with u = 2^-24: the norms
// (dim + 2) u, the sum 2 (dim + 1) u, the bound's difference u, and, while the
// bound is at most 4 (N(q) + N(r)), 4 (dim + 5) u from the direct form's own
// rounding; a larger bound lets the point through by itself).  What is
// let through waits in a small buffer; when a lane's is full the warp computes
// the distances themselves, in the direct form, and inserts them, so the lanes'
// insertions run together.  Norms above 1e37 and NaNs make the test let
// everything through.
//
// The bound of a query is the smaller of its warp's k-th distance and the
// largest, over the block's warps, of the distance in place ceil(k / warps):
// each warp holds that many pairs within it, so all together hold k.  (The
// k-th distance of one warp's share of the points alone lets several times as
// many pairs through.)  A sample of the points gives the first bound.  The
// warps' lists are merged at the end.  Pairs are 64-bit keys (distance bits,
// index): distances are never negative, so key order is by distance, then by
// index, which is the order the reference's insertion sort settles ties in; a
// NaN sorts after the empty entry and never enters.
//
// Bound by instruction issue.  20,000 points of 7 axes, k = 10: one warp per
// query with a list per lane in local memory (about 1,300 divergent insertion
// steps per query) 4,406 us; the direct form for every pair here 557 us; this
// form 452 us.
__host__ __device__ constexpr float knn_slack(int dim) { return (float) (8 * dim + 32) / 16777216.0f; }

template <int DIM>
__global__ void __launch_bounds__(1024) k_knn(const float* __restrict__ pts, uint32_t n, const KnnWeights wt, uint32_t k,
                                              const uint8_t* __restrict__ mask, uint32_t* __restrict__ idx,
                                              float* __restrict__ dist) {
    extern __shared__ __align__(16) uint64_t s_dyn[];
    __shared__ float s_rank[32][32];  // [warp][query] distance of the warp's entry number `share`
    __shared__ float s_q[DIM][32];    // the queries
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const size_t stride = knn_warp_bytes(k, DIM) / 8;
    uint64_t* list = s_dyn + stride * warp;
    uint32_t* buf = reinterpret_cast<uint32_t*>(list + 32 * k);
    float* tile = reinterpret_cast<float*>(buf + 32 * kKnnBuf);
    const uint64_t empty = ((uint64_t) __float_as_uint(FLT_MAX) << 32) | 0xFFFFFFFFu;
    const float nan = __uint_as_float(0x7FC00000u), inf = __uint_as_float(0x7F800000u);
    constexpr float kKeep = 1.0f - knn_slack(DIM), kMostNorm = 1e37f;

    const uint32_t q = blockIdx.x * 32 + lane;
    const bool live = q < n && !(mask && mask[q]);
    float norm_q = 0.f;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const float v = live ? pts[(size_t) q * DIM + d] : 0.f;
        if (warp == 0) s_q[d][lane] = v;
        norm_q = fmaf(v * v, wt.w2[d], norm_q);
    }
    uint64_t m2wq[DIM];  // -2 w2 q, twice each
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const float v = live ? pts[(size_t) q * DIM + d] : 0.f;
        const float m = norm_q <= kMostNorm ? -2.f * wt.w2[d] * v : nan;
        m2wq[d] = pack2(m, m);
    }
    norm_q *= kKeep;
    for (uint32_t j = 0; j < k; ++j) list[j * 32 + lane] = empty;
    __syncthreads();

    const uint32_t share = (k + warps - 1) / warps;
    float bound = FLT_MAX, limit = live ? FLT_MAX : -inf;  // limit: the bound less the query's norm
    int held = 0;
    auto set_bound = [&](float b) {
        if (b < bound) {
            bound = b;
            limit = live ? b - norm_q + 1e-36f : -inf;  // 1e-36: above the roundings of subnormal terms
        }
    };
    auto tighten = [&] {
        float joint = 0.f;
        for (int w = 0; w < warps; ++w) joint = fmaxf(joint, *(volatile float*) &s_rank[w][lane]);
        set_bound(joint);
    };
    float rank = FLT_MAX;
    auto publish = [&](float v) {
        rank = fminf(rank, v);
        *(volatile float*) &s_rank[warp][lane] = rank;
    };
    auto insert_held = [&] {
        for (int e = 0; e < held; ++e) {
            const uint32_t r = buf[e * 32 + lane];
            if (!live || r == q || r >= n || (mask && mask[r])) continue;
            float s = 0.f;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const float t = __fsub_rn(__ldg(pts + (size_t) r * DIM + d), s_q[d][lane]);
                s = __fmaf_rn(__fmul_rn(t, t), wt.w2[d], s);
            }
            const uint64_t key = ((uint64_t) __float_as_uint(s) << 32) | r;
            // one pass over the list: every entry is read whatever the others hold, so the reads
            // overlap (a search from the end waits for each entry before the next)
            uint64_t cur = list[(k - 1) * 32 + lane];
            bool below = key < cur;
            if (!below) continue;
#pragma unroll 4
            for (int j = (int) k - 1; j > 0; --j) {
                const uint64_t up = list[(j - 1) * 32 + lane];
                const bool next_below = key < up;
                list[j * 32 + lane] = next_below ? up : (below ? key : cur);
                cur = up;
                below = next_below;
            }
            list[lane] = below ? key : cur;
        }
        held = 0;
        set_bound(__uint_as_float((uint32_t) (list[(k - 1) * 32 + lane] >> 32)));
        publish(__uint_as_float((uint32_t) (list[(share - 1) * 32 + lane] >> 32)));
    };

    // the warps take the 32-point tiles in turn; a lane loads one point of a tile
    const uint32_t tiles = (n + 31) / 32;
    float next[DIM];
    bool next_on;
    auto load_tile = [&](uint32_t t) {
        const uint32_t r = t * 32 + lane;
        next_on = t < tiles && r < n && !(mask && mask[r]);
#pragma unroll
        for (int d = 0; d < DIM; ++d) next[d] = next_on ? __ldg(pts + (size_t) r * DIM + d) : 0.f;
    };
    auto store_tile = [&] {  // the points, then their shrunken norms (infinite: no point)
        float norm = 0.f;
        __syncwarp();
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            tile[d * 32 + lane] = next[d];
            norm = fmaf(next[d] * next[d], wt.w2[d], norm);
        }
        tile[DIM * 32 + lane] = !next_on ? inf : norm <= kMostNorm ? norm * kKeep : nan;
        __syncwarp();
    };

    // the lower bounds, less the query's norm, of points r0 .. r0 + 3 of the tile
    auto lower = [&](int r0, float* s, float* norm) {
        const ulonglong2 nr = *reinterpret_cast<const ulonglong2*>(tile + DIM * 32 + r0);
        uint64_t s01 = nr.x, s23 = nr.y;
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(tile + d * 32 + r0);
            s01 = fma2(p.x, m2wq[d], s01);
            s23 = fma2(p.y, m2wq[d], s23);
        }
        const float2 a = unpack2(s01), b = unpack2(s23), c = unpack2(nr.x), d = unpack2(nr.y);
        s[0] = a.x; s[1] = a.y; s[2] = b.x; s[3] = b.y;
        norm[0] = c.x; norm[1] = c.y; norm[2] = d.x; norm[3] = d.y;
    };

    // a first bound from a sample of the warp's points: upper bounds of its four smallest distances
    // (three slacks above the lower ones)
    {
        constexpr float kUp = 3.0f * knn_slack(DIM);
        const uint32_t mine = (tiles + warps - 1) / warps;
        const uint32_t sample = max(mine / 16, 1u);
        float m[4] = {FLT_MAX, FLT_MAX, FLT_MAX, FLT_MAX};
        load_tile(warp);
        for (uint32_t i = 0; i < sample; ++i) {
            const uint32_t t = warp + i * warps;
            store_tile();
            load_tile(t + warps);
#pragma unroll 2
            for (int r0 = 0; r0 < 32; r0 += kKnnStep) {
                float s[kKnnStep], norm[kKnnStep];
                lower(r0, s, norm);
#pragma unroll
                for (int j = 0; j < kKnnStep; ++j) {
                    float v = fminf(fmaf(kUp, norm[j], s[j]), FLT_MAX);  // a NaN counts as FLT_MAX
                    if (t * 32 + r0 + j == q) v = FLT_MAX;
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float up = fmaxf(m[c], v);
                        m[c] = fminf(m[c], v);
                        v = up;
                    }
                }
            }
        }
        const float mth = share == 1 ? m[0] : share == 2 ? m[1] : share == 3 ? m[2] : share == 4 ? m[3] : FLT_MAX;
        publish(fminf(fmaxf(mth + fmaf(kUp, norm_q, norm_q), 0.f) + 1e-36f, FLT_MAX));
    }
    __syncthreads();

    load_tile(warp);
    for (uint32_t t = warp; t < tiles; t += warps) {
        store_tile();
        load_tile(t + warps);
        tighten();
#pragma unroll 2
        for (int r0 = 0; r0 < 32; r0 += kKnnStep) {
            float s[kKnnStep], norm[kKnnStep];
            lower(r0, s, norm);
            if (__any_sync(0xffffffffu, !(min_nan(min_nan(s[0], s[1]), min_nan(s[2], s[3])) > limit))) {
#pragma unroll
                for (int j = 0; j < kKnnStep; ++j)
                    if (!(s[j] > limit)) buf[32 * held++ + lane] = t * 32 + r0 + j;
                if (__any_sync(0xffffffffu, held > kKnnBuf - kKnnStep)) {
                    insert_held();
                    tighten();
                }
            }
        }
    }
    insert_held();
    __syncthreads();

    // merge: `warps` neighbouring lanes (a power of two) per query, one list each
    const int group = threadIdx.x / warps, member = threadIdx.x % warps;  // blockDim.x / warps = 32 queries
    const uint64_t* mine = s_dyn + stride * member + group;
    const uint32_t out_q = blockIdx.x * 32 + group;
    uint32_t head = 0;
    for (uint32_t out = 0; out < k; ++out) {
        const uint64_t top = head < k ? mine[head * 32] : empty;
        uint64_t best = top;
        for (int o = warps >> 1; o > 0; o >>= 1) {
            const uint64_t other = __shfl_xor_sync(0xffffffffu, best, o);
            best = other < best ? other : best;
        }
        if (top == best && head < k) ++head;  // keys are unique, so one list advances
        if (member == 0 && out_q < n) {
            const float v = __uint_as_float((uint32_t) (best >> 32));
            idx[(size_t) out_q * k + out] = (uint32_t) best;
            dist[(size_t) out_q * k + out] = v < FLT_MAX ? sqrtf(v) : FLT_MAX;
        }
    }
}

// Edge e = (a, b) as n_wp evenly spaced configurations a + (b - a) / (n_wp - 1) * i.
__global__ void k_interp_edges(const float* __restrict__ nodes, uint32_t n_nodes, uint32_t dof,
                               const uint32_t* __restrict__ edges, uint32_t n_edges, uint32_t n_wp,
                               float* __restrict__ q, uint32_t* __restrict__ err) {
    const size_t total = (size_t) n_edges * n_wp;
    for (size_t t = blockIdx.x * (size_t) blockDim.x + threadIdx.x; t < total; t += (size_t) gridDim.x * blockDim.x) {
        const uint32_t e = (uint32_t) (t / n_wp), i = (uint32_t) (t - (size_t) e * n_wp);
        const uint32_t a = edges[2ull * e], b = edges[2ull * e + 1];
        if (a >= n_nodes || b >= n_nodes) {
            atomicOr(err, kErrRange);
            for (uint32_t d = 0; d < dof; ++d) q[t * dof + d] = 0.f;
            continue;
        }
        for (uint32_t d = 0; d < dof; ++d) {
            const float s = nodes[(size_t) a * dof + d];
            const float span = (nodes[(size_t) b * dof + d] - s) / (float) (n_wp - 1);
            q[t * dof + d] = s + span * (float) i;
        }
    }
}

// The search among few points (at most 32 * PER): a warp per query, PER keys a lane in registers, and k rounds
// of a minimum over the warp, in which the lane that gave the smallest key looks for its next one.  Keys and their
// order as in k_knn, whose ordered insertions, one lane's after the other, are the longer chain here (7 axes,
// whole call: 100 points, k = 10, 30 us against 15; k = 32, 46 against 18; 1,000 points, k = 10, 49 against
// 24.  A list per lane in local memory took 26, 35 and 78).
constexpr int kKnnFewWarps = 2;
template <int PER>
__global__ void __launch_bounds__(kKnnFewWarps * 32) k_knn_few(const float* __restrict__ pts, uint32_t n, uint32_t dim,
                                                               const KnnWeights wt, uint32_t k, const uint8_t* __restrict__ mask,
                                                               uint32_t* __restrict__ idx, float* __restrict__ dist) {
    const uint32_t lane = threadIdx.x & 31, q = blockIdx.x * kKnnFewWarps + threadIdx.x / 32;
    if (q >= n) return;  // warp-uniform
    const uint64_t empty = ((uint64_t) __float_as_uint(FLT_MAX) << 32) | 0xFFFFFFFFu;
    const bool live = !(mask && mask[q]);
    float s[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) s[i] = 0.f;
    for (uint32_t d = 0; d < dim; ++d) {
        const float qd = __ldg(pts + (size_t) q * dim + d), w2 = wt.w2[d];
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const uint32_t r = 32 * i + lane;
            const float t = r < n ? __fsub_rn(__ldg(pts + (size_t) r * dim + d), qd) : 0.f;
            s[i] = __fmaf_rn(__fmul_rn(t, t), w2, s[i]);
        }
    }
    uint64_t key[PER], best = empty;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const uint32_t r = 32 * i + lane;
        const uint64_t at = ((uint64_t) __float_as_uint(s[i]) << 32) | r;
        key[i] = live && r < n && r != q && !(mask && mask[r]) && at < empty ? at : empty;
        best = key[i] < best ? key[i] : best;
    }
    uint64_t mine = empty;  // the neighbour this lane writes
    for (uint32_t out = 0; out < k; ++out) {
        const uint32_t hi = __reduce_min_sync(0xffffffffu, (uint32_t) (best >> 32));
        const uint32_t lo = __reduce_min_sync(0xffffffffu, (uint32_t) (best >> 32) == hi ? (uint32_t) best : 0xFFFFFFFFu);
        const uint64_t top = ((uint64_t) hi << 32) | lo;
        if (lane == out) mine = top;
        if (top == best) {  // one lane's, unless empty
            best = empty;
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                if (key[i] == top) key[i] = empty;
                best = key[i] < best ? key[i] : best;
            }
        }
    }
    if (lane < k) {
        const float v = __uint_as_float((uint32_t) (mine >> 32));
        idx[(size_t) q * k + lane] = (uint32_t) mine;
        dist[(size_t) q * k + lane] = v < FLT_MAX ? sqrtf(v) : FLT_MAX;
    }
}

template <int PER>
static void launch_knn_few(const float* pts, uint32_t n, uint32_t dim, const KnnWeights& w, uint32_t k, const uint8_t* mask,
                           uint32_t* idx, float* dist, cudaStream_t s) {
    k_knn_few<PER><<<(n + kKnnFewWarps - 1) / kKnnFewWarps, kKnnFewWarps * 32, 0, s>>>(pts, n, dim, w, k, mask, idx, dist);
    cuda_check(cudaGetLastError(), "k_knn_few");
}

// flags[e] = OR of the pose flags of edge e's n_wp configurations
__global__ void k_or_rows(const uint8_t* __restrict__ pose_flags, uint32_t n_edges, uint32_t n_wp,
                          uint8_t* __restrict__ flags) {
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n_edges) return;
    uint8_t f = 0;
    for (uint32_t i = 0; i < n_wp; ++i) f |= pose_flags[(size_t) e * n_wp + i];
    flags[e] = f;
}

// Warps per block, a power of two: eight fill the SMs once there are two blocks
// of 32 queries for each; with fewer blocks the points are split over more
// warps, as far as every warp has a tile of them and the shared memory of a
// block allows.
template <int DIM>
static void launch_knn_dim(const float* pts, uint32_t n, const KnnWeights& w, uint32_t k, const uint8_t* mask,
                           uint32_t* idx, float* dist, cudaStream_t s) {
    constexpr size_t kMost = 200 * 1024;
    constexpr size_t kStatic = 4 * 32 * (32 + DIM);  // k_knn's s_rank and s_q, part of a block's 48 KB without the opt-in
    const uint32_t blocks = (n + 31) / 32;
    uint32_t warps = 1;
    while (warps < 32 && 2 * warps <= blocks && (warps < 8 || blocks * warps < 16u * (uint32_t) device_sm_count()) &&
           2 * warps * knn_warp_bytes(k, DIM) <= kMost)
        warps *= 2;
    const size_t smem = warps * knn_warp_bytes(k, DIM);
    if (smem + kStatic > 47 * 1024)
        cuda_check(cudaFuncSetAttribute(k_knn<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kMost), "k_knn");
    k_knn<DIM><<<blocks, warps * 32, smem, s>>>(pts, n, w, k, mask, idx, dist);
    cuda_check(cudaGetLastError(), "k_knn");
}

template <int DIM = 1>
static void knn_dispatch(uint32_t dim, const float* pts, uint32_t n, const KnnWeights& w, uint32_t k,
                         const uint8_t* mask, uint32_t* idx, float* dist, cudaStream_t s) {
    if (dim == (uint32_t) DIM) return launch_knn_dim<DIM>(pts, n, w, k, mask, idx, dist, s);
    if constexpr (DIM < (int) kKnnMaxDim) knn_dispatch<DIM + 1>(dim, pts, n, w, k, mask, idx, dist, s);
}

void launch_knn(const float* pts, uint32_t n, uint32_t dim, const float* w2, uint32_t k, const uint8_t* mask,
                uint32_t* idx, float* dist, cudaStream_t s) {
    if (!n) return;
    KnnWeights w{};
    for (uint32_t d = 0; d < dim; ++d) w.w2[d] = w2[d];
    if (n <= 128) return launch_knn_few<4>(pts, n, dim, w, k, mask, idx, dist, s);
    if (n <= 512) return launch_knn_few<16>(pts, n, dim, w, k, mask, idx, dist, s);
    if (n <= 1024) return launch_knn_few<32>(pts, n, dim, w, k, mask, idx, dist, s);  // as far as its registers go
    knn_dispatch(dim, pts, n, w, k, mask, idx, dist, s);
}

void launch_interp_edges(const float* nodes, uint32_t n_nodes, uint32_t dof, const uint32_t* edges, uint32_t n_edges,
                         uint32_t n_wp, float* q, uint32_t* err, cudaStream_t s) {
    const size_t total = (size_t) n_edges * n_wp;
    if (!total) return;
    const uint32_t blocks = (uint32_t) std::min<size_t>((total + 255) / 256, 148u * 16u);
    k_interp_edges<<<blocks, 256, 0, s>>>(nodes, n_nodes, dof, edges, n_edges, n_wp, q, err);
    cuda_check(cudaGetLastError(), "k_interp_edges");
}

void launch_or_rows(const uint8_t* pose_flags, uint32_t n_edges, uint32_t n_wp, uint8_t* flags, cudaStream_t s) {
    if (!n_edges) return;
    k_or_rows<<<(n_edges + 255) / 256, 256, 0, s>>>(pose_flags, n_edges, n_wp, flags);
    cuda_check(cudaGetLastError(), "k_or_rows");
}

}  // namespace rtcd

namespace {

// The reference's Halton radical inverse, with its float arithmetic
// (RTCD/Planner/sampler/sampler.h:11-25).
float halton(int n, int b) {
    float hn = 0;
    int n0 = n;
    float f = 1 / ((float) b);
    while (n0 > 0) {
        float n1 = (float) (n0 / b);
        int r = n0 - (int) (n1 * (float) b);
        hn += f * (float) r;
        f = f / (float) b;
        n0 = (int) n1;
    }
    return hn;
}

}  // namespace

extern "C" {

rtcd_status rtcd_halton_samples(uint32_t n, uint32_t dim, uint32_t skip, const float* lower, const float* upper,
                                float* out) {
    static const int kPrimes[25] = {2,  3,  5,  7,  11, 13, 17, 19, 23, 29, 31, 37, 41,
                                    43, 47, 53, 59, 61, 67, 71, 73, 79, 83, 89, 97};
    try {
        if (!lower || !upper || (n && !out)) rtcd::fail(RTCD_ERR_INVALID_ARGUMENT, "NULL argument");
        if (skip + dim > 25) rtcd::fail(RTCD_ERR_INVALID_ARGUMENT, "skip + dim must be at most 25 (prime bases)");
        for (uint32_t d = 0; d < dim; ++d)
            for (uint32_t i = 0; i < n; ++i)
                out[(size_t) i * dim + d] = halton((int) i, kPrimes[d + skip]) * (upper[d] - lower[d]) + lower[d];
        rtcd::set_last_error("");
        return RTCD_OK;
    } catch (const rtcd::Error& e) {
        rtcd::set_last_error(e.msg);
        return (rtcd_status) e.status;
    }
}

}  // extern "C"
