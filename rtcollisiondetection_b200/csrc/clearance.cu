// clearance.cu - the scene's clearance grid, read by the cull of k_prepare
// (discrete.cu): for each cell of a grid over the scene's box a lower bound of
// the distance from any point of the cell to the nearest triangle.
//
// Cells that a triangle touches are marked; the distance between two cells'
// boxes is the root of the sum of their squared gaps along the axes, so three
// passes, one per axis, give every cell the gap to its nearest marked cell
// (a minimum over a line of cells of a value plus a squared gap; the usual
// separable distance transform).
#include <algorithm>
#include <cmath>

#include "kernels.h"

namespace rtcd {

// Cells along the longest side of a scene of a metre or more.  The grid of a smaller one has cells of
// kClearLeast and is made and kept in proportion (a 5 cm part 0.41 ms instead of 4.7, 0.35 without a grid; a
// 1 m scene 4.7 ms, 2.9 without: 0.7 of it the kernels, 1.1 the 50 MB they need).
constexpr int kClearCells = 256;
constexpr float kClearLeast = 0.004f;  // m, a cell at least: a tenth of a covering sphere's usual radius
constexpr int kClearReach = 63;    // cells; a larger gap counts as this one
constexpr uint16_t kFar = kClearReach * kClearReach;

// Cells are marked from each triangle's box, grown by 1e-5 m, where the
// triangle's plane passes within a hundredth of a cell of the cell.  In FP64: of
// a sliver's FP32 normal little but rounding may be left, and a plane across it
// leaves out cells that it passes through.  Corners on one line (to 1e-14 of the
// sides) have no plane in FP64 either, and `rounding`, a bound of the normal's and the
// product's errors, then lets every cell of the box through.  A warp per
// triangle, a lane per row of cells, of which it looks at those near the plane: a
// ramp across the scene has 65,536 rows (one thread for its 16.7 million cells
// 867 ms, a lane per row for all of a row's cells 24 ms, this under 1 ms).
__global__ void k_clear_mark(const float* __restrict__ v, const uint32_t* __restrict__ tris, uint32_t n, ClearGrid g,
                             uint16_t* __restrict__ cells) {
    const uint32_t i = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    if (i >= n) return;
    const float *a = v + 3ull * tris[3ull * i], *b = v + 3ull * tris[3ull * i + 1], *c = v + 3ull * tris[3ull * i + 2];
    int lo[3], hi[3];
    for (int k = 0; k < 3; ++k) {
        const float l = fminf(a[k], fminf(b[k], c[k])), h = fmaxf(a[k], fmaxf(b[k], c[k]));
        lo[k] = clear_cell(g, k, l - 1e-5f);
        hi[k] = clear_cell(g, k, h + 1e-5f);
    }
    const double size = 1.0 / g.inv;
    const d3 p = dk(a[0], a[1], a[2]), e1 = dk(b[0], b[1], b[2]) - p, e2 = dk(c[0], c[1], c[2]) - p, n3 = cross(e1, e2);
    const auto sum = [](d3 v) { return fabs(v.x) + fabs(v.y) + fabs(v.z); };
    const double reach = (0.51 * size + 1e-5) * sum(n3), rounding = 1e-14 * sum(e1) * sum(e2);
    const int ny = hi[1] - lo[1] + 1, rows = ny * (hi[2] - lo[2] + 1);
    for (int r = threadIdx.x & 31; r < rows; r += 32) {
        const int y = lo[1] + r % ny, z = lo[2] + r / ny;
        const auto from_p = [&](double x) {
            return dk(g.org[0] + (x + 0.5) * size, g.org[1] + (y + 0.5) * size, g.org[2] + (z + 0.5) * size) - p;
        };
        // |n3 . d| is within `most` between u and v: these cells and one more on either side, or the whole
        // row where the plane is parallel to it or not finite
        const d3 d0 = from_p(lo[0]), d1 = from_p(hi[0]);
        const double most = reach + rounding * fmax(sum(d0), sum(d1)), at0 = dot(n3, d0), step = n3.x * size;
        const double u = (-most - at0) / step, v = (most - at0) / step, last = hi[0] - lo[0];
        if (step == 0.0 && fabs(at0) > most) continue;
        const bool cut = step != 0.0 && u == u && v == v;
        const int x0 = cut ? lo[0] + (int) fmax(0.0, fmin(last, fmin(u, v) - 1.0)) : lo[0];
        const int x1 = cut ? lo[0] + (int) fmin(last, fmax(0.0, fmax(u, v) + 1.0)) : hi[0];
        for (int x = x0; x <= x1; ++x) {
            const d3 d = from_p(x);
            if (!(fabs(dot(n3, d)) > reach + rounding * sum(d))) cells[clear_at(g, x, y, z)] = 0;
        }
    }
}

// The three passes, in place: a value becomes the minimum over the cells of its line along one axis, within
// kClearReach, of their value plus the squared gap between the two cells (in cells).  A line is read whole
// before any of it is written.  Along x the values are marked or not, so the nearest marked cell on either
// side is a bit of the line's masks; a warp takes a line.
__global__ void __launch_bounds__(128) k_clear_x(uint16_t* __restrict__ cells, ClearGrid g) {
    const uint32_t row = blockIdx.x * 4 + threadIdx.x / 32;
    if (row >= (uint32_t) g.dim[1] * (uint32_t) g.dim[2]) return;
    uint16_t* line = cells + (size_t) row * g.dim[0];
    const int lane = threadIdx.x & 31;
    uint32_t mask[kClearCells / 32 + 4];  // two empty words on either side: no bit is looked for beyond them
    mask[0] = mask[1] = mask[kClearCells / 32 + 2] = mask[kClearCells / 32 + 3] = 0;
#pragma unroll
    for (int w = 0; w < kClearCells / 32; ++w) {
        const int x = 32 * w + lane;
        mask[w + 2] = __ballot_sync(0xffffffffu, x < g.dim[0] && line[x] == 0);
    }
#pragma unroll
    for (int w = 0; w < kClearCells / 32; ++w) {
        // the 64 cells up to this one, the last in the top bit, and the 64 from this one on, the first in bit 0
        const uint64_t low = (uint64_t) mask[w + 1] << 32 | mask[w], high = (uint64_t) mask[w + 4] << 32 | mask[w + 3];
        const uint64_t below = lane == 31 ? (uint64_t) mask[w + 2] << 32 | mask[w + 1]
                                          : (uint64_t) mask[w + 2] << (63 - lane) | low >> (lane + 1);
        const uint64_t above = lane == 0 ? (uint64_t) mask[w + 3] << 32 | mask[w + 2]
                                         : (uint64_t) (mask[w + 2] >> lane) | high << (32 - lane);
        const int d = min(below ? __clzll(below) : 64, above ? __ffsll(above) - 1 : 64);
        const int x = 32 * w + lane;
        if (x < g.dim[0]) line[x] = d > kClearReach ? kFar : d > 1 ? (uint16_t) ((d - 1) * (d - 1)) : 0;
    }
}

// Along y, or along z (LAST), where the roots go to `out` in quarter cells, rounded down.  A block takes 32
// neighbouring lines.
template <bool LAST>
__global__ void __launch_bounds__(256) k_clear_line(uint16_t* __restrict__ cells, ClearGrid g, uint8_t* __restrict__ out) {
    __shared__ uint16_t s[kClearCells][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, x = blockIdx.x * 32 + lane;
    const int n = g.dim[LAST ? 2 : 1];
    const size_t first = LAST ? clear_at(g, x, blockIdx.y, 0) : clear_at(g, x, 0, blockIdx.y);
    const size_t step = LAST ? (size_t) g.dim[0] * g.dim[1] : g.dim[0];
    const bool on = x < g.dim[0];
    bool near = false;
    for (int i = warp; i < n; i += 8) {
        s[i][lane] = on ? cells[first + i * step] : kFar;
        near |= s[i][lane] < kFar;
    }
    near = __syncthreads_or(near);
    for (int i = warp; i < n && on; i += 8) {
        uint32_t best = s[i][lane];
        for (int d = 1; near && d <= kClearReach; ++d) {
            const uint32_t gap2 = (uint32_t) (d - 1) * (uint32_t) (d - 1);
            if (gap2 >= best) break;
            if (i - d >= 0) best = min(best, gap2 + s[i - d][lane]);
            if (i + d < n) best = min(best, gap2 + s[i + d][lane]);
        }
        best = min(best, (uint32_t) kFar);
        if (LAST) out[first + i * step] = (uint8_t) floorf(4.0f * sqrtf((float) best) * 0.99999f);
        else cells[first + i * step] = (uint16_t) best;
    }
}

bool build_clearance(const float* d_verts, const uint32_t* d_tris, uint32_t n_tris, const float* lo, const float* hi,
                     DevBuf& out, ClearGrid& g, cudaStream_t s) {
    g = ClearGrid{};
    if (!n_tris) return false;
    const float pad = 1e-3f;
    float longest = 0.f, most = 0.f;
    for (int k = 0; k < 3; ++k) {
        const float extent = hi[k] - lo[k] + 2 * pad;
        if (!(extent < 1e6f) || !(lo[k] > -1e6f)) return false;  // not finite, or cells beyond any use
        longest = std::max(longest, extent);
        most = std::max({most, std::fabs(lo[k]), std::fabs(hi[k])});
        g.org[k] = lo[k] - pad;
    }
    // the triangles lie below the last cells' lower sides
    g.inv = std::min((float) (kClearCells - 1) / longest, 1.0f / kClearLeast);
    // three axes, each with the rounding of a position (a bit of `most`) and of its cell (two of
    // `longest`), with room: 5 um for a 3 m scene around the origin, 10 mm at 10 km from it
    g.slack = 0x1p-20f * (most + longest);
    size_t cells = 1;
    for (int k = 0; k < 3; ++k) {
        g.dim[k] = std::min(kClearCells, 1 + std::max(1, (int) std::ceil((hi[k] - lo[k] + 2 * pad) * g.inv)));
        cells *= (size_t) g.dim[k];
    }
    DevBuf marks;
    marks.ensure(2 * cells);
    out.ensure(cells);
    static_assert(0x1010 > kFar, "an unmarked cell starts beyond the cap");
    cuda_check(cudaMemsetAsync(marks.p, 0x10, 2 * cells, s), "clearance memset");
    uint16_t* c = marks.as<uint16_t>();
    k_clear_mark<<<(uint32_t) ((n_tris + 3ull) / 4), 128, 0, s>>>(d_verts, d_tris, n_tris, g, c);
    k_clear_x<<<(g.dim[1] * g.dim[2] + 3) / 4, 128, 0, s>>>(c, g);
    k_clear_line<false><<<dim3((g.dim[0] + 31) / 32, g.dim[2]), 256, 0, s>>>(c, g, nullptr);
    k_clear_line<true><<<dim3((g.dim[0] + 31) / 32, g.dim[1]), 256, 0, s>>>(c, g, out.as<uint8_t>());
    cuda_check(cudaGetLastError(), "clearance grid");
    cuda_check(cudaStreamSynchronize(s), "clearance grid");  // the marks are released on return
    g.gap = out.as<uint8_t>();
    return true;
}

}  // namespace rtcd
