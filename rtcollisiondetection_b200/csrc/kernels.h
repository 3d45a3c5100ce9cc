// kernels.h - device-side views and launchers of the query kernels.
#pragma once
#include "engine.h"

namespace rtcd {

// Robot resident on the device (passed by value to the kernels).
struct RobotDev {
    Chain chain;
    uint32_t n_links;
    uint32_t first_link;            // 1 when the base link is skipped
    float obb[kMaxLinks][16];       // local OBB: centre(3), half(3), axes x/y/z (9), pad
    const float4* tri_nodes;        // link triangle LBVHs (link frames)
    const float4* tri_prims;        // 3 float4 per triangle
    uint32_t tri_root[kMaxLinks];
    const float4* edge_nodes;       // link edge LBVHs (link frames)
    const float4* edge_prims;       // 2 float4 per edge; w of the first = global edge id
    uint32_t edge_root[kMaxLinks];
    uint32_t n_edges_total;
    const float4* tri_wide;         // 4-wide copies of the link trees (8 float4 per node), same leaf references
    uint32_t tri_wide_root[kMaxLinks];   // wide node, or the binary root when that is kNone or a leaf
    const float4* edge_wide;
    uint32_t edge_wide_root[kMaxLinks];
    uint32_t tri_wide_depth, edge_wide_depth;  // deepest wide node of any link
    const float4* cover;            // spheres (link frame) that hold every triangle and edge of a link
    uint32_t cover_off[kMaxLinks + 1];
    uint32_t pair_refs;             // nonzero when every link reference fits beside a candidate's tag
    float4 link_point[kMaxLinks];   // one vertex of each link mesh (link frame)
    const float4* spheres;          // local centre xyz, radius w
    const uint32_t* sphere_link;
    uint32_t n_spheres;
};

// The scene's clearance grid (clearance.cu): cubic cells.
struct ClearGrid {
    float org[3], inv;   // cell of a coordinate: floor((x - org) * inv)
    float slack;         // what the rounding of positions may move a point or a cell's side
    int dim[3];
    const uint8_t* gap;  // [z][y][x] quarter cells, at most the distance to the nearest triangle; NULL: no grid
};
__host__ __device__ inline size_t clear_at(const ClearGrid& g, int x, int y, int z) {
    return ((size_t) z * g.dim[1] + y) * g.dim[0] + x;
}
// The cell of x along axis k, the grid's first or last one outside it.
__device__ __forceinline__ int clear_cell(const ClearGrid& g, int k, float x) {
    return (int) fminf(fmaxf((x - g.org[k]) * g.inv, 0.0f), (float) (g.dim[k] - 1));
}
// Whether every triangle is farther than r from (x, y, z).  The grid's points up to its last cells'
// lower sides hold every triangle; with c the nearest one of them to p, a triangle's squared distance
// from p is at least that from c, which the cell of c bounds, plus |p - c|^2.  Without the second term a
// scene much smaller than the robot culls nothing: its whole grid is nearer than a link's spheres are wide.
// False for what is not a number.
__device__ __forceinline__ bool clear_of(const ClearGrid& g, float x, float y, float z, float r) {
    const float at[3] = {x, y, z};
    int cell[3];
    float d2 = 0.0f;  // in cells
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float t = (at[k] - g.org[k]) * g.inv, c = fminf(fmaxf(t, 0.0f), (float) (g.dim[k] - 1));
        cell[k] = (int) c;
        d2 = fmaf(t - c, t - c, d2);
    }
    const float gap = 0.25f * (float) __ldg(g.gap + clear_at(g, cell[0], cell[1], cell[2]));
    const float reach = (r + g.slack) * g.inv * 1.00001f;
    return fmaf(gap, gap, d2) > reach * reach;
}
bool build_clearance(const float* d_verts, const uint32_t* d_tris, uint32_t n_tris, const float* lo, const float* hi,
                     DevBuf& out, ClearGrid& g, cudaStream_t s);

// Scene resident on the device.
struct SceneDev {
    ClearGrid clear;
    const float4* tri_nodes;
    const float4* tri_prims;
    uint32_t tri_root;
    uint32_t n_tris;
    const float4* edge_nodes;
    const float4* edge_prims;
    uint32_t edge_root;
    uint32_t n_edges;
    const float* obbs;  // 16 floats per obstacle: centre(3), half(3), axes(9), bounding radius
    const float4* obs_box;    // [obstacle][2]: exact box of its vertices (lo, hi)
    const float4* obs_point;  // [obstacle]: one of its vertices
    uint32_t n_obs;           // scene triangles carry their obstacle in the third float4's w
    const float4* tri_wide;   // 4-wide copies of the two trees (8 float4 per node), same leaf references
    uint32_t tri_wide_root;   // 0, or the binary root when that is kNone or a leaf
    const float4* edge_wide;
    uint32_t edge_wide_root;
    const float4* tri_cut;    // top cuts of the wide trees: child records (2 float4 each)
    const float4* edge_cut;
    uint32_t n_tri_cut, n_edge_cut;
    uint32_t edge_wide_lane;  // nonzero when a lane stack of kStack entries holds a wide edge-tree descent
    uint32_t tri_wide_depth, edge_wide_depth;
};

struct DiscreteArgs {
    const float4* T;           // [pose][link][3] link transforms
    const uint32_t* link_count;  // k_prepare's lists: items[slot * n_poses ...] holds link_count[slot] poses of the
                                 // slot's link; NULL: items is one list (n_items, item_word), which
                                 // the query kernel does not read
    uint8_t* flags;            // [pose] set with pose_hit, or NULL
    const uint32_t* items;     // compacted (pose * n_links + link); NULL = all links >= first_link
    uint32_t link_major;       // items hold (link order slot) * n_poses + pose instead (see item_word)
    const uint32_t* n_items;   // device count of items
    uint32_t n_poses;
    uint32_t* pose_hit;        // [pose] nonzero when colliding
    uint32_t* counts;          // [pose] upstream counts (ObsToRobot) or NULL
    uint32_t* edge_bits;       // [pose][edge_words] RobotToObs hit-edge bitset or NULL
    uint32_t edge_words;
    uint32_t* work_counter;    // zeroed before launch
    uint32_t* err;
    unsigned long long* stats; // [0] fp64 re-tests
    int want_counts;
};

constexpr int kFkThreads = 128;
constexpr int kTravThreads = 128;

// Wavefront form of the discrete traversal (stage_b_form 1, 2): stage A (one warp per item)
// emits (item position, scene primitive) candidates, stage B (one lane per
// candidate) runs the link-side descent.  Items whose candidates do not fit
// the buffer are flagged and re-run by the fused kernel.
struct WaveArgs {
    DiscreteArgs d;
    uint2* cand;               // (item word pose * n_links + link, scene primitive)
    uint32_t* cand_count;      // zeroed before stage A; may exceed cand_cap
    uint32_t cand_cap;
    uint8_t* item_overflow;    // [item word] set when its candidates overflowed; zeroed before stage A
    uint32_t* overflow_items;  // compacted overflowed items (item words, for the fused kernel)
    uint32_t* overflow_count;  // zeroed before stage A
    uint32_t chunk;            // stage B: consecutive candidates (lanes) or 32-candidate groups (packets) per worker
    uint32_t light_steps;      // stage B visits before a candidate moves to the heavy pass; 0 = no heavy pass
    uint2* heavy;              // [heavy_cap] candidates (item word, primitive) handed to the heavy pass
    uint32_t heavy_cap;
    uint32_t* heavy_count;     // appended (may exceed heavy_cap: those stayed in the light pass); zeroed
    uint32_t* heavy_work;      // heavy-pass work counter; zeroed
};

// Work sharing between the warps of a launch (share.cuh).
struct TaskQueue {
    unsigned long long* queue;  // tickets taken by idle warps, and tasks offered (share.cuh)
    uint32_t* live;             // warps of the blocks that have started; zeroed
    uint32_t* over;             // set once every live warp waits; zeroed
    uint32_t* err;              // device error word
    ulonglong2* slot;           // [slots] what a ticket's warp gets; all ones at first
    uint32_t slots;             // a power of two, at least twice the launch's warps
    uint32_t most_waiting;      // warps that may wait at once; a further idle one leaves
};
constexpr uint32_t kShareSlots = 32768;

// The query kernel: both stages and their load balancing in one launch.
struct QueryArgs {
    DiscreteArgs d;
    TaskQueue share;
};
constexpr int kQueryWarps = 4;

// items: an upper bound of the item count; share: percent of the resident grid it
// may take; most: largest number of blocks.
void launch_query(bool robot_to_obs, const RobotDev& R, const SceneDev& S, const QueryArgs& Q, uint64_t items,
                  uint32_t share, uint32_t most, cudaStream_t s);

constexpr int kStageAWarps = 4;
constexpr int kFrontier = 32 * (kStack + 2);  // bound of a 32-wide LIFO frontier over a tree of depth <= kStack - 2

void launch_stage_a(bool robot_to_obs, const RobotDev& R, const SceneDev& S, const WaveArgs& W, uint32_t blocks,
                    cudaStream_t s);
// Stage B's light pass (32-candidate packets, or one lane per candidate) on
// `blocks` x `threads`, then (when W.light_steps) its heavy pass on
// heavy_share percent of the full persistent grid.
void launch_stage_b(bool robot_to_obs, const RobotDev& R, const SceneDev& S, const WaveArgs& W, uint32_t blocks,
                    uint32_t threads, uint32_t heavy_share, bool packets, cudaStream_t s);
// The heavy pass alone (after a light pass that spilled into W.heavy).
void launch_stage_b_heavy(bool robot_to_obs, const RobotDev& R, const SceneDev& S, const WaveArgs& W,
                          uint32_t heavy_share, cudaStream_t s);
uint32_t stage_a_blocks(bool robot_to_obs);
uint32_t stage_b_blocks(bool robot_to_obs);
uint32_t stage_b_max_blocks_per_sm(bool robot_to_obs, uint32_t threads);  // threads: 64, 128 or 256

void launch_fk_poses(const Chain& ch, const float* d_q, uint32_t n, float4* d_T, cudaStream_t s);
// The compacted items of launch_cull / launch_all_items as launch_prepare's lists.
void launch_split_lists(const uint32_t* d_items, const uint32_t* d_n_items, uint32_t n, uint32_t n_links,
                        uint32_t* d_lists, uint32_t* d_link_count, cudaStream_t s);
// FK, cull and per-link item lists in one launch: transforms (of the items kept), pose_hit and
// flags zeroed, link_count (zeroed before) and items filled.  all: no cull.
void launch_prepare(const RobotDev& R, const SceneDev& S, const float* d_q, uint32_t n, bool all, float4* d_T,
                    uint32_t* d_hit, uint8_t* d_flags, uint32_t* d_link_count, uint32_t* d_items, cudaStream_t s);
// link_major: the mask (and so the compacted items) in link order, every pose's
// last link before any pose's next-to-last one (item_word decodes it).
void launch_cull(const RobotDev& R, const SceneDev& S, const float4* d_T, uint32_t n, uint8_t* d_mask, bool link_major,
                 unsigned long long* d_stats, cudaStream_t s);
void launch_all_items(const RobotDev& R, uint32_t n, uint32_t* d_items, uint32_t* d_count, cudaStream_t s);
void launch_discrete(bool robot_to_obs, const RobotDev& R, const SceneDev& S, const DiscreteArgs& A, uint32_t blocks,
                     cudaStream_t s);
void launch_popcount_rows(const uint32_t* d_bits, uint32_t words, uint32_t rows, uint32_t* d_out, cudaStream_t s);
// flags[i] = (hit[i] != 0) | 2 * (contain[i] != 0); contain may be NULL.
void launch_flags(const uint32_t* d_hit, uint32_t n, uint8_t* d_flags, cudaStream_t s,
                  const uint32_t* d_contain = nullptr);
// flags[i] = hit[i] != 0 for the n trajectories, seg[i] = hit[n + i] != 0 for the pieces.
void launch_sweep_flags(const uint32_t* d_hit, uint32_t n, uint8_t* d_flags, uint32_t pieces, uint8_t* d_seg,
                        cudaStream_t s);
// Containment of the items' poses not yet hit (sets contain[pose] = 1).
void launch_contain(const RobotDev& R, const SceneDev& S, const DiscreteArgs& A, uint32_t* d_contain, cudaStream_t s);
uint32_t discrete_persistent_blocks(bool robot_to_obs);

// ---- sweeps
// A sweep unit handed to the heavy pass: its geometry (linear: capsule axis
// P0-P1; quadratic: Bezier piece P0 P1 P2, or an end sphere), radius, owner.
struct SweepRec {
    float4 P0, P1, P2;
    float r;
    uint32_t traj, piece_g, pad;
};

struct SweepArgs {
    const float4* centers;     // [waypoint][sphere] world centre xyz, radius w
    const float4* ctrl;        // [control point][sphere] (quadratic) or NULL
    const uint32_t* traj_piece_off;  // [n_traj + 1] prefix of pieces
    const uint32_t* traj_wp_off;     // [n_traj + 1] waypoint offsets
    const uint32_t* traj_ctrl_off;   // [n_traj + 1] control point offsets (quadratic)
    const uint32_t* piece_traj;      // [pieces] owning trajectory of each piece
    uint32_t n_traj;
    uint32_t n_spheres;
    uint32_t total_units;      // pieces * spheres
    int quad;
    int endpoints;
    int surface;               // entering-ray semantics over the loop edges (leaf_hit_surface)
    uint32_t* traj_hit;        // [n_traj]
    uint32_t* piece_hit;       // [pieces] or NULL
    uint32_t* counts;          // [n_traj] or NULL
    uint32_t* work_counter;
    uint32_t* err;
    unsigned long long* stats;
    int want_counts;
    int want_pieces;
    uint32_t light_steps;      // visits before a unit moves to the heavy pass; 0 = no heavy pass
    uint32_t descend_cap;      // light pass: visits a lane makes per descent before the warp's lanes
                               // without work take new units (its descent resumes after); 0 = until a leaf
    int binary_tree;           // light pass on the binary edge tree (else the 4-wide one where the scene allows)
    SweepRec* heavy;           // [heavy_cap] units handed to the heavy pass
    uint32_t heavy_cap;
    uint32_t* heavy_count;     // units appended (may exceed heavy_cap: those stayed in the light pass)
    uint2* rest;               // [rest_cap] (heavy record, wide edge-tree node): what is left of their descents
    uint32_t rest_cap;
    uint32_t* rest_count;      // appended (may exceed rest_cap: those units stayed in the light pass)
    uint32_t* rest_work;       // heavy-pass work counter
    TaskQueue share;
    // the staged light pass (k_sweep_traj): a block takes `group` consecutive trajectories at a time
    // from work_counter, runs their FK (and quadratic fit) into shared memory and their units from there
    const float* q;            // [waypoint][dof] joint values
    const float* W;            // quadratic fit tables, W_off[n] = the table of n waypoints
    const uint32_t* W_off;
    uint32_t max_wp, max_nc, max_pieces;  // largest trajectory of the batch (shared-memory sizing)
    uint32_t group;            // staged: trajectories per claim, 0 = chosen at launch (1..kSweepMaxGroup)
};
constexpr uint32_t kSweepMaxGroup = 8;

void launch_fk_spheres(const RobotDev& R, const float* d_q, uint32_t n_wp, float4* d_centers, cudaStream_t s);
void launch_fit(const float4* d_centers, const uint32_t* d_wp_off, const uint32_t* d_ctrl_off, const float* d_W,
                const uint32_t* d_W_off, uint32_t n_traj, uint32_t n_spheres, float4* d_ctrl, cudaStream_t s);
// The light pass on `blocks` blocks of `threads`, then (when A.light_steps)
// the heavy pass on heavy_share percent of its full persistent grid.
// ev_light (optional) is recorded between the two passes.  The heavy pass
// counts into the second stats bank (A.stats + kStatBank).  staged: the
// light pass stages each trajectory's FK (and fit) in shared memory
// (k_sweep_traj) instead of reading A.centers / A.ctrl.
void launch_sweep(const SceneDev& S, const RobotDev& R, const SweepArgs& A, uint32_t blocks, uint32_t threads,
                  uint32_t heavy_share, bool staged, cudaStream_t s, cudaEvent_t ev_light = nullptr);
// Shared memory of the staged light pass for a batch; 0 when it does not fit (the caller then
// computes the centres and control points in global memory and runs the unstaged light pass).
size_t sweep_staged_smem(bool quad, uint32_t n_links, uint32_t max_wp, uint32_t max_nc, uint32_t max_pieces);
uint32_t sweep_persistent_blocks(bool quad);
uint32_t sweep_max_blocks_per_sm(bool quad, uint32_t threads);  // threads: 64, 128 or 256

// diagnostics of the exact tests (discrete.cu, sweep.cu)
void launch_probe_segtri(const float* d_seg, const float* d_tri, uint32_t n, float* d_cls, double* d_dec,
                         cudaStream_t s);
void launch_probe_sweep(bool quad, const float* d_seg, const float* d_piece, uint32_t n, float* d32, double* d64,
                        cudaStream_t s);

// planner side (planner.cu)
constexpr uint32_t kKnnMaxK = 32;
constexpr uint32_t kKnnMaxDim = 16;
// w2: the squared weights (host).
void launch_knn(const float* pts, uint32_t n, uint32_t dim, const float* w2, uint32_t k, const uint8_t* mask,
                uint32_t* idx, float* dist, cudaStream_t s);
void launch_interp_edges(const float* nodes, uint32_t n_nodes, uint32_t dof, const uint32_t* edges, uint32_t n_edges,
                         uint32_t n_wp, float* q, uint32_t* err, cudaStream_t s);
void launch_or_rows(const uint8_t* pose_flags, uint32_t n_edges, uint32_t n_wp, uint8_t* flags, cudaStream_t s);

}  // namespace rtcd
