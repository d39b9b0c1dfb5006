// bcc_pipeline.cuh -- robot-templated kernels and launchers of the batch edge
// collision checker (sm_100a).
//
// Included by exactly one translation unit per robot (bcc_robot_<name>.cu),
// which defines the robot's __constant__ tables, specialises tab<Model>() to
// return them and instantiates everything below for its model through
// robot_ops_of<Model>().
//
// Pipeline of one check (all on one stream):
//   1. edge_steps_kernel   n per edge (reference discretisation, src/batch_cc.cu:103-107)
//   2. scan_kernel         exclusive prefix sum of 32 n -> per-edge sample offsets
//   3. fk_staged_kernel    FK of every (edge, sample) into the sample table,
//                          env-independent, computed once instead of once per
//                          environment as in the reference
//   4.                     and, while the rows are in shared memory, their
//                          self-collision (src/utils.cuh:1192-5440 for Panda),
//                          OR-reduced per edge, and the segments' spheres
//   5. swept_kernel        per (edge, link) AABB of the link's cull sphere over
//                          all the edge's samples
//   6. probe_kernel        one lane per (environment, edge) pair: decides most pairs
//                          from the environment's probe grid (a voxel grid of
//                          nearest primitives and distances) and queues the rest
//   7. walk_kernel         persistent CTAs pull queued pairs, one environment at a
//                          time, its primitive records staged into shared memory by
//                          a cp.async.bulk copy.  Per pair, lane g turns link g's
//                          swept AABB into three slab ranges and ANDs three 64-bit
//                          primitive masks of the environment's interval-mask tables
//                          (the cull, read through L1), the surviving (primitive,
//                          link) pairs are compacted (lane g writes link g's), and
//                          the warp walks (sample, pair) items 32 at a time in check
//                          order with a warp-ballot exit on the first hit.
// or, for both, check_kernel: CTA = one environment x a tile of edges, every pair
// walked as above (the queued learned order's probe, and launch configurations
// without the first pass).
//
// Gate semantics.  The reference tests a link's leaves only after the link's
// bounding sphere hit SOME primitive (fkcc: `if (bound in collision) { if
// (leaf in collision) return false; ... }`).  Where the leaves lie inside the
// bound a leaf's hit implies its bound's, so any order of tests gives the
// reference's verdict: the walk by segments goes from a segment's sphere to the
// leaves, the walk by samples tests the bound against a primitive and, on a hit,
// every leaf against it.  (Environments where a hit does not imply the bound's:
// kEnvIrregular.)  For the leaves that stick out of their bound (Fetch, Baxter:
// up to 0.6 mm, the model's env_over_count / env_cull_pad) the checker also
// tests them against primitives the bound misses but the padded bound reaches,
// and a hit there counts only after a scan of the whole environment confirms
// that the bound hits some primitive at that sample.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#include <cuda_bf16.h>

#include "bcc_device.cuh"
#include "bcc_kernels.h"
#include "bcc_mlp.h"

namespace bcc {

constexpr unsigned kFull = 0xffffffffu;
constexpr float kSegMargin = 1e-4f;  // FP32 rounding of centres and distances (~1e-6 m), generously

// ------------------------------------------------------------------ tables
// Scalar type of a robot's forward kinematics.
template <class M>
using FkReal = typename std::conditional<M::fk_precision == 64, double, float>::type;

template <class M>
struct DevTables {
    int env_bound[M::num_env_groups];
    int leaf_begin[M::num_env_groups + 1];
    unsigned char leaf_group[M::num_env_leaves], leaf_over[M::num_env_leaves];  // group, overhangs its bound
    int over_count[M::num_env_groups];
    float cull_pad[M::num_env_groups];
    // Certain-hit radius of env group g (0: none): a primitive whose core lies
    // within rho + cert_r[g] of the bound's centre is hit by a leaf of g.
    float cert_r[M::num_env_groups];
    float gate_r[M::num_env_groups];   // the bound's radius, inflated
    float seg_pad[M::num_env_groups];  // radius + inflation + overhang + margin
    // Groups by descending certain-hit radius (the probe's order).
    int probe_group[M::num_env_groups];
    int self_bound[M::num_self_groups][2];
    int self_pair_begin[M::num_self_groups + 1];
    unsigned char self_pairs[M::num_self_pairs][2];
    // Self groups whose leaf pairs are every leaf of side 0 against every leaf
    // of side 1 (self_prod[g] = 1; at most 32 leaves a side, each side's leaves
    // rigid with its bound): the sides' leaves (row positions) and, per side,
    // how far its leaves may reach outside its bound plus a margin for FP32
    // rounding.  A leaf that misses the other side's bound grown by that side's
    // pad misses every leaf of that side.
    unsigned char self_prod[M::num_self_groups];
    int self_la_begin[M::num_self_groups + 1], self_lb_begin[M::num_self_groups + 1];
    unsigned char self_la[M::num_self_pairs], self_lb[M::num_self_pairs];
    float self_pad[M::num_self_groups][2];
    unsigned char self_frame[M::num_self_groups][2];  // frames of a group's bounds
    unsigned char frame_at[M::num_spheres];           // frame by sample-table position
    // Spheres by frame (frame f: entries fk_begin[f] .. fk_begin[f + 1], the first up
    // to fk_x_end[f] with their x product rounded first, see fk_x_first): offset in the
    // frame and radius, row position.
    int fk_begin[M::dof + 2], fk_x_end[M::dof + 1];
    struct alignas(16) FkSphere {  // read as whole 16-byte words
        FkReal<M> x, y, z;
        float r;
        int pos;
    } fk[M::num_spheres];
    float sphere_radius[M::num_spheres];  // by sample-table position
    // The reference's own groups, as row positions (walk_exact).
    unsigned char ref_bound[M::num_ref_env_groups];
    int ref_leaf_begin[M::num_ref_env_groups + 1];
    unsigned char ref_leaf[sizeof(M::ref_env_leaves) / sizeof(int)];
    float s_m[M::dof], s_a[M::dof];       // joint-limit scale q = u * s_m + s_a
};

// Specialised by the robot's translation unit to return its __constant__ tables.
template <class M>
__device__ __forceinline__ const DevTables<M>& tab();
// ... and its copy in global memory, for reads whose index differs by lane:
// constant memory serialises those, one pass per distinct address.
template <class M>
__device__ __forceinline__ const DevTables<M>& lane_tab();

// Margin (m) added to a side's containment excess in the self groups' leaf
// filter: far above the FP32 rounding of FK-computed centres (~1e-6 m).
constexpr double kSelfFilterMargin = 1e-4;

// Certain-hit radius of an environment group.  Leaf l (rigid with the bound's
// frame, centre c_l, radius r_l) hits a primitive when the distance from c_l
// to the primitive's core is below r_l + kEnvInflate + rho, and that distance
// is at most the bound centre's distance d_b plus |c_l - c_b| (distance to a
// convex set is 1-Lipschitz).  So d_b < rho + max_l (r_l + kEnvInflate -
// |c_l - c_b|) proves a leaf hit: the leaf penetrates by more than the margin
// subtracted here, far above FP32 rounding of FK-computed centres, so the
// reference's own leaf test (src/utils.cuh:806-1190) finds that hit too.
constexpr double kCertMargin = 1e-4;

template <class M>
float cert_radius(int g) {
    const int b = M::env_bound[g];
    double best = 0.0;
    for (int k = M::env_leaf_begin[g]; k < M::env_leaf_begin[g + 1]; ++k) {
        const int l = M::env_leaves[k];
        if (M::sphere_frame[l] != M::sphere_frame[b]) continue;  // not rigid with the bound
        // r_l <= r_b keeps the radius within r_b + kEnvInflate, so a certain hit
        // is also a bound hit (the reference tests leaves only after one)
        if (M::sphere_radius[l] > M::sphere_radius[b]) continue;
        double d2 = 0.0;
        for (int c = 0; c < 3; ++c) {
            const double d = M::sphere_local[l][c] - M::sphere_local[b][c];
            d2 += d * d;
        }
        const double v = (double)M::sphere_radius[l] + (double)kEnvInflate - std::sqrt(d2) - kCertMargin;
        best = v > best ? v : best;
    }
    // rounded down to float: the test stays conservative
    float f = (float)best;
    if ((double)f > best) f = std::nextafter(f, 0.0f);
    return f;
}

// A sphere's centre is R0 x + R1 y + R2 z + p in fused multiply-adds, and which
// product is rounded by itself decides its last bit: R1 y, or R0 x for the row
// positions a robot's specialisation names.  Verdicts at contact follow those
// bits, so a robot's spheres keep the order they have always been computed in.
template <class M>
constexpr bool fk_x_first(int pos) {
    return false;
}

template <class M>
void self_products(DevTables<M>& t) {
    int na_tot = 0, nb_tot = 0;
    for (int g = 0; g < M::num_self_groups; ++g) {
        const int k0 = M::self_pair_begin[g], k1 = M::self_pair_begin[g + 1];
        int la[M::num_spheres], lb[M::num_spheres], na = 0, nb = 0;
        bool in_a[M::num_spheres] = {}, in_b[M::num_spheres] = {};
        for (int k = k0; k < k1; ++k) {
            const int a = M::self_pairs[k][0], b = M::self_pairs[k][1];
            if (!in_a[a]) { in_a[a] = true; la[na++] = a; }
            if (!in_b[b]) { in_b[b] = true; lb[nb++] = b; }
        }
        // a product: as many distinct pairs as |A| x |B| (each pair is in A x B)
        bool prod = na <= 32 && nb <= 32 && na * nb == k1 - k0;
        for (int k = k0; k < k1 && prod; ++k)
            for (int k2 = k0; k2 < k; ++k2)
                if (M::self_pairs[k2][0] == M::self_pairs[k][0] && M::self_pairs[k2][1] == M::self_pairs[k][1])
                    prod = false;
        for (int side = 0; side < 2 && prod; ++side) {
            const int b = M::self_bound[g][side];
            double excess = 0.0;
            for (int i = 0; i < (side ? nb : na); ++i) {
                const int l = side ? lb[i] : la[i];
                if (M::sphere_frame[l] != M::sphere_frame[b]) { prod = false; break; }
                double d2 = 0.0;
                for (int c = 0; c < 3; ++c) {
                    const double d = M::sphere_local[l][c] - M::sphere_local[b][c];
                    d2 += d * d;
                }
                const double ex = std::sqrt(d2) + M::sphere_radius[l] - M::sphere_radius[b];
                excess = ex > excess ? ex : excess;
            }
            t.self_pad[g][side] = (float)(excess + kSelfFilterMargin);
        }
        t.self_prod[g] = prod ? 1 : 0;
        for (int side = 0; side < 2; ++side)
            t.self_frame[g][side] = (unsigned char)M::sphere_frame[M::self_bound[g][side]];
        t.self_la_begin[g] = na_tot;
        t.self_lb_begin[g] = nb_tot;
        if (prod) {
            for (int i = 0; i < na; ++i) t.self_la[na_tot++] = (unsigned char)M::table_pos[la[i]];
            for (int i = 0; i < nb; ++i) t.self_lb[nb_tot++] = (unsigned char)M::table_pos[lb[i]];
        } else {
            t.self_pad[g][0] = t.self_pad[g][1] = 0.0f;
        }
    }
    t.self_la_begin[M::num_self_groups] = na_tot;
    t.self_lb_begin[M::num_self_groups] = nb_tot;
}

template <class M>
DevTables<M> host_tables() {
    static_assert(M::num_env_groups <= kMaxEnvGroups, "one cull lane per link group");
    static_assert(M::num_spheres <= kMaxTableSpheres, "sample-table row width");
    static_assert(M::num_spheres <= 256, "self pairs hold 8-bit row positions");
    DevTables<M> t;
    for (int g = 0; g < M::num_env_groups; ++g) {
        t.env_bound[g] = M::env_bound[g];
        t.over_count[g] = M::env_over_count[g];
        t.cull_pad[g] = M::env_cull_pad[g];
        t.cert_r[g] = cert_radius<M>(g);
    }
    for (int g = 0; g < M::num_env_groups; ++g) t.probe_group[g] = g;
    std::stable_sort(t.probe_group, t.probe_group + M::num_env_groups,
                     [&](int a, int b) { return t.cert_r[a] > t.cert_r[b]; });
    for (int g = 0; g <= M::num_env_groups; ++g) t.leaf_begin[g] = M::env_leaf_begin[g];
    for (int g = 0; g < M::num_env_groups; ++g)
        for (int l = t.leaf_begin[g]; l < t.leaf_begin[g + 1]; ++l) {
            t.leaf_group[l] = (unsigned char)g;
            t.leaf_over[l] = l < t.leaf_begin[g] + M::env_over_count[g];
        }
    // Self tables hold sample-table row positions, not sphere indices.
    for (int g = 0; g < M::num_self_groups; ++g) {
        t.self_bound[g][0] = M::table_pos[M::self_bound[g][0]];
        t.self_bound[g][1] = M::table_pos[M::self_bound[g][1]];
    }
    for (int g = 0; g <= M::num_self_groups; ++g) t.self_pair_begin[g] = M::self_pair_begin[g];
    for (int i = 0; i < M::num_self_pairs; ++i) {
        t.self_pairs[i][0] = (unsigned char)M::table_pos[M::self_pairs[i][0]];
        t.self_pairs[i][1] = (unsigned char)M::table_pos[M::self_pairs[i][1]];
    }
    self_products<M>(t);
    for (int s = 0; s < M::num_spheres; ++s) {
        t.sphere_radius[M::table_pos[s]] = M::sphere_radius[s];
        t.frame_at[M::table_pos[s]] = (unsigned char)M::sphere_frame[s];
    }
    int at = 0;
    for (int f = 0; f <= M::dof; ++f) {
        t.fk_begin[f] = at;
        for (int y_first = 0; y_first < 2; ++y_first) {
            for (int s = 0; s < M::num_spheres; ++s)
                if (M::sphere_frame[s] == f && fk_x_first<M>(M::table_pos[s]) == !y_first) {
                    t.fk[at++] = {(FkReal<M>)M::sphere_local[s][0], (FkReal<M>)M::sphere_local[s][1],
                                  (FkReal<M>)M::sphere_local[s][2], M::sphere_radius[s], M::table_pos[s]};
                }
            if (!y_first) t.fk_x_end[f] = at;
        }
    }
    t.fk_begin[M::dof + 1] = at;
    for (int g = 0; g < M::num_ref_env_groups; ++g)
        t.ref_bound[g] = (unsigned char)M::table_pos[M::ref_env_bound[g]];
    for (int g = 0; g <= M::num_ref_env_groups; ++g) t.ref_leaf_begin[g] = M::ref_env_leaf_begin[g];
    for (int l = 0; l < t.ref_leaf_begin[M::num_ref_env_groups]; ++l)
        t.ref_leaf[l] = (unsigned char)M::table_pos[M::ref_env_leaves[l]];
    for (int g = 0; g < M::num_env_groups; ++g) t.gate_r[g] = t.sphere_radius[g] + kEnvInflate;
    for (int g = 0; g < M::num_env_groups; ++g)
        t.seg_pad[g] = t.sphere_radius[g] + kEnvInflate + t.cull_pad[g] + kSegMargin;
    for (int j = 0; j < M::dof; ++j) {
        t.s_m[j] = M::s_m[j];
        t.s_a[j] = M::s_a[j];
    }
    return t;
}

// The robot's tables into both of its symbols, complete on return: the copies, from
// pageable memory, may return with their last DMA in flight on the legacy stream,
// which a non-blocking stream's kernels are not ordered after.
template <class M>
cudaError_t upload_to(const DevTables<M>& global, const DevTables<M>& constant) {
    const DevTables<M> t = host_tables<M>();
    cudaError_t err = cudaMemcpyToSymbol(global, &t, sizeof(t));
    if (err == cudaSuccess) err = cudaMemcpyToSymbol(constant, &t, sizeof(t));
    return err == cudaSuccess ? cudaStreamSynchronize(cudaStreamLegacy) : err;
}

// Bits of the link-group index in a packed (primitive, group) pair.
template <class M>
constexpr int group_bits() {
    return M::num_env_groups <= 16 ? 4 : 5;
}

// Largest primitive count per environment the 16-bit pair packing allows.
template <class M>
constexpr int max_prims_of() {
    return (1 << (16 - group_bits<M>())) - 1;
}

template <class M>
constexpr bool has_overhang() {
    for (int g = 0; g < M::num_env_groups; ++g)
        if (M::env_over_count[g] > 0) return true;
    return false;
}

// ------------------------------------------------------------------ 1. steps
// Step count of edge e.  Non-finite endpoints would give an unbounded one: clamped,
// and the host rejects the resulting sample total (BCC_ERR_LIMIT).
template <class M>
__device__ __forceinline__ int clamped_steps(const float* __restrict__ edges, int e, int resolution) {
    float s[M::dof], t[M::dof];
#pragma unroll
    for (int j = 0; j < M::dof; ++j) {
        s[j] = edges[(size_t)e * 2 * M::dof + j];
        t[j] = edges[(size_t)e * 2 * M::dof + M::dof + j];
    }
    const int n = edge_steps<M::dof>(s, t, resolution);
    return (n < 1 || n > (1 << 20)) ? (1 << 20) : n;
}

template <class M>
__global__ void edge_steps_kernel(const float* __restrict__ edges, int E, int resolution,
                                  int* __restrict__ steps) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < E) steps[e] = clamped_steps<M>(edges, e, resolution);
}

// Steps and sample offsets of at most 1024 edges in one launch of one CTA (see
// scan_kernel): small calls are a chain of launches.
constexpr int kFusedSteps = 1024;

template <class M>
__global__ void __launch_bounds__(kFusedSteps) edge_offsets_kernel(const float* __restrict__ edges, int E,
                                                                   int resolution, int* __restrict__ steps,
                                                                   int* __restrict__ offs,
                                                                   int* __restrict__ host_total) {
    __shared__ long long sums[32];
    const int e = threadIdx.x;
    long long v = 0;
    if (e < E) {
        const int n = clamped_steps<M>(edges, e, resolution);
        steps[e] = n;
        v = (long long)kLanes * n;
    }
    long long total;
    const long long at = block_scan_exclusive(v, sums, total);
    if (e < E) offs[e] = (int)min(at, 2147483647ll);
    if (e == 0) {
        offs[E] = (int)min(total, 2147483647ll);
        if (host_total) *host_total = (int)min(total, 2147483647ll);
    }
}

// ------------------------------------------------------------------ 3. FK
// Sample table row: num_spheres float4 (centre xyz, radius) in table_pos order
// (env-group bounds, then env leaves, then the rest), one row per (edge,
// sample) in edge order then sample index order.
__device__ __forceinline__ bool self_hit(float4 a, float4 b) {
    const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    const float rs = a.w + b.w;
    return fmaf(dx, dx, fmaf(dy, dy, dz * dz)) - rs * rs < 0.0f;
}

__device__ __forceinline__ bool self_hit_pad(float4 a, float4 b, float pad) {
    const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    const float rs = a.w + b.w + pad;
    return fmaf(dx, dx, fmaf(dy, dy, dz * dz)) - rs * rs < 0.0f;
}

__device__ __forceinline__ float dist2(float4 a, float4 b) {
    const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

// A segment's (kSegment consecutive samples of an edge) spheres are centred at
// its middle sample, row kSegMid.  Group g's entry (R, rho) of segment s: the
// sphere of radius R around the bound's centre there holds all that group g can
// hit with at any of the samples (bound, overhang, inflation, margin); a leaf's
// centre stays within rho of where it is at the middle sample (robots whose groups
// are rigid, see groups_are_rigid).
template <class M>
constexpr bool groups_are_rigid() {
    for (int g = 0; g < M::num_env_groups; ++g)
        for (int k = M::env_leaf_begin[g]; k < M::env_leaf_begin[g + 1]; ++k)
            if (M::sphere_frame[M::env_leaves[k]] != M::sphere_frame[M::env_bound[g]]) return false;
    return true;
}
constexpr int kSegMid = kSegment / 2;

// Shared state of a staged block of 32 rows: how far any sphere of a frame moves
// from its place at its segment's middle row, and how far each group's bound does
// (squared, as bits: they order like the values), and the (self group, segment)
// items still in question.
constexpr int kBlockSegs = 32 / kSegment;
template <class M>
struct BlockState {
    int move2[M::dof + 1][kBlockSegs];
    float bound2[M::num_env_groups][kBlockSegs];
    int num_items;
    unsigned short items[M::num_self_groups * kBlockSegs];
};

// The block's movements: every lane measures its row (row l at srow + l * STRIDE)
// against its segment's middle one, eight lanes reduce.  The warps share out every
// frame's spheres and the groups' bounds.
template <class M, int STRIDE>
__device__ __forceinline__ void block_movements(const float4* srow, int warp, int warps, BlockState<M>& B) {
    const DevTables<M>& T = tab<M>();
    const int lane = threadIdx.x & 31, sg = lane / kSegment;
    const float4* mine = srow + lane * STRIDE;
    const float4* mid = srow + ((lane & ~(kSegment - 1)) + kSegMid) * STRIDE;
    auto reduce = [&](float v) {
#pragma unroll
        for (int o = 1; o < kSegment; o <<= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
        return v;
    };
    const bool lead = (lane & (kSegment - 1)) == 0;
    if constexpr (groups_are_rigid<M>()) {  // a group's spheres are one frame's and contiguous in the row
        constexpr int G = M::num_env_groups;
        for (int g = warp; g < G; g += warps) {
            const float b = reduce(dist2(mine[g], mid[g]));
            float l = 0.0f;
            const int end = T.leaf_begin[g + 1];
#pragma unroll 4
            for (int i = T.leaf_begin[g]; i < end; ++i) l = fmaxf(l, dist2(mine[G + i], mid[G + i]));
            l = reduce(l);
            if (lead) {
                B.bound2[g][sg] = b;
                atomicMax(&B.move2[T.frame_at[g]][sg], __float_as_int(fmaxf(b, l)));
            }
        }
        for (int p = G + M::num_env_leaves + warp; p < M::num_spheres; p += warps) {
            const float d = reduce(dist2(mine[p], mid[p]));
            if (lead) atomicMax(&B.move2[T.frame_at[p]][sg], __float_as_int(d));
        }
    } else {
        for (int f = 0; f <= M::dof; ++f) {
            const int begin = T.fk_begin[f] + warp, end = T.fk_begin[f + 1];
            if (begin >= end) continue;
            float d = 0.0f;
#pragma unroll 4
            for (int i = begin; i < end; i += warps) d = fmaxf(d, dist2(mine[T.fk[i].pos], mid[T.fk[i].pos]));
            d = reduce(d);
            if (lead) atomicMax(&B.move2[f][sg], __float_as_int(d));
        }
        for (int g = warp; g < M::num_env_groups; g += warps) {
            const float b = reduce(dist2(mine[g], mid[g]));
            if (lead) B.bound2[g][sg] = b;
        }
    }
}

// Does (self group, segment) item `item` hold a hit: a sample whose bound pair
// overlaps and one of whose leaf pairs does (the reference's gate-then-leaves,
// src/utils.cuh:1192-5440)?  Whole warp.  A product group first drops, at the
// middle sample, the leaves of either side that stay clear of the other side's
// bound over the whole segment (that bound grown by its containment pad and by
// what both frames move), then the pairs that stay clear of each other; the
// surviving pairs are tested at the segment's eight samples.  Other groups drop
// pairs only.
template <class M, int STRIDE>
__device__ __forceinline__ bool self_item_hit(const float4* srow, int item, const BlockState<M>& B, uint8_t (*list)[32],
                                              uint8_t (*pair)[2]) {
    const DevTables<M>& T = tab<M>();
    const DevTables<M>& L = lane_tab<M>();
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int g = item / kBlockSegs, sg = item - g * kBlockSegs;
    const float4* rows = srow + sg * kSegment * STRIDE;
    const float4* mid = rows + kSegMid * STRIDE;
    const int b0 = T.self_bound[g][0], b1 = T.self_bound[g][1];
    // leaf pair (x, y) at sample k of the segment, counted where the bounds overlap
    auto hit_at = [&](int k, int x, int y) {
        const float4* r = rows + k * STRIDE;
        return self_hit(r[x], r[y]) && self_hit(r[b0], r[b1]);
    };
    auto move_of = [&](int frame) { return sqrtf(__int_as_float(B.move2[frame][sg])) * 1.00001f; };
    // 32 leaf pairs (x, y), `near` marking those within reach of each other over the
    // segment: all of its samples.
    auto expand = [&](bool near, int x, int y) {
        const unsigned nm = __ballot_sync(kFull, near);
        if (near) {
            uint8_t* d = pair[__popc(nm & lt)];
            d[0] = (uint8_t)x;
            d[1] = (uint8_t)y;
        }
        __syncwarp();
        const int n = __popc(nm) * kSegment;
        bool hit = false;
        for (int q = lane; q - lane < n && !hit; q += 32) {
            const uint8_t* d = pair[min(q, n - 1) / kSegment];
            hit = __any_sync(kFull, q < n && hit_at(q & (kSegment - 1), d[0], d[1]));
        }
        __syncwarp();
        return hit;
    };
    if (!T.self_prod[g]) {
        const int k0 = T.self_pair_begin[g], m = T.self_pair_begin[g + 1] - k0;
        for (int t0 = 0; t0 < m; t0 += 32) {
            const int k = k0 + min(t0 + lane, m - 1);
            const int x = L.self_pairs[k][0], y = L.self_pairs[k][1];
            const float move = move_of(L.frame_at[x]) + move_of(L.frame_at[y]);
            if (expand(t0 + lane < m && self_hit_pad(mid[x], mid[y], move + kSegMargin), x, y)) return true;
        }
        return false;
    }
    const float move = move_of(T.self_frame[g][0]) + move_of(T.self_frame[g][1]);
    const int a0 = T.self_la_begin[g], na = T.self_la_begin[g + 1] - a0;
    const int c0 = T.self_lb_begin[g], nb = T.self_lb_begin[g + 1] - c0;
    const float4 ba = mid[b0], bb = mid[b1];
    const int la = lane < na ? L.self_la[a0 + lane] : 0, lb = lane < nb ? L.self_lb[c0 + lane] : 0;
    const bool ka = lane < na && self_hit_pad(mid[la], bb, T.self_pad[g][1] + move);
    const bool kb = lane < nb && self_hit_pad(mid[lb], ba, T.self_pad[g][0] + move);
    const unsigned ma = __ballot_sync(kFull, ka), mb = __ballot_sync(kFull, kb);
    if (!ma || !mb) return false;
    if (ka) list[0][__popc(ma & lt)] = (uint8_t)la;
    if (kb) list[1][__popc(mb & lt)] = (uint8_t)lb;
    __syncwarp();
    const int cb = __popc(mb), m = __popc(ma) * cb;
    const float inv = __frcp_rn((float)cb);
    for (int t0 = 0; t0 < m; t0 += 32) {
        const int t = min(t0 + lane, m - 1);
        const int i = (int)(((float)t + 0.5f) * inv);  // t / cb, exact: t < 1024, cb <= 32
        const int x = list[0][i], y = list[1][t - i * cb];
        if (expand(t0 + lane < m && self_hit_pad(mid[x], mid[y], move + kSegMargin), x, y)) return true;
    }
    return false;
}

// Edge of table row `row` (the last e with offs[e] <= row), whole warp: each
// round probes 32 offsets at once, three dependent loads for 10 000 edges where a
// binary search makes fourteen.
__device__ __forceinline__ int edge_of_row(const int* __restrict__ offs, int E, int row) {
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = E;
    while (hi - lo > 1) {
        const int step = (hi - lo + 31) >> 5, i = lo + lane * step;
        const unsigned m = __ballot_sync(kFull, i < hi && offs[i] <= row);  // lane 0 holds
        lo += (__popc(m) - 1) * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

// FK: a CTA of four (or eight) warps computes 32 consecutive rows
// (one edge's: every edge has 32 n rows and starts on a multiple of 32) into
// shared memory, lane l row l.  The warps share out the joints' sines and cosines,
// then each evaluates the frames and its share of every frame's spheres; the rows
// leave as one bulk copy (a row length that is odd makes the shared layout the
// table's; else a copy a row).  While it runs the warps share out the segments'
// spheres and the self-collision check: one thread per (self group, segment) tests the
// bounds at the segment's middle sample, grown by what their frames move within
// it, and the warps take the items that leaves (self_item_hit).  The CTA strides
// over 32-row blocks.  Shared memory (39 KB for Panda) holds five CTAs an SM, and
// a block's instruction chain bounds it.  One warp a block, straight-line code for
// every sphere and one lane per row walking the self groups took 0.252 ms for the
// uneven workload's 11 300 blocks (0.315 with the segments' spheres); four warps
// alone gave 0.352 (the code, several times the instruction cache, was read once
// per warp), sphere and joint tables read in loops and the self check by segments
// 0.194 ms: 9 650 instructions a block, half of the issue slots.
// Robots with wide rows fit three CTAs an SM: eight warps each (Fetch 0.225 ms at
// four, 0.182 at eight; Baxter 0.297, 0.270), against Panda's four (0.194; eight
// 0.217).  One coordinate of half of the frames per warp, a sixth of the FP64
// multiply-adds, was slower (Fetch 0.239, Baxter 0.398): its scalar stores conflict.
template <class M>
constexpr int fk_warps() {
    return M::fk_precision == 64 ? 8 : 4;
}
// CTAs an SM the rows leave room for: the register budget the kernel is compiled to.
template <class M>
constexpr int fk_ctas() {
    return 200 * 1024 / (32 * (M::num_spheres | 1) * 16);
}

// Frame FR's spheres, every fk_warps-th from `warp`, into the row at out (fk_x_first).
template <class M, int FR>
__device__ __forceinline__ void emit_listed(const Frames<M, FkReal<M>>& F, int warp, float4* out) {
    const DevTables<M>& T = tab<M>();
    const FkReal<M>* R = F.R[FR];
    const FkReal<M>* p = F.p[FR];
    const int begin = T.fk_begin[FR], mid = T.fk_x_end[FR], end = T.fk_begin[FR + 1];
    if constexpr (M::fk_precision == 32) {
#pragma unroll 2
        for (int i = begin + warp; i < mid; i += fk_warps<M>()) {
            const auto l = T.fk[i];
            float4 c;
            c.x = __fadd_rn(__fmaf_rn(R[2], l.z, __fmaf_rn(R[1], l.y, __fmul_rn(R[0], l.x))), p[0]);
            c.y = __fadd_rn(__fmaf_rn(R[5], l.z, __fmaf_rn(R[4], l.y, __fmul_rn(R[3], l.x))), p[1]);
            c.z = __fadd_rn(__fmaf_rn(R[8], l.z, __fmaf_rn(R[7], l.y, __fmul_rn(R[6], l.x))), p[2]);
            c.w = l.r;
            out[l.pos] = c;
        }
#pragma unroll 2
        for (int i = mid + warp; i < end; i += fk_warps<M>()) {
            const auto l = T.fk[i];
            float4 c;
            c.x = __fadd_rn(__fmaf_rn(R[2], l.z, __fmaf_rn(R[0], l.x, __fmul_rn(R[1], l.y))), p[0]);
            c.y = __fadd_rn(__fmaf_rn(R[5], l.z, __fmaf_rn(R[3], l.x, __fmul_rn(R[4], l.y))), p[1]);
            c.z = __fadd_rn(__fmaf_rn(R[8], l.z, __fmaf_rn(R[6], l.x, __fmul_rn(R[7], l.y))), p[2]);
            c.w = l.r;
            out[l.pos] = c;
        }
    } else {  // FP64: the order is far below the rounding to float
#pragma unroll 2
        for (int i = begin + warp; i < end; i += fk_warps<M>()) {
            const auto l = T.fk[i];
            float4 c;
            c.x = (float)(R[0] * l.x + R[1] * l.y + R[2] * l.z + p[0]);
            c.y = (float)(R[3] * l.x + R[4] * l.y + R[5] * l.z + p[1]);
            c.z = (float)(R[6] * l.x + R[7] * l.y + R[8] * l.z + p[2]);
            c.w = l.r;
            out[l.pos] = c;
        }
    }
}

// Joints K, K + 1, ... of one row from their values (q[k * 32]) and sines and
// cosines, the warp's share of every frame's spheres.
template <class M, int K>
__device__ __forceinline__ void fk_rows(const float* q, const FkReal<M>* sn, const FkReal<M>* cs,
                                        Frames<M, FkReal<M>>& F, int warp, float4* out) {
    if constexpr (K == 0) {
        fk_base<M, FkReal<M>>(F);
        emit_listed<M, 0>(F, warp, out);
    }
    if constexpr (K < M::dof) {
        fk_advance<M, K, FkReal<M>>((FkReal<M>)q[K * 32], sn[K * 32], cs[K * 32], F);
        emit_listed<M, K + 1>(F, warp, out);
        fk_rows<M, K + 1>(q, sn, cs, F, warp, out);
    }
}

template <class M>
__global__ void __launch_bounds__(32 * fk_warps<M>(), fk_ctas<M>()) fk_staged_kernel(const float* __restrict__ edges, int E,
                                                                  const int* __restrict__ steps,
                                                                  const int* __restrict__ offs, int cap,
                                                                  float4* __restrict__ table,
                                                                  int* __restrict__ edge_self,
                                                                  float2* __restrict__ seg) {
    constexpr int NS = M::num_spheres, STRIDE = NS | 1;  // conflict-free
    constexpr int G = M::num_env_groups;
    extern __shared__ __align__(128) float4 srow[];  // [32][STRIDE]
    __shared__ BlockState<M> B;
    __shared__ uint8_t s_list[fk_warps<M>()][2][32], s_pair[fk_warps<M>()][32][2];
    __shared__ float s_q[M::dof][32];
    __shared__ FkReal<M> s_sin[M::dof][32], s_cos[M::dof][32];
    const DevTables<M>& L = lane_tab<M>();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int total = offs[E];
    if (total > cap) return;
    for (int base = blockIdx.x * 32; base < total; base += gridDim.x * 32) {
        const int e = edge_of_row(offs, E, base);
        const int n = steps[e], k = base + lane - offs[e];
        const float* ends = edges + (size_t)e * 2 * M::dof;
#pragma unroll 1
        for (int j = warp; j < M::dof; j += fk_warps<M>()) {
            const float v = edge_sample_joint(ends[j], ends[M::dof + j], n, k);
            s_q[j][lane] = v;
            sin_cos((FkReal<M>)v, &s_sin[j][lane], &s_cos[j][lane]);
        }
        __syncthreads();
        {
            Frames<M, FkReal<M>> F;
            fk_rows<M, 0>(&s_q[0][lane], &s_sin[0][lane], &s_cos[0][lane], F, warp, srow + lane * STRIDE);
        }
        if (threadIdx.x < (M::dof + 1) * kBlockSegs) (&B.move2[0][0])[threadIdx.x] = 0;
        if (threadIdx.x == 0) B.num_items = 0;
        fence_async_shared();
        __syncthreads();
        const bool copies = STRIDE == NS ? threadIdx.x == 0 : threadIdx.x < 32;
        if (STRIDE == NS) {
            if (copies) bulk_copy_s2g(table + (size_t)base * NS, srow, 32 * NS * sizeof(float4));
        } else if (copies) {
            bulk_copy_s2g(table + (size_t)(base + lane) * NS, srow + lane * STRIDE, NS * sizeof(float4));
        }
        block_movements<M, STRIDE>(srow, warp, fk_warps<M>(), B);
        __syncthreads();
        if (seg)
            for (int i = threadIdx.x; i < G * kBlockSegs; i += 32 * fk_warps<M>()) {
                const int sg = i / G, g = i - sg * G;  // consecutive threads write consecutive entries
                const float r = sqrtf(B.bound2[g][sg]) * 1.00001f + L.seg_pad[g];
                const float move = sqrtf(__int_as_float(B.move2[L.frame_at[g]][sg])) * 1.00001f + kSegMargin;
                seg[(size_t)base / kSegment * G + i] = make_float2(r, move);
            }
        // any hit marks the edge; skipped when another block or warp already has
        if (*(volatile const int*)(edge_self + e) == 0) {
            for (int i = threadIdx.x; i < M::num_self_groups * kBlockSegs; i += 32 * fk_warps<M>()) {
                const int g = i / kBlockSegs, sg = i - g * kBlockSegs;
                const float4* mid = srow + (sg * kSegment + kSegMid) * STRIDE;
                const float move = sqrtf(__int_as_float(B.move2[L.self_frame[g][0]][sg])) +
                                   sqrtf(__int_as_float(B.move2[L.self_frame[g][1]][sg]));
                if (self_hit_pad(mid[L.self_bound[g][0]], mid[L.self_bound[g][1]], move * 1.00001f + kSegMargin))
                    B.items[atomicAdd(&B.num_items, 1)] = (unsigned short)i;
            }
        }
        __syncthreads();
        for (int i = warp; i < B.num_items; i += fk_warps<M>())
            if (self_item_hit<M, STRIDE>(srow, B.items[i], B, s_list[warp], s_pair[warp])) {
                if (lane == 0) atomicOr(edge_self + e, 1);
                break;
            }
        if (copies) bulk_wait_read();
        __syncthreads();  // the next block overwrites srow
    }
    if (threadIdx.x < 32) bulk_wait();
}

// ------------------------------------------------------------------ 5. swept
// Slab of x on one axis: the largest s in [0, kGridSlabs) with b[s] <= x (0
// below b[0]); b holds the axis' kGridSlabs + 1 increasing boundaries.
__device__ __forceinline__ int slab_of(const float* __restrict__ b, float x) {
    int s = 0;
#pragma unroll
    for (int step = kGridSlabs / 2; step; step >>= 1)
        if (b[s + step] <= x) s += step;
    return s;
}

// Slab index range of [lo, hi] on one axis of the environment set's cull grid,
// as a triangular table index; -1 when the interval misses every primitive.
__device__ __forceinline__ int slab_tri(float lo, float hi, const float* __restrict__ b) {
    if (!(hi >= b[0]) || !(lo < b[kGridSlabs])) return -1;
    return tri_index(slab_of(b, lo), slab_of(b, hi));
}

// One warp per edge: AABB (lo, hi) of every link group's bounding sphere over
// the edge's samples, inflated by radius + 0.005 + the group's leaf overhang +
// cull margin, written where swept is given (the records check); and (edge_tri
// non-null) its slab ranges on the set's cull grid, packed tx | ty << 10 | tz << 20
// (-1 when some axis misses every primitive); and (mid non-null) the bound's centre
// at the edge's middle sample with the radius, inflated likewise, of the sphere
// around it that holds them all.
// Lane g ends up holding group g's box: it scans group g's bound down the rows (a
// row's bounds are contiguous), 32 / G rows at a time.
template <class M>
__global__ void swept_kernel(const float4* __restrict__ table, const int* __restrict__ offs, int E, int cap,
                             float4* __restrict__ swept, int* __restrict__ edge_tri,
                             const float* __restrict__ bounds, float4* __restrict__ mid) {
    constexpr int G = M::num_env_groups;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= E || offs[E] > cap) return;
    const int r0 = offs[warp], r1 = offs[warp + 1];
    const DevTables<M>& T = tab<M>();
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    float far2 = 0.0f;  // largest squared distance of the bound's centre from its middle one
    const int rm = r0 + ((r1 - r0) >> 1);
    // 32 / G row streams: lane s G + g scans group g's bound on rows
    // r0 + s, r0 + s + 32 / G, ... (bounds lead every table row); lane g then
    // folds in the other streams' boxes.
    constexpr int RS = kLanes / G;
    const int rs = lane / G, gl = lane - rs * G;
    if (rs < RS) {
        const float4 m = table[table_index<M>(rm, gl)];
        for (int r = r0 + rs; r < r1; r += RS) {
            const float4 c = table[table_index<M>(r, gl)];
            far2 = fmaxf(far2, dist2(c, m));
            lo[0] = fminf(lo[0], c.x); lo[1] = fminf(lo[1], c.y); lo[2] = fminf(lo[2], c.z);
            hi[0] = fmaxf(hi[0], c.x); hi[1] = fmaxf(hi[1], c.y); hi[2] = fmaxf(hi[2], c.z);
        }
    }
#pragma unroll
    for (int t = 1; t < RS; ++t) {
        const int src = min(lane + t * G, kLanes - 1);  // lanes >= G read a valid lane and discard it
        far2 = fmaxf(far2, __shfl_sync(kFull, far2, src));
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = fminf(lo[a], __shfl_sync(kFull, lo[a], src));
            hi[a] = fmaxf(hi[a], __shfl_sync(kFull, hi[a], src));
        }
    }
    if (lane >= G) return;
    const int g = lane;
    const float pad = T.sphere_radius[g] + kEnvInflate + T.cull_pad[g] + kCullMargin;
    if (mid) {  // group-major: the probe's lanes read consecutive edges
        float4 c = table[table_index<M>(rm, g)];
        c.w = sqrtf(far2) * 1.00001f + pad;
        mid[(size_t)g * E + warp] = c;
    }
    const float4 l = make_float4(lo[0] - pad, lo[1] - pad, lo[2] - pad, 0.0f);
    const float4 h = make_float4(hi[0] + pad, hi[1] + pad, hi[2] + pad, 0.0f);
    if (swept) {
        swept[((size_t)warp * G + g) * 2 + 0] = l;
        swept[((size_t)warp * G + g) * 2 + 1] = h;
    }
    if (edge_tri) {
        const int tx = slab_tri(l.x, h.x, bounds);
        const int ty = slab_tri(l.y, h.y, bounds + (kGridSlabs + 1));
        const int tz = slab_tri(l.z, h.z, bounds + 2 * (kGridSlabs + 1));
        edge_tri[(size_t)warp * G + g] = (tx < 0 || ty < 0 || tz < 0) ? -1 : (tx | (ty << 10) | (tz << 20));
    }
}

// ------------------------------------------------------------------ 6. check
// Whole warp: does link group g's bounding sphere at sample k hit any of the
// environment's np primitives (the reference's gate, every primitive)?
template <class M>
__device__ __forceinline__ bool bound_hits_any(const float4* __restrict__ table, size_t row0, int k, int g,
                                               const float4* prim, int np) {
    const int lane = threadIdx.x & 31;
    float4 b = table[table_index<M>(row0 + (size_t)k, g)];
    b.w += kEnvInflate;
    bool any = false;
    for (int p = lane; p < np; p += 32) any |= sphere_hits_prim(b, prim + p * kPrimF4);
    return __any_sync(kFull, any);
}

// Learned order, rank r -> sample index: segments in the order perm gives
// (descending MLP score), each walked from its last sample back to its first.
// The MLP scores a segment at its last sample (queue_features_kernel), so the
// scored sample is the first one checked; a collision that starts inside an
// edge whose start is free usually extends to the edge's end, so within a
// segment the later samples are the likelier hits.
__device__ __forceinline__ int learned_rank_to_sample(const uint8_t* perm, int r) {
    return (int)perm[r >> 3] * kSegment + (kSegment - 1 - (r & (kSegment - 1)));
}

// Per-pair walk counts (32 bits: a pair walks at most 32 n C items, far below
// 2^32; the registers and adds are paid on every walk, counting or not).
struct WalkStats {
    unsigned chunks = 0, gates = 0, leaf = 0;
};

// Leaf steps of the overhang-aware walk fetch their item's fields (pair code,
// gate bit, leaf offset) with one shuffle where that measured faster: Fetch
// (+1.5 %); Baxter's larger walk spills more with the packed value live (-1.5 %)
// and keeps one shuffle per field.  The group count separates the two models.
template <class M>
constexpr bool pack_overhang_leaf() {
    return M::num_env_groups <= 16;
}

// Lane g's copy of link group g's leaf range, packed (first leaf | leaf count
// << 16).  The walk fetches a group's range with one shuffle: its lanes hold
// items of different groups, and indexing __constant__ memory with a
// lane-dependent group serialises the access once per distinct group.
struct GroupLanes {
    int fc;
    float cert;  // lane g: group g's certain-hit radius
};

template <class M>
__device__ __forceinline__ GroupLanes group_lanes() {
    const DevTables<M>& T = tab<M>();
    const int g = min(threadIdx.x & 31, M::num_env_groups - 1);
    const int first = T.leaf_begin[g];
    GroupLanes r;
    r.fc = first | ((T.leaf_begin[g + 1] - first) << 16);
    r.cert = T.cert_r[g];
    return r;
}

// Whole warp, one step of 32 (sample, candidate) items: lane's item is sample k
// of the edge (rows from row0) and the packed (primitive, group) pair pr, if
// live.  The bounds are tested (one per item); a bound centre deep enough proves
// a leaf hit (cert_radius); else the leaf work of the items whose bound hit is
// flattened over the warp (item j owns leaf slots [incl_j - cnt_j, incl_j)).
// Returns whether some item collides.
template <class M>
__device__ __forceinline__ bool walk_items(const float4* __restrict__ table, size_t row0, int k, uint32_t pr, bool live,
                                           const float4* prim, int np, const GroupLanes& GL, WalkStats& st) {
    constexpr int G = M::num_env_groups;
    constexpr int GB = group_bits<M>();
    constexpr bool kOver = has_overhang<M>();
    const int lane = threadIdx.x & 31;
    const int g = (int)(pr & ((1u << GB) - 1u)), p = (int)(pr >> GB);
    bool gate = false, cert = false;
    int cnt = 0, first = 0;
    if constexpr (!kOver) {
        // the group's leaf range by shuffle (measured faster for Panda than
        // lane-indexed constant memory)
        const int fc = __shfl_sync(kFull, GL.fc, g);
        const float cr = __shfl_sync(kFull, GL.cert, g);
        first = fc & 0xffff;
        if (live) {
            float4 bs = table[table_index<M>(row0 + (size_t)k, g)];
            bs.w += kEnvInflate;
            float rho;
            const float d2 = prim_core_d2(bs, prim + p * kPrimF4, &rho);
            const float rr = bs.w + rho, rc = rho + cr;
            gate = d2 - rr * rr < 0.0f;
            cert = cr > 0.0f && d2 - rc * rc < 0.0f;
            cnt = gate ? fc >> 16 : 0;
        }
    } else {
        // The overhang-aware walk reads its group fields from constant memory,
        // which leaves its longer body the registers it needs (measured faster
        // for Fetch and Baxter).
        const DevTables<M>& T = tab<M>();
        if (live) {
            float4 bs = table[table_index<M>(row0 + (size_t)k, g)];
            bs.w += kEnvInflate;
            float rho;
            const float d2 = prim_core_d2(bs, prim + p * kPrimF4, &rho);
            const float rr = bs.w + rho;
            gate = d2 - rr * rr < 0.0f;
            const float rc = rho + T.cert_r[g];
            cert = T.cert_r[g] > 0.0f && d2 - rc * rc < 0.0f;
            cnt = gate ? T.leaf_begin[g + 1] - T.leaf_begin[g] : 0;
            // overhanging leaves (listed first) near a primitive the bound misses
            if (!gate && T.over_count[g] > 0) {
                const float rp = rr + T.cull_pad[g];
                if (d2 - rp * rp < 0.0f) cnt = T.over_count[g];
            }
        }
        first = T.leaf_begin[g];
    }
    ++st.chunks;
    if (__any_sync(kFull, cert)) return true;  // a leaf hit is certain: no leaf step
    if (__any_sync(kFull, cnt > 0)) {
        ++st.gates;
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += y;
        }
        const int L = __shfl_sync(kFull, incl, 31);
        // Without overhang a slot needs only its item's sample, primitive
        // and leaf offset: p | (first - exclusive count) << 12, one shuffle.
        int dp = 0;
        if constexpr (!kOver) {
            static_assert(max_prims_of<M>() < 4096, "primitive index packs into 12 bits");
            dp = (int)(((unsigned)(first - (incl - cnt)) << 12) | (unsigned)p);
        } else if constexpr (pack_overhang_leaf<M>()) {
            // the 16-bit pair code (p << GB | g), the gate bit, the leaf offset
            dp = (int)(((unsigned)(first - (incl - cnt)) << 17) | ((unsigned)gate << 16) |
                       ((unsigned)p << GB) | (unsigned)g);
        }
        for (int t0 = 0; t0 < L; t0 += 32) {
            const int t = t0 + lane;
            // owner j: the first lane whose inclusive count exceeds t
            int j = 0;
#pragma unroll
            for (int step = 16; step; step >>= 1) {
                const int v = __shfl_sync(kFull, incl, j + step - 1);
                if (v <= t) j += step;
            }
            int j_k, j_p, leaf, jd = 0;
            if constexpr (!kOver) {
                jd = __shfl_sync(kFull, dp, j);
                j_k = __shfl_sync(kFull, k, j);
                j_p = jd & 4095;
                leaf = t + (jd >> 12);
            } else if constexpr (pack_overhang_leaf<M>()) {
                jd = __shfl_sync(kFull, dp, j);
                j_k = __shfl_sync(kFull, k, j);
                j_p = (jd & 0xffff) >> GB;
                leaf = t + (jd >> 17);
            } else {
                const int j_incl = __shfl_sync(kFull, incl, j);
                const int j_cnt = __shfl_sync(kFull, cnt, j);
                const int j_first = __shfl_sync(kFull, first, j);
                j_k = __shfl_sync(kFull, k, j);
                j_p = __shfl_sync(kFull, p, j);
                leaf = j_first + (t - (j_incl - j_cnt));
            }
            bool hit = false;
            if (t < L) {
                float4 ls = table[table_index<M>(row0 + (size_t)j_k, G + leaf)];
                ls.w += kEnvInflate;
                hit = sphere_hits_prim(ls, prim + j_p * kPrimF4);
            }
            ++st.leaf;
            if constexpr (kOver) {
                const bool j_gate = pack_overhang_leaf<M>() ? ((jd >> 16) & 1) != 0
                                                            : __shfl_sync(kFull, (int)gate, j) != 0;
                if (__any_sync(kFull, hit && j_gate)) return true;
                // Hits of overhanging leaves whose bound missed this primitive:
                // they count once the bound hits some primitive at that sample.
                const int j_g = pack_overhang_leaf<M>() ? (jd & ((1 << GB) - 1)) : __shfl_sync(kFull, g, j);
                uint32_t pend = __ballot_sync(kFull, hit);
                while (pend) {
                    const int u = __ffs(pend) - 1;
                    const int uk = __shfl_sync(kFull, j_k, u);
                    const int ug = __shfl_sync(kFull, j_g, u);
                    if (bound_hits_any<M>(table, row0, uk, ug, prim, np)) return true;
                    pend &= ~__ballot_sync(kFull, j_k == uk && j_g == ug);
                }
            } else {
                if (__any_sync(kFull, hit)) return true;
            }
        }
    }
    return false;
}

// Whole warp: walk (sample rank, pair) items 32 at a time in check order --
// plain reference order, or with `perm` the edge's segments in learned order --
// and return whether some item collides.  Items [w_begin, w_end) are walked
// (w_end < 0: all).  MODE 1 (probe) with overhang: after the chunk that
// completes rank 0, when at least queue_min_items remain, the whole warp calls
// queue(); if that queues the pair, the walk stops with `undecided` set,
// otherwise it goes on in plain order (robots without overhang make that
// decision in check_pair, between two walks).
// Each chunk is a walk_items step and the first one with a hit ends the walk.
// MODE 2 (finish): the CTA's warps split the pair -- this warp walks the
// chunks at w_begin, w_begin + 32 stride, ... and all stop once one of them
// sets *stop.
template <class M, int MODE, class Queue>
__device__ __forceinline__ bool walk_pairs(const float4* __restrict__ table, size_t row0, int n, int C,
                                           const uint16_t* pairs, const float4* prim, int np, const uint8_t* perm,
                                           int queue_min_items, const GroupLanes& GL, bool& undecided,
                                           WalkStats& st, Queue&& queue, int w_begin = 0, int w_end = -1,
                                           int stride = 1, volatile int* stop = nullptr) {
    constexpr bool kOver = has_overhang<M>();
    // rank -> sample: reference order (MODE 0, 1, or no perm), learned order (MODE 2, 3)
    auto sample_of = [&](int rr) {
        if constexpr (MODE == 0 || MODE == 1) {
            return reference_rank_to_sample(rr, n);
        } else {
            return perm ? learned_rank_to_sample(perm, rr) : reference_rank_to_sample(rr, n);
        }
    };
    const int lane = threadIdx.x & 31;
    const int total = kLanes * n * C;
    const int w_last = w_end < 0 ? total : w_end;
    const int w_step = 32 * stride;
    int dr, dc, r, c;
    if (MODE != 2 && w_begin == 0) {
        // a / C for a <= 32 and 1 <= C <= kPairCap: floor((a + 0.5) / C) in FP32 is
        // exact (the quotient stays >= 1 / 2048 away from an integer), and cheaper
        // than an integer division by a runtime divisor.
        const float inv_c = __frcp_rn((float)C);
        dr = (int)(32.5f * inv_c);
        dc = 32 - dr * C;
        r = (int)(((float)lane + 0.5f) * inv_c);
        c = lane - r * C;
    } else {
        dr = w_step / C;
        dc = w_step - dr * C;
        r = (w_begin + lane) / C;
        c = w_begin + lane - r * C;
    }
    bool collide = false;
    {
        for (int w0 = w_begin; w0 < w_last; w0 += w_step) {
            if constexpr (MODE == 2) {  // another warp of the CTA found a hit
                int s = 0;
                if (lane == 0) s = *stop;
                if (__shfl_sync(kFull, s, 0)) break;
            }
            const bool live = w0 + lane < total;
            // c < C on every lane, also past the last item
            if (walk_items<M>(table, row0, live ? sample_of(r) : 0, pairs[c], live, prim, np, GL, st)) {
                collide = true;
                break;
            }
            // Probe (overhang-aware walk): the queue decision stays inside the
            // loop, measured 5 % faster for Baxter than a separate first walk.
            if constexpr (MODE == 1 && kOver) {
                if (w0 == (((C - 1) >> 5) << 5) && total - (w0 + 32) >= queue_min_items && queue()) {
                    undecided = true;
                    break;
                }
            }
            c += dc;
            r += dr;
            if (c >= C) {
                c -= C;
                ++r;
            }
        }
    }
    if constexpr (MODE == 2) {
        if (collide && lane == 0) *stop = 1;
    }
    return collide;
}

// Whole warp: the walk of plain and inline learned checks.  Items are
// (segment rank, candidate) pairs, 32 a step, segments in order (ascending, or
// as `order` ranks them).
//   1. Per item the segment's sphere of the candidate's group against its
//      primitive: a miss rules out all of the segment's samples.  At the middle
//      sample the test is exact where it matters: a bound centre deep enough
//      proves a leaf hit (cert_radius).
//   2. Items that survive, robots whose leaves lie inside their bounds: every
//      leaf of the group at the middle sample, flattened over the warp -- an
//      exact hit test, and with the leaf's reach over the segment a test that
//      rules out its other samples.
//   3. What survives that: the leaf at each of the segment's samples.
// Robots with overhanging leaves take the per-sample bound, certain-hit and leaf
// tests (walk_items) on the segments that survive 1.
// A collision-free pair then costs a test per segment and near-miss instead of
// one per sample: the walk is bound by instruction issue, and on the uneven
// Panda workload most of it went to pairs that never collide.
template <class M>
__device__ __forceinline__ bool walk_segments(const float4* __restrict__ table, const float2* __restrict__ seg,
                                              size_t row0, int n, int C, const uint16_t* pairs, const float4* prim, int np,
                                              const uint8_t* order, const GroupLanes& GL, uint2* scratch,
                                              WalkStats& st) {
    constexpr int G = M::num_env_groups;
    constexpr int GB = group_bits<M>();
    constexpr bool kOver = has_overhang<M>();
    static_assert(kSegment == 8, "segments are expanded eight lanes an item");
    static_assert(kOver || groups_are_rigid<M>(), "a leaf moves no further than its group's frame");
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int S = kLanes / kSegment * n;
    // A learned order's segments, two a lane, by one load a pair: uneven workload's walk
    // 0.597 ms, against 0.623 with a load a step ahead of the rows' (plain order 0.553).
    static_assert(kMaxSegments == 64, "two segments of an order a lane");
    const unsigned ord = order ? reinterpret_cast<const uint16_t*>(order)[lane] : 0u;
    const float4* __restrict__ rows = table + table_index<M>(row0, 0);
    const float2* __restrict__ segs = seg + row0 / kSegment * G;
    // a / C in FP32, exact (walk_pairs)
    const float inv_c = __frcp_rn((float)C);
    const int dr = (int)(32.5f * inv_c), dc = 32 - dr * C;
    int r = (int)(((float)lane + 0.5f) * inv_c);
    int c = lane - r * C;
    const unsigned steps = (unsigned)(((long long)S * C + 31) / 32);
    for (unsigned w = 0; w < steps; ++w) {
        const uint32_t pr = pairs[c];  // c < C on every lane
        const int g = (int)(pr & ((1u << GB) - 1u)), p = (int)(pr >> GB);
        const float cr = __shfl_sync(kFull, GL.cert, g);
        const int fc = __shfl_sync(kFull, GL.fc, g);
        bool near = false, cert = false;
        int k = 0, sg = r;
        float reach = 0.0f;
        if (order) sg = (int)(__shfl_sync(kFull, ord, r >> 1) >> (8 * (r & 1)) & 255u);
        if (r < S) {
            k = sg * kSegment + kSegMid;
            const float4 bs = rows[table_index<M>((size_t)k, g)];
            const float2 sr = segs[(size_t)sg * G + g];
            float rho;
            const float d2 = prim_core_d2(bs, prim + p * kPrimF4, &rho);
            const float rs = sr.x + rho, rc = rho + cr;
            near = d2 - rs * rs < 0.0f;
            cert = cr > 0.0f && d2 - rc * rc < 0.0f;
            reach = sr.y;
        }
        ++st.chunks;
        if (__any_sync(kFull, cert)) return true;
        const unsigned nm = __ballot_sync(kFull, near);
        if (nm) {
            ++st.gates;
            if constexpr (!kOver) {
                const int cnt = near ? fc >> 16 : 0;
                int incl = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += y;
                }
                const int L = __shfl_sync(kFull, incl, 31);
                static_assert(max_prims_of<M>() < 4096, "primitive index packs into 12 bits");
                const int dp = (int)(((unsigned)((fc & 0xffff) - (incl - cnt)) << 12) | (unsigned)p);
                for (int t0 = 0; t0 < L; t0 += 32) {
                    const int t = t0 + lane;
                    int j = 0;  // owner: the first lane whose inclusive count exceeds t
#pragma unroll
                    for (int step = 16; step; step >>= 1) {
                        const int v = __shfl_sync(kFull, incl, j + step - 1);
                        if (v <= t) j += step;
                    }
                    const int jd = __shfl_sync(kFull, dp, j);
                    const int jk = __shfl_sync(kFull, k, j);
                    const float jr = __shfl_sync(kFull, reach, j);
                    const int jp = jd & 4095, leaf = G + t + (jd >> 12);
                    bool hit = false, open = false;
                    if (t < L) {
                        float4 ls = rows[table_index<M>((size_t)jk, leaf)];
                        ls.w += kEnvInflate;
                        float rho;
                        const float d2 = prim_core_d2(ls, prim + jp * kPrimF4, &rho);
                        const float rr = ls.w + rho, ro = rr + jr;
                        hit = d2 - rr * rr < 0.0f;
                        open = d2 - ro * ro < 0.0f;
                    }
                    ++st.leaf;
                    if (__any_sync(kFull, hit)) return true;
                    const unsigned om = __ballot_sync(kFull, open);
                    if (om) {
                        if (open) scratch[__popc(om & lt)] = make_uint2((unsigned)(jk - kSegMid), (unsigned)(leaf << 12 | jp));
                        __syncwarp();
                        const int m = __popc(om) * kSegment;
                        for (int q = lane; q - lane < m; q += 32) {
                            bool h = false;
                            if (q < m) {
                                const uint2 x = scratch[q / kSegment];
                                float4 ls = rows[table_index<M>((size_t)(x.x + (unsigned)(q & (kSegment - 1))),
                                                                (int)(x.y >> 12))];
                                ls.w += kEnvInflate;
                                h = sphere_hits_prim(ls, prim + (x.y & 4095u) * kPrimF4);
                            }
                            ++st.leaf;
                            if (__any_sync(kFull, h)) return true;
                        }
                        __syncwarp();  // scratch is read before the next step's writes
                    }
                }
            } else {
                if (near) scratch[__popc(nm & lt)] = make_uint2((unsigned)(k - kSegMid), pr);
                __syncwarp();
                const int m = __popc(nm) * kSegment;
                for (int q = lane; q - lane < m; q += 32) {
                    const uint2 x = scratch[min(q, m - 1) / kSegment];
                    if (walk_items<M>(table, row0, (int)x.x + (q & (kSegment - 1)), x.y, q < m, prim, np,
                                      GL, st))
                        return true;
                }
                __syncwarp();
            }
        }
        c += dc;
        r += dr;
        if (c >= C) {
            c -= C;
            ++r;
        }
    }
    return false;
}

// ------------------------------------------------------------------ irregular environments
// Whole warp, one row of the sample table against np records: the reference's
// environment test as it stands (fkcc, src/utils.cuh:806-1190) -- each of its groups'
// bounds against every primitive, then the leaves of the groups whose bound hit one
// against every primitive -- with nothing ruled out by distance.
template <class M>
__device__ __forceinline__ bool exact_hit(const float4* row, const float4* prim, int np) {
    const DevTables<M>& L = lane_tab<M>();
    const int lane = threadIdx.x & 31;
    // items [0, spheres x np), primitives innermost
    const int ds = 32 / np, dp = 32 - ds * np;
    auto any_of = [&](const unsigned char* pos, int spheres, auto&& found) {
        int s = lane / np, p = lane - s * np;
        for (int i0 = 0; i0 < spheres * np; i0 += 32) {
            bool hit = false;
            if (s < spheres) {
                float4 c = row[pos[s]];
                c.w += kEnvInflate;
                // (a centre that is not finite is nowhere, as in the culls of the other walks)
                hit = isfinite(c.x + c.y + c.z) && sphere_hits_prim(c, prim + p * kPrimF4);
            }
            if (found(hit, s)) return true;
            s += ds;
            p += dp;
            if (p >= np) {
                p -= np;
                ++s;
            }
        }
        return false;
    };
    unsigned gates = 0u;
    any_of(L.ref_bound, M::num_ref_env_groups, [&](bool hit, int g) {
        gates |= hit ? 1u << g : 0u;
        return false;
    });
    gates = __reduce_or_sync(kFull, gates);
    for (; gates; gates &= gates - 1u) {
        const int g = __ffs((int)gates) - 1;
        const int l0 = L.ref_leaf_begin[g], l1 = L.ref_leaf_begin[g + 1];
        if (any_of(L.ref_leaf + l0, l1 - l0, [](bool hit, int) { return __any_sync(kFull, hit) != 0; })) return true;
    }
    return false;
}

// ... over an edge's samples in the reference's order.
template <class M>
__device__ __noinline__ bool walk_exact(const float4* __restrict__ table, size_t row0, int n, const float4* prim, int np) {
    static_assert(M::num_ref_env_groups <= 32, "a bit per group");
    for (int r = 0; r < kLanes * n; ++r)
        if (exact_hit<M>(table + table_index<M>(row0 + (size_t)reference_rank_to_sample(r, n), 0), prim, np))
            return true;
    return false;
}

// Learned order, whole warp: perm_buf[rank] = segment, the edge's nseg <= 64
// segments in descending MLP score (scores[0 .. nseg)), ties by index, NaN
// last, with first_ahead segment 0 before all others; returns segment 0's rank.
__device__ __forceinline__ int rank_segments(const float* scores, int nseg, uint8_t* perm_buf,
                                             bool first_ahead = false) {
    const int lane = threadIdx.x & 31;
    float v0 = lane < nseg ? scores[lane] : -INFINITY;
    float v1 = lane + 32 < nseg ? scores[lane + 32] : -INFINITY;
    v0 = isnan(v0) ? -INFINITY : v0;
    v1 = isnan(v1) ? -INFINITY : v1;
    if (first_ahead && lane == 0) v0 = INFINITY;
    int rank0 = 0, rank1 = 0;
    for (int i = 0; i < nseg; ++i) {
        const float vi = __shfl_sync(kFull, i < 32 ? v0 : v1, i & 31);
        rank0 += (vi > v0 || (vi == v0 && i < lane)) ? 1 : 0;
        rank1 += (vi > v1 || (vi == v1 && i < lane + 32)) ? 1 : 0;
    }
    if (lane < nseg) perm_buf[rank0] = (uint8_t)lane;
    if (lane + 32 < nseg) perm_buf[rank1] = (uint8_t)(lane + 32);
    return __shfl_sync(kFull, rank0, 0);
}

__device__ __forceinline__ void learned_perm(const CheckParams& P, int seg_row, int nseg, uint8_t* perm_buf) {
    rank_segments(P.logits + seg_row, nseg, perm_buf);
}

// Learned-order queue: lane 0 of a probing warp reserves a queue entry and the
// 4 n MLP rows of the pair's segments with one 64-bit atomic on q_head (entries
// in the high word, rows in the low word).  Returns the pair's first MLP row,
// or -1 when the pair keeps the plain order (more than kMaxSegments segments,
// or the row budget or the queue spent) and the probe walks on.  The low word
// only grows while it is at most row_cap, so it stays far below 2^32.
__device__ __forceinline__ int queue_pair(const CheckParams& P, int e, int env, int n) {
    const int rows = 4 * n;
    if (rows > kMaxSegments) return -1;
    const unsigned used = *reinterpret_cast<volatile const unsigned*>(P.q_head);
    if ((long long)used + rows > P.row_cap) return -1;
    const unsigned long long old = atomicAdd(P.q_head, (1ull << 32) | (unsigned long long)rows);
    const long long idx = (long long)(old >> 32);
    if (idx >= P.q_cap) return -1;
    const unsigned ro = (unsigned)old;
    const int r = (long long)ro + rows <= P.row_cap ? (int)ro : -1;
    P.q_pairs[idx] = make_int2(e, env);
    P.q_rows[idx] = r;
    return r;
}

// The calling warp's 32 scratch entries (walk_segments); at most 8 warps a CTA.
__device__ __forceinline__ uint2* warp_scratch() {
    __shared__ uint2 scratch[8][32];
    return scratch[threadIdx.x >> 5];
}

// Inline learned order of pair (env, e): the segment order scored for the
// environment's cluster; null for edges of too many segments (plain order).
__device__ __forceinline__ const uint8_t* inline_perm(const CheckParams& P, int env, int e, int n) {
    return 4 * n <= kMaxSegments ? P.perms + ((size_t)P.env_cluster[env] * P.num_edges + e) * kMaxSegments : nullptr;
}

// One (environment, edge) pair, whole warp: cull, pair-list compaction and the
// walk.  MODE 0: plain order, full walk.  MODE 1 (learned pipeline, phase 1):
// plain order; a pair still undecided once rank 0 (its first sample) is walked may be
// queued (with MLP rows for its segments) instead of getting a verdict.  MODE 2
// (phase 3): a queued pair (first MLP row seg_row) walked in descending
// segment score, its chunks split over the CTA's warps; MODE 3 (phase 3, one
// warp per pair): the same walk by this warp alone, which writes the verdict.
// `prim` holds the environment's records (shared or global memory), `masks`
// its cull masks, W 64-bit words per mask; `alive` the groups that can hit at
// all (bit g; the others are left out of the cull).
template <class M, int MODE>
__device__ __forceinline__ void check_pair(const CheckParams& P, int env, int e, int seg_row, const float4* prim,
                                           const uint64_t* __restrict__ masks, int np, int W, uint16_t* pairs,
                                           uint8_t* perm_buf, const GroupLanes& GL, int chunk0 = 0, int stride = 1,
                                           volatile int* stop = nullptr, unsigned alive = kFull) {
    constexpr int G = M::num_env_groups;
    constexpr int GB = group_bits<M>();
    const int lane = threadIdx.x & 31;
    const int K = P.pairs_per_warp;
    uint8_t* out = P.results + (size_t)e * P.num_envs + env;
    const int self = P.edge_self[e];
    if (np == 0 || self) {  // a self-colliding sample collides in every environment
        if (lane == 0) {
            *out = self ? 1 : 0;
            if (MODE == 2 && self) *stop = 1;  // the finish kernel writes s_hit as the verdict
        }
        return;
    }
    // Cull: lane g < G takes link g's slab ranges on the set's grid (computed
    // once per edge) and ANDs the environment's three masks over them.
    const int code = lane < G && ((alive >> lane) & 1u) ? P.edge_tri[(size_t)e * G + lane] : -1;
    // Word w of link g's candidate mask (only the packed code stays live
    // across the walk; the three offsets are re-derived where needed).
    auto mask_word = [&](int w) {
        const int tx = code & 1023, ty = (code >> 10) & 1023, tz = code >> 20;
        return __ldg(masks + tx * W + w) & __ldg(masks + (kGridTri + ty) * W + w) &
               __ldg(masks + (2 * kGridTri + tz) * W + w);
    };
    // Compact the surviving (primitive, link) pairs, link-major: lane g counts
    // link g's candidates, an exclusive warp scan gives each link its offset,
    // and every lane writes its own link's pairs in primitive order.
    int cnt = 0;
    if (code >= 0)
        for (int w = 0; w < W; ++w) cnt += __popcll(mask_word(w));
    int off = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, off, o);
        if (lane >= o) off += y;
    }
    const int C = __shfl_sync(kFull, off, 31);
    off -= cnt;

    bool collide = false, undecided = false;
    WalkStats st;
    // Pair list entries [seg0, seg1): lane g writes link g's candidates that
    // fall in the range.
    auto write_seg = [&](int seg0, int seg1) {
        if (cnt > 0 && off < seg1 && off + cnt > seg0) {
            int idx = off;
            for (int w = 0; w < W && idx < seg1; ++w) {
                uint64_t m = mask_word(w);
                while (m && idx < seg1) {
                    const int b = __ffsll((long long)m) - 1;
                    if (idx >= seg0) pairs[idx - seg0] = (uint16_t)(((w * 64 + b) << GB) | lane);
                    ++idx;
                    m &= m - 1;
                }
            }
        }
        __syncwarp();
    };
    auto queue = [&]() {
        int ro = -1;
        if (lane == 0) ro = queue_pair(P, e, env, P.steps[e]);
        return __shfl_sync(kFull, ro, 0) >= 0;
    };
    auto walk_seg = [&](int Cs) {
        const int n = P.steps[e];
        const size_t row0 = (size_t)P.offs[e];
        // Learned order: rank the edge's 4 n segments by their MLP score
        // (descending, ties by index; NaN scores last).
        const int nseg = 4 * n;
        const bool learned = (MODE == 2 || MODE == 3) && seg_row >= 0 && nseg <= kMaxSegments;
        if (learned) {
            learned_perm(P, seg_row, nseg, perm_buf);
            __syncwarp();
        }
        if constexpr (MODE == 1 && !has_overhang<M>()) {
            // Probe: walk up to the chunk that completes rank 0 (the edge's first
            // sample against every candidate, where most colliding pairs
            // collide); when at least queue_min_items items remain, queue the
            // pair for the learned order or, if queue() declines, walk on.  Two
            // plain walks, so no chunk of either pays for the decision.
            const int total = kLanes * n * Cs;
            const int w_dec = (((Cs - 1) >> 5) << 5) + 32;
            if (total - w_dec >= P.queue_min_items) {
                collide = walk_pairs<M, 0>(P.table, row0, n, Cs, pairs, prim, np, nullptr, 0, GL, undecided, st,
                                           queue, 0, w_dec);
                if (!collide) {
                    if (queue())
                        undecided = true;
                    else
                        collide = walk_pairs<M, 0>(P.table, row0, n, Cs, pairs, prim, np, nullptr, 0, GL, undecided,
                                                   st, queue, w_dec);
                }
            } else {
                collide = walk_pairs<M, 0>(P.table, row0, n, Cs, pairs, prim, np, nullptr, 0, GL, undecided, st,
                                           queue);
            }
        } else if constexpr (MODE == 0 || MODE == 4) {
            collide = walk_segments<M>(P.table, P.seg, row0, n, Cs, pairs, prim, np, MODE == 4 ? inline_perm(P, env, e, n) : nullptr,
                                       GL, warp_scratch(), st);
        } else {
            collide = walk_pairs<M, MODE>(P.table, row0, n, Cs, pairs, prim, np, learned ? perm_buf : nullptr,
                                          P.queue_min_items, GL, undecided, st, queue, 32 * chunk0, -1, stride,
                                          stop);
        }
        __syncwarp();  // every lane is done with this segment's pairs
    };
    // Robots whose leaves all lie inside their bounds have a small walk: a
    // separate copy for the usual single-segment case keeps the segment
    // bookkeeping out of it.  The overhang-aware walk stays in one copy.
    bool single = false;
    if constexpr (!has_overhang<M>()) single = C > 0 && C <= K;
    // The whole list fits the buffer (the usual case): no segment bounds to test
    // while writing.
    auto write_all = [&]() {
        if (cnt > 0) {
            int idx = off;
            for (int w = 0; w < W; ++w) {
                uint64_t m = mask_word(w);
                while (m) {
                    const int b = __ffsll((long long)m) - 1;
                    pairs[idx++] = (uint16_t)(((w * 64 + b) << GB) | lane);
                    m &= m - 1;
                }
            }
        }
        __syncwarp();
    };
    if (single) {
        write_all();
        walk_seg(C);
    } else {
        for (int seg0 = 0; seg0 < C && !collide && !undecided; seg0 += K) {
            const int seg1 = min(C, seg0 + K);
            if (C <= K)
                write_all();
            else
                write_seg(seg0, seg1);
            walk_seg(seg1 - seg0);
        }
    }
    if (MODE == 1 && undecided) return;  // queued: the finish pass writes the verdict
    if (MODE == 2) {  // the CTA's warps split the pair: the finish kernel writes the verdict
        if (lane == 0 && P.counters) {
            if (chunk0 == 0) atomicAdd(P.counters + 1, (unsigned long long)C);
            atomicAdd(P.counters + 2, (unsigned long long)st.chunks);
            atomicAdd(P.counters + 3, (unsigned long long)st.gates);
            atomicAdd(P.counters + 4, (unsigned long long)st.leaf);
        }
        return;
    }
    if (lane == 0) {
        *out = collide ? 1 : 0;
        if (P.counters) {
            atomicAdd(P.counters + 0, 1ull);
            atomicAdd(P.counters + 1, (unsigned long long)C);
            atomicAdd(P.counters + 2, (unsigned long long)st.chunks);
            atomicAdd(P.counters + 3, (unsigned long long)st.gates);
            atomicAdd(P.counters + 4, (unsigned long long)st.leaf);
            atomicAdd(P.counters + 5, collide ? 1ull : 0ull);
        }
    }
}

// Pairs whose cull and compaction one warp does together: lanes are grouped G
// to a pair (Panda 10 -> 3 pairs, Fetch 15 -> 2, Baxter 32 -> 1), so the
// per-pair set-up -- slab-range loads, mask ANDs, counts, the scan and the
// list writes -- runs on 30 (or 30, 32) lanes instead of G.
template <class M>
constexpr int pairs_per_setup() {
    return kLanes / M::num_env_groups;
}

// The walk of one pair whose whole candidate list is in `pairs` (C entries,
// C <= pairs_per_warp), whole warp, and its verdict: MODE 0 plain order;
// MODE 1 probe (plain walk of rank 0, then queue the pair or walk on); MODE 4
// inline learned order.
template <class M, int MODE>
__device__ __forceinline__ void walk_listed_pair(const CheckParams& P, int env, int e, int C, const uint16_t* pairs,
                                                 const float4* prim, int np, const GroupLanes& GL) {
    const int lane = threadIdx.x & 31;
    const int n = P.steps[e];
    const size_t row0 = (size_t)P.offs[e];
    bool collide = false, undecided = false;
    WalkStats st;
    auto queue = [&]() {
        int ro = -1;
        if (lane == 0) ro = queue_pair(P, e, env, n);
        return __shfl_sync(kFull, ro, 0) >= 0;
    };
    if constexpr (MODE == 1 && !has_overhang<M>()) {
        // Probe, as in check_pair: two plain walks split at the chunk that
        // completes rank 0, the queue decision between them.
        const int total = kLanes * n * C;
        const int w_dec = (((C - 1) >> 5) << 5) + 32;
        if (total - w_dec >= P.queue_min_items) {
            collide = walk_pairs<M, 0>(P.table, row0, n, C, pairs, prim, np, nullptr, 0, GL, undecided, st, queue, 0,
                                       w_dec);
            if (!collide) {
                if (queue())
                    undecided = true;
                else
                    collide = walk_pairs<M, 0>(P.table, row0, n, C, pairs, prim, np, nullptr, 0, GL, undecided, st,
                                               queue, w_dec);
            }
        } else {
            collide = walk_pairs<M, 0>(P.table, row0, n, C, pairs, prim, np, nullptr, 0, GL, undecided, st, queue);
        }
    } else if constexpr (MODE == 0 || MODE == 4) {
        collide = walk_segments<M>(P.table, P.seg, row0, n, C, pairs, prim, np, MODE == 4 ? inline_perm(P, env, e, n) : nullptr, GL,
                                   warp_scratch(), st);
    } else {
        collide = walk_pairs<M, MODE>(P.table, row0, n, C, pairs, prim, np, nullptr, P.queue_min_items, GL, undecided,
                                      st, queue);
    }
    if (MODE == 1 && undecided) return;  // queued: the finish pass walks, counts and writes the verdict
    if (lane == 0) {
        P.results[(size_t)e * P.num_envs + env] = collide ? 1 : 0;
        if (P.counters) {
            atomicAdd(P.counters + 0, 1ull);
            atomicAdd(P.counters + 1, (unsigned long long)C);
            atomicAdd(P.counters + 2, (unsigned long long)st.chunks);
            atomicAdd(P.counters + 3, (unsigned long long)st.gates);
            atomicAdd(P.counters + 4, (unsigned long long)st.leaf);
            atomicAdd(P.counters + 5, collide ? 1ull : 0ull);
        }
    }
}

// Pairs (env, e0 .. e0 + count - 1), or with a list (env, list[0 .. count).x)
// and their alive groups (.y), count <= pairs_per_setup<M>(), whole warp: lane group s = lane / G culls pair s (lane g of the group ANDs link
// g's three masks), a scan inside each group gives every link its offset,
// the groups' lists are laid out one after another in `pairs` and written in
// one pass; then the warp walks the pairs one at a time.  When the lists do
// not fit the warp's buffer together, each pair goes through check_pair
// (segments).
template <class M, int MODE>
__device__ __forceinline__ void check_pair_group(const CheckParams& P, int env, int e0, int count,
                                                 const uint2* list, const float4* prim,
                                                 const uint64_t* __restrict__ masks, int np, int W, uint16_t* pairs,
                                                 const GroupLanes& GL) {
    constexpr int G = M::num_env_groups;
    constexpr int GB = group_bits<M>();
    constexpr int SUB = pairs_per_setup<M>();
    const int lane = threadIdx.x & 31;
    const int sub = lane / G;
    const int g = lane - sub * G;
    const bool live = sub < count;
    const uint2 entry = list ? list[live ? sub : 0] : make_uint2((unsigned)(e0 + (live ? sub : 0)), kFull);
    const int e = (int)entry.x;
    const int self = live ? P.edge_self[e] : 1;
    const int code = (live && !self && np > 0 && ((entry.y >> g) & 1u)) ? P.edge_tri[(size_t)e * G + g] : -1;
    auto mask_word = [&](int w) {
        const int tx = code & 1023, ty = (code >> 10) & 1023, tz = code >> 20;
        return __ldg(masks + tx * W + w) & __ldg(masks + (kGridTri + ty) * W + w) &
               __ldg(masks + (2 * kGridTri + tz) * W + w);
    };
    // One mask word (np <= 64, the common case) stays in registers for the
    // list writes; more words are re-read there.
    int cnt = 0;
    uint64_t m1 = 0;
    if (code >= 0) {
        if (W == 1) {
            m1 = mask_word(0);
            cnt = __popcll(m1);
        } else {
            for (int w = 0; w < W; ++w) cnt += __popcll(mask_word(w));
        }
    }
    // inclusive scan inside each group of G lanes
    int inc = cnt;
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
        const int y = __shfl_up_sync(kFull, inc, o);
        if (g >= o) inc += y;
    }
    // every pair's candidate count and list base
    int Cs[SUB], base[SUB], total = 0;
#pragma unroll
    for (int t = 0; t < SUB; ++t) {
        Cs[t] = __shfl_sync(kFull, inc, t * G + G - 1);
        base[t] = total;
        total += t < count ? Cs[t] : 0;
    }
    if (total > P.pairs_per_warp) {
        for (int t = 0; t < count; ++t)
            check_pair<M, MODE>(P, env, list ? (int)list[t].x : e0 + t, -1, prim, masks, np, W, pairs, nullptr, GL, 0,
                                1, nullptr, list ? list[t].y : kFull);
        return;
    }
    if (cnt > 0) {
        int idx = inc - cnt;
#pragma unroll
        for (int t = 0; t < SUB; ++t)
            if (t == sub) idx += base[t];
        if (W == 1) {  // 32-bit halves: cheaper bit steps than 64-bit ones
            uint32_t lo = (uint32_t)m1, hi = (uint32_t)(m1 >> 32);
            while (lo) {
                pairs[idx++] = (uint16_t)(((__ffs((int)lo) - 1) << GB) | g);
                lo &= lo - 1u;
            }
            while (hi) {
                pairs[idx++] = (uint16_t)(((__ffs((int)hi) + 31) << GB) | g);
                hi &= hi - 1u;
            }
        } else {
            for (int w = 0; w < W; ++w) {
                uint64_t m = mask_word(w);
                while (m) {
                    const int b = __ffsll((long long)m) - 1;
                    pairs[idx++] = (uint16_t)(((w * 64 + b) << GB) | g);
                    m &= m - 1;
                }
            }
        }
    }
    __syncwarp();
#pragma unroll 1
    for (int t = 0; t < count; ++t) {
        const int et = __shfl_sync(kFull, e, t * G);
        const int self_t = __shfl_sync(kFull, self, t * G);
        if (np == 0 || self_t) {  // decided without a walk (not counted as walked, as in check_pair)
            if (lane == 0) P.results[(size_t)et * P.num_envs + env] = self_t ? 1 : 0;
            continue;
        }
        if (Cs[t] == 0) {  // nothing survives the cull: free
            if (lane == 0) {
                P.results[(size_t)et * P.num_envs + env] = 0;
                if (P.counters) atomicAdd(P.counters + 0, 1ull);
            }
            continue;
        }
        int bt = 0;
#pragma unroll
        for (int u = 0; u < SUB; ++u)
            if (u == t) bt = base[u];
        walk_listed_pair<M, MODE>(P, env, et, Cs[t], pairs + bt, prim, np, GL);
    }
    __syncwarp();  // every lane is done with the lists before the next group's writes
}

// Bytes of an environment's primitive records (what a CTA stages).
__device__ __forceinline__ uint32_t record_bytes_of(float4 h1) {
    return (__float_as_uint(h1.w) & 0xffffu) * kPrimF4 * 16u;
}

// Check CTAs are compiled for M::check_warps_per_sm resident warps per SM (a
// register budget of 65536 / (32 x that) per thread), at most 32 CTAs per SM.
template <class M, int WARPS>
constexpr int check_min_ctas() {
    return M::check_warps_per_sm / WARPS < 32 ? M::check_warps_per_sm / WARPS : 32;
}

// Voxel lookup: the word of the voxel nearest to c and the squared distance r2 (m^2,
// rounded up) of c from its centre; c's signed distance to the nearest primitive
// then lies in [lo - sqrt(r2), lo + kVoxStep + 2 kVoxSlack + sqrt(r2)), lo =
// voxel_low(word).
struct VoxelGrid {
    const uint16_t* vox;
    float inv_h, bx, by, bz, mx, my, mz, sy, sz, h2;
    __device__ __forceinline__ VoxelGrid(const ProbeGrid& V, const uint16_t* words)
        : vox(words), inv_h(V.inv_h), bx(-V.ox * V.inv_h), by(-V.oy * V.inv_h), bz(-V.oz * V.inv_h),
          mx((float)(V.nx - 1)), my((float)(V.ny - 1)), mz((float)(V.nz - 1)), sy((float)V.nx),
          sz((float)(V.nx * V.ny)), h2(V.h * V.h * 1.0002f) {}
    __device__ __forceinline__ unsigned at(float4 c, float& r2) const {
        constexpr float kRound = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer
        // position in voxels from the centre of voxel 0, the nearest voxel, the offset from it
        const float fx = fmaf(c.x, inv_h, bx), fy = fmaf(c.y, inv_h, by), fz = fmaf(c.z, inv_h, bz);
        const float ix = (fminf(fmaxf(fx, 0.0f), mx) + kRound) - kRound;
        const float iy = (fminf(fmaxf(fy, 0.0f), my) + kRound) - kRound;
        const float iz = (fminf(fmaxf(fz, 0.0f), mz) + kRound) - kRound;
        const float rx = fx - ix, ry = fy - iy, rz = fz - iz;
        r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz)) * h2;
        return vox[(int)fmaf(iz, sz, fmaf(iy, sy, ix))];
    }
    // ... the voxel's primitive alone.
    __device__ __forceinline__ unsigned nearest(float4 c) const {
        float r2;
        return at(c, r2) >> 8;
    }
};
__device__ __forceinline__ float voxel_low(unsigned word) {
    return fmaf((float)(word & 255u), kVoxStep, kVoxMin - kVoxSlack);
}

// Is c, looked up as (word, r2), certainly within `reach` of some primitive
// (signed distance below it)?  By the voxel's distance where that decides, else by
// the exact test on the voxel's nearest primitive (a non-finite centre is left to
// the walk).
__device__ __forceinline__ bool voxel_hit(float4 c, unsigned word, float r2, float lo, float reach, const float4* prim) {
    const float up = reach - (lo + kVoxStep + 2.0f * kVoxSlack), dn = lo - reach;
    if (up > 0.0f && up * up > r2) return true;
    if ((dn > 0.0f && dn * dn > r2) || !(r2 < 1e30f) || (word >> 8) == kVoxUnknown) return false;
    float rho;
    const float d2 = prim_core_d2(c, prim + (word >> 8) * kPrimF4, &rho);
    const float rc = rho + reach;
    return d2 - rc * rc < 0.0f;
}

// Probe of pair (env, e), one lane per pair (decided: the lane has none).  Per
// group P.mid holds the bound's centre at the edge's middle sample and the
// radius R of the sphere around it that holds the group's leaves, inflated,
// over all of the edge's samples.  A centre within the certain-hit radius
// (cert_radius) of a primitive proves a leaf hit at the middle sample; a distance
// above R proves the group free along the whole edge.  Returns whether a hit is
// proved; `alive` gets the groups not proved free (none: the pair is free), `near`
// those whose bound may touch a primitive at the middle sample.
// Groups in descending certain-hit radius; the warp leaves once all its lanes are
// decided.
template <class M>
__device__ __forceinline__ bool probe_pair(const CheckParams& P, int e, bool decided, const VoxelGrid& V,
                                           const float4* prim, unsigned& alive, unsigned& near) {
    const DevTables<M>& T = tab<M>();
    bool hit = false;
    alive = near = 0u;
    for (int i = 0; i < M::num_env_groups; ++i) {
        if (__all_sync(kFull, decided)) break;
        const int g = T.probe_group[i];
        if (!decided) {
            const float4 c = P.mid[(size_t)g * P.num_edges + e];
            const float kappa = T.cert_r[g];
            float r2;
            const unsigned w = V.at(c, r2);
            const float lo = voxel_low(w), miss = lo - c.w;
            if (miss > 0.0f && miss * miss > r2) continue;
            alive |= 1u << g;
            const float clear = lo - T.gate_r[g];
            if (!(clear > 0.0f && clear * clear > r2)) near |= 1u << g;
            if (kappa > 0.0f) hit = decided = voxel_hit(c, w, r2, lo, kappa, prim);
        }
    }
    return hit;
}

// Second probe of an undecided pair, whole warp, lanes over the leaves (a row's are
// contiguous): those of its `near` groups at the middle sample against the nearest
// primitive of the voxel they lie in.  A hit is a leaf hit the walk would find:
// exactly its test for robots whose leaves lie inside their bounds; for the others
// only leaves inside their bounds count, by kCertMargin (a hit then implies the
// bound's).  Most pairs that collide in contact shallower than the groups'
// certain-hit radii end here.  bits[k]: the group bit of this lane's leaf 32 k +
// lane, 0 where none counts.
template <class M>
constexpr int kLeafSteps = (M::num_env_leaves + 31) / 32;

template <class M>
__device__ __forceinline__ void leaf_bits(unsigned (&bits)[kLeafSteps<M>]) {
    const DevTables<M>& L = lane_tab<M>();
#pragma unroll
    for (int k = 0; k < kLeafSteps<M>; ++k) {
        const int l = 32 * k + (threadIdx.x & 31);
        bits[k] = l < M::num_env_leaves && !L.leaf_over[l] ? 1u << L.leaf_group[l] : 0u;
    }
}

template <class M>
__device__ __forceinline__ bool probe_leaves(const CheckParams& P, int e, unsigned near, const VoxelGrid& V,
                                             const float4* prim, const unsigned (&bits)[kLeafSteps<M>]) {
    constexpr float kInflate = has_overhang<M>() ? kEnvInflate - (float)kCertMargin : kEnvInflate;
    const float4* row = P.table + table_index<M>((size_t)P.offs[e] + 16 * (size_t)P.steps[e], M::num_env_groups) +
                        (threadIdx.x & 31);
#pragma unroll
    for (int k = 0; k < kLeafSteps<M>; ++k) {
        const bool mine = (near & bits[k]) != 0u;
        if (!__any_sync(kFull, mine)) continue;
        bool hit = false;
        if (mine) {
            const float4 c = row[32 * k];
            const unsigned id = V.nearest(c);
            // (a non-finite centre is left to the walk)
            if (id != kVoxUnknown && fabsf(c.x + c.y + c.z) < 1e30f) {
                float rho;
                const float d2 = prim_core_d2(c, prim + id * kPrimF4, &rho);
                const float rr = c.w + kInflate + rho;
                hit = d2 - rr * rr < 0.0f;
            }
        }
        if (__any_sync(kFull, hit)) return true;
    }
    return false;
}

// First pass of a check with probe grids: CTA = one environment x Q.batch
// edges, one lane per pair (probe_pair), then one warp per undecided pair
// (probe_leaves).  Decided pairs get their verdict; the others go to the queue (Q)
// as (edge, alive groups), contiguous per CTA, with one work item per Q.chunk of
// them.  Bound by instruction issue.  On the uneven Panda workload (1000 x 10000)
// walking every pair took 390 warp instructions a pair and 4.2 ms.  The bounds
// alone decide 84 % of the pairs in 0.33 ms (29 instructions a pair), probe and walk
// 1.38 ms; the leaves settle two thirds of the colliding rest: 0.70 ms (61 a pair),
// probe and walk 1.19 ms.  Five CTAs an SM against four: 1.19 and 1.23 ms.
constexpr int kProbeThreads = 256;
constexpr int kProbeCtas = 5;

template <class M>
__global__ void __launch_bounds__(kProbeThreads, kProbeCtas) probe_kernel(CheckParams P, ProbeQueue Q, int env0) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t bar;
    __shared__ int s_cnt, s_open, s_base, s_item;
    if (P.offs[P.num_edges] > P.cap_rows) return;
    const int env = env0 + blockIdx.x, e0 = blockIdx.y * Q.batch;
    const int nb = min(Q.batch, P.num_edges - e0);
    const int lane = threadIdx.x & 31;
    const float4 h0 = P.env_hdr[2 * env + 0];
    const float4 h1 = P.env_hdr[2 * env + 1];
    const uint32_t bytes = record_bytes_of(h1);
    const int np = (int)(__float_as_uint(h1.w) & 0xffffu);
    if (__float_as_uint(h1.z) & kEnvIrregular) return;  // exact_kernel's
    const bool probe = np > 0;
    const float4* prim = reinterpret_cast<const float4*>(smem);
    uint2* list = reinterpret_cast<uint2*>(smem + P.blob_smem + P.probe.stride);
    unsigned* list_near = reinterpret_cast<unsigned*>(list + Q.batch);
    if (threadIdx.x == 0) {
        s_cnt = s_open = 0;
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (probe) {
        if (threadIdx.x == 0) {
            bulk_expect(&bar, bytes + P.probe.stride);
            bulk_copy_part(smem, P.blobs + (size_t)__float_as_uint(h0.w), bytes, &bar);
            bulk_copy_part(smem + P.blob_smem, P.probe.vox + (size_t)env * (P.probe.stride / 2), P.probe.stride, &bar);
        }
        // One path for the whole CTA (see check_kernel).
        const bool ok = mbar_wait_bounded(&bar, 0u, 1u << 22);
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) atomicOr(P.error_flag, 1);
            mbar_wait_bounded(&bar, 0u, 1u << 22);
            return;
        }
    }
    const VoxelGrid V(P.probe, reinterpret_cast<const uint16_t*>(smem + P.blob_smem));
    // Undecided pairs to list[from s_cnt on]; verdicts of the decided ones.
    auto settle = [&](bool live, bool hit, bool open, int e, unsigned alive, unsigned near) {
        if (live && !open) P.results[(size_t)e * P.num_envs + env] = hit ? 1 : 0;
        const unsigned m = __ballot_sync(kFull, open);
        int at = 0;
        if (lane == 0 && m) at = atomicAdd(&s_cnt, __popc(m));
        at = __shfl_sync(kFull, at, 0);
        if (open) {
            at += __popc(m & ((1u << lane) - 1u));
            list[at] = make_uint2((unsigned)e, alive);
            list_near[at] = near;
        }
    };
    auto count = [&](bool decided, bool hit) {  // pairs settled here (self-colliding ones are not counted)
        const unsigned dec = __ballot_sync(kFull, decided), col = __ballot_sync(kFull, hit);
        if (lane == 0) {
            atomicAdd(P.counters + 0, (unsigned long long)__popc(dec));
            atomicAdd(P.counters + 5, (unsigned long long)__popc(col));
        }
    };
    for (int i0 = threadIdx.x & ~31; i0 < nb; i0 += kProbeThreads) {
        const int i = i0 + lane, e = e0 + min(i, nb - 1);
        const int self = i < nb ? P.edge_self[e] : 1;
        unsigned alive = np > 0 ? kFull : 0u, near = 0u;
        bool hit = self != 0;
        if (probe) hit = probe_pair<M>(P, e, hit, V, prim, alive, near) || hit;
        const bool open = !hit && alive != 0u;
        settle(i < nb, hit, open, e, alive, near);
        if (P.counters && np > 0) count(!open && !self, hit && !self);
    }
    __syncthreads();
    const int n = s_cnt;
    unsigned bits[kLeafSteps<M>];
    leaf_bits<M>(bits);
    for (int i = threadIdx.x >> 5; i < n; i += kProbeThreads / 32) {
        const unsigned near = list_near[i];  // none without a probe
        if (near == 0u) continue;
        const int e = (int)list[i].x;
        if (probe_leaves<M>(P, e, near, V, prim, bits)) {
            if (lane == 0) {
                P.results[(size_t)e * P.num_envs + env] = 1;
                list[i].y = 0u;  // settled
            }
            if (P.counters) count(lane == 0, lane == 0);
        }
    }
    __syncthreads();
    for (int i0 = threadIdx.x & ~31; i0 < n; i0 += kProbeThreads) {
        const unsigned m = __ballot_sync(kFull, i0 + lane < n && list[i0 + lane].y != 0u);
        if (lane == 0 && m) atomicAdd(&s_open, __popc(m));
    }
    __syncthreads();
    const int u = s_open;
    if (u == 0) return;
    const int items = (u + Q.chunk - 1) / Q.chunk;
    if (threadIdx.x == 0) {
        s_base = atomicAdd(Q.head + 0, u);
        s_item = atomicAdd(Q.head + 1, items);
        s_cnt = 0;
    }
    __syncthreads();
    for (int i0 = threadIdx.x & ~31; i0 < n; i0 += kProbeThreads) {
        const uint2 x = i0 + lane < n ? list[i0 + lane] : make_uint2(0u, 0u);
        const unsigned m = __ballot_sync(kFull, x.y != 0u);
        int at = 0;
        if (lane == 0 && m) at = atomicAdd(&s_cnt, __popc(m));
        at = s_base + __shfl_sync(kFull, at, 0);
        if (x.y) Q.entries[at + __popc(m & ((1u << lane) - 1u))] = x;
    }
    for (int i = threadIdx.x; i < items; i += kProbeThreads)
        Q.items[s_item + i] = make_int4(env, s_base + i * Q.chunk, min(Q.chunk, u - i * Q.chunk), 0);
}

// Resident warps per SM the walk is compiled for: 48 registers a thread.  Swept
// on 1000 x 20000 stress pairs: 5.97 ms at 48 warps, 5.16 at 40, 5.73 at 32,
// 6.34 at 24 (with a probe of 0.77 ms by the bounds alone; 4.78 since the probe
// tests leaves too).
constexpr int kWalkWarps = 40;

template <class M, int WARPS>
constexpr int walk_min_ctas() {
    return kWalkWarps / WARPS < 32 ? kWalkWarps / WARPS : 32;
}

// Second pass: persistent CTAs pull work items (an environment and up to
// Q.chunk of its undecided pairs), stage the environment's records when it
// changes, and their warps take pairs_per_setup pairs at a time from a shared
// counter.  Items of a few dozen pairs even out what a tile of edges could not:
// the undecided pairs of a set cluster in its sparse environments.
template <class M, int WARPS, int MODE>
__global__ void __launch_bounds__(WARPS * 32, walk_min_ctas<M, WARPS>()) walk_kernel(CheckParams P, ProbeQueue Q) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t bar;
    __shared__ int4 s_work;
    __shared__ int s_next;
    constexpr int SUB = pairs_per_setup<M>();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total = Q.head[1];
    const float4* prim = reinterpret_cast<const float4*>(smem);
    uint16_t* pairs = reinterpret_cast<uint16_t*>(smem + P.blob_smem) + (size_t)warp * P.pairs_per_warp;
    const GroupLanes GL = group_lanes<M>();
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    int staged = -1;
    uint32_t phase = 0;
    for (;;) {
        __syncthreads();  // every warp is done with the previous item
        if (threadIdx.x == 0) {
            const int i = atomicAdd(Q.head + 2, 1);
            s_work = i < total ? Q.items[i] : make_int4(-1, 0, 0, 0);
            s_next = 0;
        }
        __syncthreads();
        const int4 work = s_work;
        const int env = work.x;
        if (env < 0) break;
        const float4 h0 = P.env_hdr[2 * env + 0];
        const float4 h1 = P.env_hdr[2 * env + 1];
        if (env != staged) {  // an item's environment has primitives
            if (threadIdx.x == 0)
                bulk_copy_g2s(smem, P.blobs + (size_t)__float_as_uint(h0.w), record_bytes_of(h1), &bar);
            const bool ok = mbar_wait_bounded(&bar, phase, 1u << 22);
            if (__syncthreads_or(!ok)) {  // one path for the whole CTA (see check_kernel)
                if (threadIdx.x == 0) atomicOr(P.error_flag, 1);
                mbar_wait_bounded(&bar, phase, 1u << 22);
                break;
            }
            phase ^= 1u;
            staged = env;
        }
        const uint32_t shape = __float_as_uint(h1.w);
        const int np = (int)(shape & 0xffffu), W = (int)(shape >> 16);
        const uint64_t* __restrict__ masks =
            reinterpret_cast<const uint64_t*>(P.blobs + (size_t)__float_as_uint(h0.w) + (size_t)np * kPrimF4);
        const uint2* list = Q.entries + work.y;
        for (;;) {
            int slot = 0;
            if (lane == 0) slot = atomicAdd(&s_next, SUB);
            slot = __shfl_sync(kFull, slot, 0);
            if (slot >= work.z) break;
            if constexpr (SUB > 1)
                check_pair_group<M, MODE>(P, env, 0, min(SUB, work.z - slot), list + slot, prim, masks, np, W, pairs,
                                          GL);
            else
                check_pair<M, MODE>(P, env, (int)list[slot].x, -1, prim, masks, np, W, pairs, nullptr, GL, 0, 1,
                                    nullptr, list[slot].y);
        }
    }
}

// check_tile processes the edges of one (environment, edge tile) work item
// (modes 0, 1 and 4) with the environment's records already staged in shared
// memory.  Each warp takes pairs_per_setup consecutive edges at a time.
template <class M, int WARPS, int MODE>
__device__ __forceinline__ void check_tile(const CheckParams& P, int env, int tile, int n_slots,
                                           const unsigned char* smem, float4 h0, float4 h1, int* s_next) {
    constexpr int SUB = pairs_per_setup<M>();
    const int e_begin = tile * P.edges_per_cta;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t shape = __float_as_uint(h1.w);
    const int np = (int)(shape & 0xffffu);
    const int W = (int)(shape >> 16);  // 64-bit words per primitive mask
    const float4* prim = reinterpret_cast<const float4*>(smem);
    // the mask tables stay in global memory (read through L1): each pair reads
    // only the few words its slab ranges select
    const uint64_t* __restrict__ masks =
        reinterpret_cast<const uint64_t*>(P.blobs + (size_t)__float_as_uint(h0.w) + (size_t)np * kPrimF4);
    uint16_t* pairs =
        reinterpret_cast<uint16_t*>(const_cast<unsigned char*>(smem) + P.blob_smem) + (size_t)warp * P.pairs_per_warp;
    const GroupLanes GL = group_lanes<M>();
    // Warps take the tile's next pass from a shared counter: a pass costs
    // from one chunk (a pair colliding at its first sample) to dozens (a
    // collision-free pair), so a fixed stride leaves warps idle while the
    // CTA's last one finishes.
    for (;;) {
        int slot = 0;
        if (lane == 0) slot = atomicAdd(s_next, SUB);
        slot = __shfl_sync(kFull, slot, 0);
        if (slot >= n_slots) break;
        if constexpr (SUB > 1)
            check_pair_group<M, MODE>(P, env, e_begin + slot, min(SUB, n_slots - slot), nullptr, prim, masks, np, W,
                                      pairs, GL);
        else
            check_pair<M, MODE>(P, env, e_begin + slot, -1, prim, masks, np, W, pairs, nullptr, GL);
    }
}

__device__ __forceinline__ int tile_slots(const CheckParams& P, int tile) {
    const int e_begin = tile * P.edges_per_cta;
    return min(P.edges_per_cta, P.num_edges - e_begin);
}

// One CTA per (environment, edge tile): blockIdx.x = environment, blockIdx.y = tile.
template <class M, int WARPS, int MODE>
__global__ void __launch_bounds__(WARPS * 32, check_min_ctas<M, WARPS>()) check_kernel(CheckParams P) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t bar;
    __shared__ int s_next;
    const int env = blockIdx.x, tile = blockIdx.y;
    const int n_slots = tile_slots(P, tile);
    if (n_slots <= 0 || P.offs[P.num_edges] > P.cap_rows) return;
    const float4 h0 = P.env_hdr[2 * env + 0];
    const float4 h1 = P.env_hdr[2 * env + 1];
    if (__float_as_uint(h1.z) & kEnvIrregular) return;  // exact_kernel's
    const uint32_t bytes = record_bytes_of(h1);
    if (threadIdx.x == 0) s_next = 0;
    if (bytes) {
        if (threadIdx.x == 0) {
            mbar_init(&bar, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
        if (threadIdx.x == 0) bulk_copy_g2s(smem, P.blobs + (size_t)__float_as_uint(h0.w), bytes, &bar);
        // The whole CTA takes one path: if any thread gave up, all flag, wait once
        // more (bounded) for the copy in flight, and return together.
        const bool ok = mbar_wait_bounded(&bar, 0u, 1u << 22);
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) atomicOr(P.error_flag, 1);
            mbar_wait_bounded(&bar, 0u, 1u << 22);
            return;
        }
    } else {
        __syncthreads();  // s_next is set before any warp takes a pass
    }
    check_tile<M, WARPS, MODE>(P, env, tile, n_slots, smem, h0, h1, &s_next);
}

// The pairs of the irregular environments, one warp a pair, environments outermost;
// records are read through L1.  Every sample takes every test (300 x 3000 pairs of the
// uneven law, every cuboid stretched: 8.8 ms; a walk by samples with cull and bounds,
// which misses collisions there, 1.5): such environments are the exception.
constexpr int kExactWarps = 4;

template <class M>
__global__ void __launch_bounds__(32 * kExactWarps) exact_kernel(CheckParams P) {
    const int lane = threadIdx.x & 31, E = P.num_edges;
    if (P.offs[E] > P.cap_rows) return;
    const long long pairs = (long long)P.num_irregular * E, step = (long long)gridDim.x * kExactWarps;
    for (long long i = (long long)blockIdx.x * kExactWarps + (threadIdx.x >> 5); i < pairs; i += step) {
        const int env = P.irregular[i / E], e = (int)(i % E);
        const float4 h0 = P.env_hdr[2 * env], h1 = P.env_hdr[2 * env + 1];
        const int np = (int)(__float_as_uint(h1.w) & 0xffffu);  // at least one
        const bool self = P.edge_self[e] != 0;
        const bool hit = self || walk_exact<M>(P.table, (size_t)P.offs[e], P.steps[e],
                                               P.blobs + (size_t)__float_as_uint(h0.w), np);
        if (lane == 0) {
            P.results[(size_t)e * P.num_envs + env] = hit ? 1 : 0;
            if (P.counters && !self) {
                atomicAdd(P.counters + 0, 1ull);
                atomicAdd(P.counters + 5, hit ? 1ull : 0ull);
            }
        }
    }
}

// Learned order, phase 3: each CTA pulls queued pairs from finish_counter, one
// at a time, and its warps split each pair's walk (warp w takes chunks w,
// w + WARPS, ... of the learned order; a hit in any stops all): the queued
// pairs are the longest walks of the check, and one warp per pair would leave
// the slowest single walk as the kernel's critical path.  The verdict is the
// OR over all items, so the split changes no verdict.  Consecutive pulls
// belong to different environments, so the primitive records are read from
// global memory (L1/L2) rather than staged; shared memory holds the warps'
// pair lists only (each warp compacts its own copy).  Compiled for at most 32
// resident warps per SM: its walk holds 64-bit record pointers and the segment
// permutation, and spills in the plain check kernel's tighter register budget.
template <class M, int WARPS>
constexpr int finish_min_ctas() {
    return (M::check_warps_per_sm < 32 ? M::check_warps_per_sm : 32) / WARPS;
}

// Learned order, phase 3, one warp per queued pair: each warp pulls entries
// from finish_counter on its own, culls, ranks the segments and walks the
// pair in learned order (MODE 3).  No CTA barrier per pair, so many pairs are
// in flight per SM; a long walk is not split, so the longest queued pair sets
// the tail.  Compiled like finish_kernel.
template <class M, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, finish_min_ctas<M, WARPS>()) finish_warp_kernel(CheckParams P) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint8_t s_perm[WARPS][kMaxSegments];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long queued = (long long)(*P.q_head >> 32);
    const int total = (int)min(queued, (long long)P.q_cap);
    uint16_t* pairs = reinterpret_cast<uint16_t*>(smem) + (size_t)warp * P.pairs_per_warp;
    const GroupLanes GL = group_lanes<M>();
    for (;;) {
        int i = 0;
        if (lane == 0) i = atomicAdd(P.finish_counter, 1);
        i = __shfl_sync(kFull, i, 0);
        if (i >= total) break;
        const int ro = P.q_rows[i];
        if (ro < 0) continue;  // the probe walked this pair on
        const int2 pe = P.q_pairs[i];
        const float4 h0 = P.env_hdr[2 * pe.y + 0];
        const float4 h1 = P.env_hdr[2 * pe.y + 1];
        const uint32_t shape = __float_as_uint(h1.w);
        const int np = (int)(shape & 0xffffu);
        const int W = (int)(shape >> 16);
        const float4* prim = P.blobs + __float_as_uint(h0.w);
        const uint64_t* masks = reinterpret_cast<const uint64_t*>(prim + (size_t)np * kPrimF4);
        check_pair<M, 3>(P, pe.y, pe.x, ro, prim, masks, np, W, pairs, s_perm[warp], GL);
    }
}

template <class M, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, finish_min_ctas<M, WARPS>()) finish_kernel(CheckParams P) {
    constexpr int G = M::num_env_groups;
    constexpr int GB = group_bits<M>();
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint8_t s_perm[WARPS][kMaxSegments];
    __shared__ int s_item, s_C;
    __shared__ volatile int s_hit;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long queued = (long long)(*P.q_head >> 32);
    const int total = (int)min(queued, (long long)P.q_cap);
    // Warp 0 culls and compacts each pair once into the CTA's list (all the
    // warps' buffers together); a pair whose list would not fit falls back to
    // per-warp lists (each warp its own copy, walked in segments).
    uint16_t* cta_pairs = reinterpret_cast<uint16_t*>(smem);
    const int cta_cap = WARPS * P.pairs_per_warp;
    uint16_t* pairs = cta_pairs + (size_t)warp * P.pairs_per_warp;
    const GroupLanes GL = group_lanes<M>();
    for (;;) {
        if (threadIdx.x == 0) {
            s_item = atomicAdd(P.finish_counter, 1);
            s_hit = 0;
        }
        __syncthreads();
        const int i = s_item;
        if (i >= total) break;  // CTA-uniform
        const int ro = P.q_rows[i];
        const int2 pe = ro >= 0 ? P.q_pairs[i] : make_int2(0, 0);
        if (ro >= 0) {  // ro < 0: the probe walked this pair on
            const int env = pe.y, e = pe.x;
            const float4 h0 = P.env_hdr[2 * env + 0];
            const float4 h1 = P.env_hdr[2 * env + 1];
            const uint32_t shape = __float_as_uint(h1.w);
            const int np = (int)(shape & 0xffffu);
            const int W = (int)(shape >> 16);
            const float4* prim = P.blobs + __float_as_uint(h0.w);
            const uint64_t* masks = reinterpret_cast<const uint64_t*>(prim + (size_t)np * kPrimF4);
            const int n = P.steps[e];
            const int nseg = 4 * n;
            if (warp == 0) {
                // A queued pair passed the probe's self-collision test and has
                // candidates; the cull below repeats the probe's exactly.
                const int code = lane < G ? P.edge_tri[(size_t)e * G + lane] : -1;
                auto mask_word = [&](int w) {
                    const int tx = code & 1023, ty = (code >> 10) & 1023, tz = code >> 20;
                    return __ldg(masks + tx * W + w) & __ldg(masks + (kGridTri + ty) * W + w) &
                           __ldg(masks + (2 * kGridTri + tz) * W + w);
                };
                int cnt = 0;
                if (code >= 0 && np > 0)
                    for (int w = 0; w < W; ++w) cnt += __popcll(mask_word(w));
                int off = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(kFull, off, o);
                    if (lane >= o) off += y;
                }
                const int C = __shfl_sync(kFull, off, 31);
                off -= cnt;
                const bool fits = C <= cta_cap && nseg <= kMaxSegments;
                if (fits && cnt > 0) {
                    int idx = off;
                    for (int w = 0; w < W; ++w) {
                        uint64_t m = mask_word(w);
                        while (m) {
                            const int b = __ffsll((long long)m) - 1;
                            cta_pairs[idx++] = (uint16_t)(((w * 64 + b) << GB) | lane);
                            m &= m - 1;
                        }
                    }
                }
                if (fits) learned_perm(P, ro, nseg, s_perm[0]);
                if (lane == 0) {
                    s_C = fits ? C : -1;
                    if (fits && P.counters) atomicAdd(P.counters + 1, (unsigned long long)C);
                }
            }
            __syncthreads();
            const int C = s_C;
            if (C > 0) {
                bool undecided = false;
                WalkStats st;
                walk_pairs<M, 2>(P.table, (size_t)P.offs[e], n, C, cta_pairs, prim, np, s_perm[0], 0, GL, undecided,
                                 st, [] { return false; }, 32 * warp, -1, WARPS, &s_hit);
                if (lane == 0 && P.counters) {
                    atomicAdd(P.counters + 2, (unsigned long long)st.chunks);
                    atomicAdd(P.counters + 3, (unsigned long long)st.gates);
                    atomicAdd(P.counters + 4, (unsigned long long)st.leaf);
                }
            } else if (C < 0) {
                check_pair<M, 2>(P, env, e, ro, prim, masks, np, W, pairs, s_perm[warp], GL, warp, WARPS, &s_hit);
            }
        }
        __syncthreads();  // every warp is done with this pair (and with s_item)
        if (threadIdx.x == 0 && ro >= 0) {
            P.results[(size_t)pe.x * P.num_envs + pe.y] = s_hit ? 1 : 0;
            if (P.counters) {
                atomicAdd(P.counters + 0, 1ull);
                atomicAdd(P.counters + 5, s_hit ? 1ull : 0ull);
            }
        }
    }
}

// ------------------------------------------------------------------ learned order
// One MLP feature row: joints normalised to [-1, 1] by the joint limits, the
// environment code, zeros, and in column kMlpIn - 2 the sample's position
// along its edge (sample k of 32 n mapped to [-1, 1]: where on an edge whose
// start is free a collision lies is the strongest per-sample signal the
// walk order can use); column kMlpIn - 1 stays zero (the forward kernel's bias
// input).  BF16, kMlpIn values.
__device__ __forceinline__ float sample_position(int k, int n) {
    return 2.0f * (float)k / (float)(kLanes * n - 1) - 1.0f;
}

template <class M>
__device__ __forceinline__ void write_features(const float* q, const float* code, float pos, uint16_t* dst) {
    static_assert(M::dof + kEnvCode <= kMlpIn - 2, "feature row too narrow for this robot");
    const DevTables<M>& T = tab<M>();
    float f[kMlpIn];
#pragma unroll
    for (int j = 0; j < kMlpIn; ++j) f[j] = 0.0f;
#pragma unroll
    for (int j = 0; j < M::dof; ++j) f[j] = 2.0f * (q[j] - T.s_a[j]) / T.s_m[j] - 1.0f;
#pragma unroll
    for (int j = 0; j < kEnvCode; ++j) f[M::dof + j] = code[j];
    f[kMlpIn - 2] = pos;
    uint32_t w[kMlpIn / 2];
#pragma unroll
    for (int j = 0; j < kMlpIn / 2; ++j) {
        __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
        w[j] = *reinterpret_cast<uint32_t*>(&h);
    }
    uint4* d = reinterpret_cast<uint4*>(dst);
#pragma unroll
    for (int j = 0; j < kMlpIn / 8; ++j) d[j] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
}

// Features of every queued pair's segments: row ro + j is segment j scored at
// its last sample k = 8 j + 7, the first one the finish walk checks.  Eight
// lanes per queue entry (four entries per
// warp in flight, grid-strided), each lane one segment at a time: the loads
// of an entry form a dependent chain, so several entries per warp hide it.
constexpr int kFeatureLanes = 8;

template <class M>
__global__ void queue_features_kernel(CheckParams P, const float* __restrict__ edges, const float* __restrict__ code,
                                      uint16_t* __restrict__ x) {
    const int sl = threadIdx.x & (kFeatureLanes - 1);
    const long long queued = (long long)(*P.q_head >> 32);
    const int total = (int)min(queued, (long long)P.q_cap);
    const int per_cta = blockDim.x / kFeatureLanes;
    const int stride = gridDim.x * per_cta;
    for (int i = blockIdx.x * per_cta + threadIdx.x / kFeatureLanes; i < total; i += stride) {
        const int ro = P.q_rows[i];
        if (ro < 0) continue;
        const int2 pe = P.q_pairs[i];
        const int e = pe.x, env = pe.y;
        const int n = P.steps[e];
        float s[M::dof], t[M::dof], q[M::dof];
#pragma unroll
        for (int j = 0; j < M::dof; ++j) {
            s[j] = edges[(size_t)e * 2 * M::dof + j];
            t[j] = edges[(size_t)e * 2 * M::dof + M::dof + j];
        }
        for (int seg = sl; seg < 4 * n; seg += kFeatureLanes) {
            const int k = seg * kSegment + kSegment - 1;
            edge_sample<M::dof>(s, t, n, k, q);
            write_features<M>(q, code + (size_t)env * kEnvCode, sample_position(k, n), x + (size_t)(ro + seg) * kMlpIn);
        }
    }
}

// Inline learned order, features: row c * S + s (S = the check's segments,
// offs[E] / 8) is segment s of its edge scored at its last sample with the
// code of environment cluster c.  One thread per row.
template <class M>
__global__ void cluster_features_kernel(CheckParams P, const float* __restrict__ edges,
                                        const float* __restrict__ centroids, int K, uint16_t* __restrict__ x) {
    const long long S = P.total_segs;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S * K) return;
    const int c = (int)(i / S);
    const int sg = (int)(i - (long long)c * S);
    // the segment's edge: segments never straddle edges (offs[e] % 32 == 0);
    // binary search over the sample offsets (the FK table may not exist yet)
    const int row = sg * kSegment;
    int lo = 0, hi = P.num_edges - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (P.offs[mid] <= row) lo = mid; else hi = mid - 1;
    }
    const int e = lo;
    const int j = sg - P.offs[e] / kSegment;
    float s[M::dof], t[M::dof], q[M::dof];
#pragma unroll
    for (int d = 0; d < M::dof; ++d) {
        s[d] = edges[(size_t)e * 2 * M::dof + d];
        t[d] = edges[(size_t)e * 2 * M::dof + M::dof + d];
    }
    const int k = j * kSegment + kSegment - 1;
    edge_sample<M::dof>(s, t, P.steps[e], k, q);
    write_features<M>(q, centroids + (size_t)c * kEnvCode, sample_position(k, P.steps[e]), x + (size_t)i * kMlpIn);
}

// Inline learned order, one warp per (cluster c, edge e): perms[(c * E + e) *
// kMaxSegments + rank] = segment, segment 0 first (the scores tell where an edge
// with a free start collides), the others by descending score (row c * S +
// offs[e] / 8 + segment).  Edges of more segments keep the plain order.
template <class M>
__global__ void cluster_perm_kernel(CheckParams P, int K, uint8_t* __restrict__ perms) {
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int E = P.num_edges;
    if (warp >= (long long)K * E) return;
    const int c = (int)(warp / E);
    const int e = (int)(warp - (long long)c * E);
    const int nseg = 4 * P.steps[e];
    if (nseg > kMaxSegments) return;
    rank_segments(P.logits + (size_t)c * P.total_segs + P.offs[e] / kSegment, nseg,
                  perms + (size_t)warp * kMaxSegments, true);
}

// Training rows: row i draws (environment, edge, sample) from a hash of
// (seed, i); features as above at that sample; label = the sample's
// environment collision with the reference's gate semantics (bound against
// every primitive, then the leaves against every primitive).
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Environment verdict of one sample-table row against environment env, one
// thread: each link group's bound against every primitive and, once some
// primitive hits it, the group's leaves against every primitive -- the
// reference's gate semantics (fkcc, src/utils.cuh:806-1190).  Self-collision
// is not part of it (env-independent, decided per edge before any walk).
template <class M>
__device__ __forceinline__ bool sample_hits_env(const CheckParams& P, int env, size_t row) {
    constexpr int G = M::num_env_groups;
    const float4 hd0 = P.env_hdr[2 * env], hd1 = P.env_hdr[2 * env + 1];
    const float4* rec = P.blobs + __float_as_uint(hd0.w);
    const int np = (int)(__float_as_uint(hd1.w) & 0xffffu);
    const float4* r = P.table + table_index<M>(row, 0);
    const DevTables<M>& T = tab<M>();
    for (int g = 0; g < G; ++g) {
        float4 b = r[g];
        b.w += kEnvInflate;
        bool gate = false;
        for (int p = 0; p < np && !gate; ++p) gate = sphere_hits_prim(b, rec + p * kPrimF4);
        if (!gate) continue;
        for (int li = T.leaf_begin[g]; li < T.leaf_begin[g + 1]; ++li) {
            float4 l = r[G + li];
            l.w += kEnvInflate;
            for (int p = 0; p < np; ++p)
                if (sphere_hits_prim(l, rec + p * kPrimF4)) return true;
        }
    }
    return false;
}

// Learned-order population: the environment verdict of every sample of every
// queued pair (one warp per queue entry, lanes over the 32 n samples):
// lab[8 ro + k] for sample k of the entry whose first MLP row is ro, and
// y[ro + j] = the verdict at segment j's scored sample 8 j + 7.
template <class M>
__global__ void queue_labels_kernel(CheckParams P, uint8_t* __restrict__ lab, uint8_t* __restrict__ y) {
    const int lane = threadIdx.x & 31;
    const long long queued = (long long)(*P.q_head >> 32);
    const int total = (int)min(queued, (long long)P.q_cap);
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < total; i += warps) {
        const int ro = P.q_rows[i];
        if (ro < 0) continue;
        const int2 pe = P.q_pairs[i];
        const int n = P.steps[pe.x];
        const size_t row0 = (size_t)P.offs[pe.x];
        for (int k = lane; k < kLanes * n; k += 32) {
            const uint8_t h = sample_hits_env<M>(P, pe.y, row0 + (size_t)k) ? 1 : 0;
            lab[(size_t)ro * kSegment + k] = h;
            if ((k & (kSegment - 1)) == kSegment - 1) y[ro + k / kSegment] = h;
        }
    }
}

template <class M>
__global__ void training_rows_kernel(CheckParams P, const float* __restrict__ edges, const float* __restrict__ code,
                                     long long rows, unsigned long long seed, uint16_t* __restrict__ x,
                                     uint8_t* __restrict__ y) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows) return;
    const unsigned long long h1 = mix64(seed ^ (unsigned long long)i), h2 = mix64(h1), h3 = mix64(h2);
    const int env = (int)(h1 % (unsigned long long)P.num_envs);
    const int e = (int)(h2 % (unsigned long long)P.num_edges);
    const int n = P.steps[e];
    const int k = (int)(h3 % (unsigned long long)(kLanes * n));
    float s[M::dof], t[M::dof], q[M::dof];
#pragma unroll
    for (int j = 0; j < M::dof; ++j) {
        s[j] = edges[(size_t)e * 2 * M::dof + j];
        t[j] = edges[(size_t)e * 2 * M::dof + M::dof + j];
    }
    edge_sample<M::dof>(s, t, n, k, q);
    write_features<M>(q, code + (size_t)env * kEnvCode, sample_position(k, n), x + (size_t)i * kMlpIn);
    y[i] = sample_hits_env<M>(P, env, (size_t)P.offs[e] + k) ? 1 : 0;
}

// ------------------------------------------------------------------ records variant
// regular_rec (bcc_api.cu) of a record on the device.
__device__ __forceinline__ bool regular_prim(const float4* rec) {
    const float4 c = rec[0], a1 = rec[1], a2 = rec[2], a3 = rec[3];
    auto zero = [](float4 v) { return 0.0f * v.x + 0.0f * v.y + (0.0f * v.z + 0.0f * v.w); };  // unless not finite
    auto dot = [](float4 u, float4 v) { return fmaf(u.x, v.x, fmaf(u.y, v.y, u.z * v.z)); };
    const float xy = fabsf(dot(a1, a2)), xz = fabsf(dot(a1, a3)), yz = fabsf(dot(a2, a3));
    return zero(c) + zero(a1) + (zero(a2) + zero(a3)) == 0.0f && c.w >= 0.0f &&
           fabsf(dot(a1, a1) - 1.0f) + xy + xz <= kAxesTol && fabsf(dot(a2, a2) - 1.0f) + xy + yz <= kAxesTol &&
           fabsf(dot(a3, a3) - 1.0f) + xz + yz <= kAxesTol;
}

// Environment check from the host-packed rounded-box records of bcc_pack_envs
// (no interval-mask tables), used by the allocation-free entry point: culls
// (primitive, link) pairs with an exact AABB overlap test, one primitive per
// lane; the walk over (sample, pair) items is check_kernel's.
template <class M, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) check_records_kernel(RecordsParams P) {
    constexpr int G = M::num_env_groups;
    constexpr int GB = group_bits<M>();
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t bar;
    __shared__ float4 boxes[WARPS][G][2];

    if (P.offs[P.num_edges] > P.cap_rows) return;
    const int env = blockIdx.x;
    const int e_begin = blockIdx.y * P.edges_per_cta;
    const int e_end = min(e_begin + P.edges_per_cta, P.num_edges);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p_begin = P.env_off[env];
    const int np = P.env_off[env + 1] - p_begin;

    const float4* prim = reinterpret_cast<const float4*>(smem);
    uint16_t* pairs = reinterpret_cast<uint16_t*>(smem + (size_t)P.max_prims * kPrimF4 * 16) +
                      (size_t)warp * P.pairs_per_warp;
    if (np < 0 || np > P.max_prims) {  // shared memory was sized from the caller's max_prims
        if (threadIdx.x == 0) atomicOr(P.error_flag, 2);
        return;
    }
    if (np > 0) {
        if (threadIdx.x == 0) {
            mbar_init(&bar, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
        if (threadIdx.x == 0)
            bulk_copy_g2s(smem, P.records + (size_t)p_begin * kPrimF4, (uint32_t)np * kPrimF4 * 16u, &bar);
        // One path for the whole CTA (see check_kernel).
        const bool ok = mbar_wait_bounded(&bar, 0u, 1u << 22);
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) atomicOr(P.error_flag, 1);
            mbar_wait_bounded(&bar, 0u, 1u << 22);
            return;
        }
    }
    // Whether the environment is irregular is not in the records: found here.
    bool odd = false;
    for (int p = threadIdx.x; p < np; p += WARPS * 32) odd |= !regular_prim(prim + p * kPrimF4);
    const bool exact = __syncthreads_or(odd) != 0;
    const uint32_t lt = (1u << lane) - 1u;
    const GroupLanes GL = group_lanes<M>();

    for (int e = e_begin + warp; e < e_end; e += WARPS) {
        uint8_t* out = P.results + (size_t)e * P.num_envs + env;
        const int self = P.edge_self[e];
        if (np == 0 || self) {
            if (lane == 0) *out = self ? 1 : 0;
            continue;
        }
        if (exact) {
            const bool hit = walk_exact<M>(P.table, (size_t)P.offs[e], P.steps[e], prim, np);
            if (lane == 0) *out = hit ? 1 : 0;
            continue;
        }
        if (lane < G) {
            boxes[warp][lane][0] = P.swept[((size_t)e * G + lane) * 2 + 0];
            boxes[warp][lane][1] = P.swept[((size_t)e * G + lane) * 2 + 1];
        }
        __syncwarp();
        // Exact AABB cull, one primitive per lane; pairs compacted link-major
        // within each block of 32 primitives.
        int C = 0;
        for (int p0 = 0; p0 < np; p0 += 32) {
            const int p = p0 + lane;
            uint32_t mask = 0;
            if (p < np) {
                const float4 c = prim[p * kPrimF4 + 0];
                const float4 h = prim[p * kPrimF4 + 4];
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const float4 lo = boxes[warp][g][0], hi = boxes[warp][g][1];
                    const bool ov = c.x - h.x <= hi.x && c.x + h.x >= lo.x && c.y - h.y <= hi.y &&
                                    c.y + h.y >= lo.y && c.z - h.z <= hi.z && c.z + h.z >= lo.z;
                    mask |= (uint32_t)ov << g;
                }
            }
#pragma unroll 1
            for (int g = 0; g < G; ++g) {
                const uint32_t bits = __ballot_sync(kFull, (mask >> g) & 1u);
                if ((mask >> g) & 1u) pairs[C + __popc(bits & lt)] = (uint16_t)((p << GB) | g);
                C += __popc(bits);
            }
        }
        __syncwarp();

        bool collide = false;
        WalkStats st;
        if (C > 0)
            collide = walk_segments<M>(P.table, P.seg, (size_t)P.offs[e], P.steps[e], C, pairs, prim, np, nullptr, GL,
                                       warp_scratch(), st);
        __syncwarp();
        if (lane == 0) *out = collide ? 1 : 0;
    }
}

// ------------------------------------------------------------------ launchers
template <class M>
cudaError_t run_steps(const PipelineArgs& a, cudaStream_t st) {
    const int E = a.num_edges;
    if (a.stage_events) cudaEventRecord(a.stage_events[0], st);
    if (E <= kFusedSteps) {
        edge_offsets_kernel<M><<<1, kFusedSteps, 0, st>>>(a.d_edges, E, a.resolution, a.steps, a.offs,
                                                                a.host_total);
        return cudaGetLastError();
    }
    edge_steps_kernel<M><<<(E + 255) / 256, 256, 0, st>>>(a.d_edges, E, a.resolution, a.steps);
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    return launch_scan(a.steps, E, a.offs, a.host_total, st);
}

// Probe and walk, in slabs of environments whose pairs fit the queue.
template <class M, int W, int MODE>
cudaError_t launch_probed(const CheckParams& P, int E, cudaStream_t st) {
    const size_t smem = P.blob_smem + P.probe.stride + P.queue.batch * kProbeEntryBytes;
    const size_t walk_smem = check_smem_bytes(P.max_prims, M::num_env_groups, P.blob_smem, W);
    cudaError_t err = cudaFuncSetAttribute(probe_kernel<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    err = cudaFuncSetAttribute(walk_kernel<M, W, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)walk_smem);
    if (err != cudaSuccess) return err;
    int per_sm = 0, dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, walk_kernel<M, W, MODE>, W * 32, walk_smem);
    if (err != cudaSuccess) return err;
    const int slots = std::max(per_sm, 1) * std::max(sms, 1);
    ProbeQueue Q = P.queue;
    const int slab = (int)std::min<long long>(P.num_envs, Q.cap / E);
    err = cudaMemsetAsync(Q.head, 0, (size_t)((P.num_envs + slab - 1) / slab) * 16, st);
    if (err != cudaSuccess) return err;
    for (int env0 = 0; env0 < P.num_envs; env0 += slab, Q.head += 4) {
        const int n = std::min(slab, P.num_envs - env0);
        probe_kernel<M><<<dim3(n, (E + Q.batch - 1) / Q.batch), kProbeThreads, smem, st>>>(P, Q, env0);
        const long long most = (long long)n * E;  // every pair undecided
        const int grid = (int)std::min<long long>(slots, (most + Q.chunk - 1) / Q.chunk);
        walk_kernel<M, W, MODE><<<grid, W * 32, walk_smem, st>>>(P, Q);
    }
    return cudaGetLastError();
}

template <class M, int W, int MODE>
cudaError_t launch_check_wm(CheckParams P, int E, cudaStream_t st) {
    P.pairs_per_warp = std::min((P.max_prims * M::num_env_groups + 7) & ~7, kPairCap);
    const size_t smem = check_smem_bytes(P.max_prims, M::num_env_groups, P.blob_smem, W);
    if constexpr (MODE != 1)
        if (P.probe.vox) return launch_probed<M, W, MODE>(P, E, st);
    cudaError_t err = cudaFuncSetAttribute(check_kernel<M, W, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem);
    if (err != cudaSuccess) return err;
    dim3 grid(P.num_envs, (E + P.edges_per_cta - 1) / P.edges_per_cta);
    check_kernel<M, W, MODE><<<grid, W * 32, smem, st>>>(P);
    return cudaGetLastError();
}

// Learned order, phase 3: a grid of the resident capacity; the queue length
// is read on the device.
template <class M, int W>
cudaError_t launch_finish_w(CheckParams P, cudaStream_t st) {
    P.pairs_per_warp = std::min((P.max_prims * M::num_env_groups + 7) & ~7, kPairCap);
    const size_t smem = (size_t)W * P.pairs_per_warp * sizeof(uint16_t);
    auto kern = P.finish_split ? finish_kernel<M, W> : finish_warp_kernel<M, W>;
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    int per_sm = 0, dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, W * 32, smem);
    if (err != cudaSuccess) return err;
    err = cudaMemsetAsync(P.finish_counter, 0, sizeof(int), st);
    if (err != cudaSuccess) return err;
    kern<<<std::max(per_sm, 1) * std::max(sms, 1), W * 32, smem, st>>>(P);
    return cudaGetLastError();
}

template <class M, int W>
cudaError_t launch_check_w(CheckParams P, int E, cudaStream_t st, int mode) {
    switch (mode) {
        case 1: return launch_check_wm<M, W, 1>(P, E, st);
        case 2: return launch_finish_w<M, W>(P, st);
        case 4: return launch_check_wm<M, W, 4>(P, E, st);
        default: return launch_check_wm<M, W, 0>(P, E, st);
    }
}

template <class M>
cudaError_t check_by_warps(const CheckParams& P, int E, int warps, int mode, cudaStream_t st) {
    switch (warps) {
        case 8: return launch_check_w<M, 8>(P, E, st, mode);
        case 4: return launch_check_w<M, 4>(P, E, st, mode);
        case 2: return launch_check_w<M, 2>(P, E, st, mode);
        case 1: return launch_check_w<M, 1>(P, E, st, mode);
        default: return cudaErrorInvalidValue;
    }
}

// FK table, self-collision and swept volumes (no environment check); records
// stage events 1-4 when profiling.
template <class M>
cudaError_t run_prep(const PipelineArgs& a, cudaStream_t st) {
    const int E = a.num_edges;
    const int R = a.total_rows >= 0 ? a.total_rows : a.cap_rows;  // at most: the kernels read the total
    cudaEvent_t* ev = a.stage_events;
    if (ev) cudaEventRecord(ev[1], st);
    cudaError_t err = cudaMemsetAsync(a.edge_self, 0, sizeof(int) * E, st);
    if (err != cudaSuccess) return err;
    if (R > 0) {
        // FK and self-collision in one kernel; a grid of the resident CTAs strides
        // over the 32-row blocks
        const size_t smem = 32 * (size_t)(M::num_spheres | 1) * sizeof(float4);
        err = cudaFuncSetAttribute(fk_staged_kernel<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err != cudaSuccess) return err;
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fk_staged_kernel<M>, 32 * fk_warps<M>(), smem);
        if (err != cudaSuccess) return err;
        const int blocks = (R + 31) / 32;
        const int grid = std::min(blocks, std::max(per_sm, 1) * std::max(sms, 1));
        fk_staged_kernel<M><<<grid, 32 * fk_warps<M>(), smem, st>>>(a.d_edges, E, a.steps, a.offs, a.cap_rows, a.table,
                                                                    a.edge_self, a.seg);
    }
    if (ev) cudaEventRecord(ev[2], st);
    if (ev) cudaEventRecord(ev[3], st);
    swept_kernel<M><<<(E * 32 + 255) / 256, 256, 0, st>>>(a.table, a.offs, E, a.cap_rows, a.swept,
                                                           a.grid_bounds ? a.edge_tri : nullptr, a.grid_bounds, a.mid);
    if (ev) cudaEventRecord(ev[4], st);
    return cudaGetLastError();
}

// Environment check only (the FK/self/swept stages already ran), in a.mode.
template <class M>
cudaError_t run_check_mode(const PipelineArgs& a, cudaStream_t st) {
    const CheckParams P = params_of(a);
    if (P.num_irregular > 0 && a.mode != 2) {  // (the finish pass has none of their pairs)
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const long long ctas = ((long long)P.num_irregular * P.num_edges + kExactWarps - 1) / kExactWarps;
        exact_kernel<M><<<(unsigned)std::min<long long>(ctas, 16 * std::max(sms, 1)), 32 * kExactWarps, 0, st>>>(P);
        const cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) return err;
    }
    return check_by_warps<M>(P, a.num_edges, a.warps, a.mode, st);
}

template <class M>
cudaError_t run_check(const PipelineArgs& a, cudaStream_t st) {
    cudaError_t err = run_prep<M>(a, st);
    if (err != cudaSuccess) return err;
    err = run_check_mode<M>(a, st);
    if (a.stage_events) cudaEventRecord(a.stage_events[5], st);
    return err;
}

template <class M>
cudaError_t run_queue_features(const PipelineArgs& a, const float* env_code, uint16_t* x, int grid,
                               cudaStream_t st) {
    if (grid <= 0) return cudaSuccess;
    queue_features_kernel<M><<<grid, 128, 0, st>>>(params_of(a), a.d_edges, env_code, x);
    return cudaGetLastError();
}

template <class M>
cudaError_t run_cluster_order_inputs(const PipelineArgs& a, const float* centroids, int K, uint16_t* x,
                                     cudaStream_t st) {
    const long long rows = (long long)K * a.total_segs;
    if (rows <= 0) return cudaSuccess;
    cluster_features_kernel<M><<<(unsigned)((rows + 127) / 128), 128, 0, st>>>(params_of(a), a.d_edges, centroids, K,
                                                                               x);
    return cudaGetLastError();
}

template <class M>
cudaError_t run_cluster_perms(const PipelineArgs& a, int K, uint8_t* perms, cudaStream_t st) {
    const long long warps = (long long)K * a.num_edges;
    if (warps <= 0) return cudaSuccess;
    cluster_perm_kernel<M><<<(unsigned)((warps * 32 + 255) / 256), 256, 0, st>>>(params_of(a), K, perms);
    return cudaGetLastError();
}

template <class M>
cudaError_t run_training_rows(const PipelineArgs& a, const float* env_code, long long rows, unsigned long long seed,
                              uint16_t* x, uint8_t* y, cudaStream_t st) {
    if (rows <= 0) return cudaSuccess;
    training_rows_kernel<M><<<(unsigned)((rows + 127) / 128), 128, 0, st>>>(params_of(a), a.d_edges, env_code, rows,
                                                                           seed, x, y);
    return cudaGetLastError();
}

template <class M>
cudaError_t run_queue_labels(const PipelineArgs& a, uint8_t* lab, uint8_t* y, int grid, cudaStream_t st) {
    if (grid <= 0) return cudaSuccess;
    queue_labels_kernel<M><<<grid, 256, 0, st>>>(params_of(a), lab, y);
    return cudaGetLastError();
}

template <class M>
cudaError_t run_check_records(RecordsParams P, cudaStream_t st) {
    constexpr int W = kRecordsWarps;
    if (P.max_prims > max_prims_of<M>()) return cudaErrorInvalidValue;
    P.pairs_per_warp = (P.max_prims * M::num_env_groups + 7) & ~7;
    const size_t smem = records_smem_bytes(P.max_prims, M::num_env_groups, W);
    cudaError_t err = cudaFuncSetAttribute(check_records_kernel<M, W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem);
    if (err != cudaSuccess) return err;
    dim3 grid(P.num_envs, (P.num_edges + P.edges_per_cta - 1) / P.edges_per_cta);
    check_records_kernel<M, W><<<grid, W * 32, smem, st>>>(P);
    return cudaGetLastError();
}

// The robot's entry points, as the robot-independent code calls them.
template <class M>
RobotOps robot_ops_of(int robot, cudaError_t (*upload)()) {
    RobotOps o;
    o.robot = robot;
    o.dof = M::dof;
    o.num_spheres = M::num_spheres;
    o.num_env_groups = M::num_env_groups;
    o.max_prims = max_prims_of<M>();
    o.reach_lo = M::reach_lo;
    o.reach_hi = M::reach_hi;
    o.upload_tables = upload;
    o.steps = run_steps<M>;
    o.check = run_check<M>;
    o.prep = run_prep<M>;
    o.check_mode = run_check_mode<M>;
    o.queue_features = run_queue_features<M>;
    o.training_rows = run_training_rows<M>;
    o.queue_labels = run_queue_labels<M>;
    o.cluster_features = run_cluster_order_inputs<M>;
    o.cluster_perms = run_cluster_perms<M>;
    o.check_records = run_check_records<M>;
    return o;
}

}  // namespace bcc
