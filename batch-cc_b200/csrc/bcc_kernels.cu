// bcc_kernels.cu -- robot-independent kernels of the batch edge collision
// checker (sm_100a): the environment arena, the sample-offset scan, the environment code of the
// learned check order, shared-memory sizing, and the robot registry.  The
// robot-templated pipeline lives in bcc_pipeline.cuh and is instantiated once
// per robot in bcc_robot_<name>.cu.
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "bcc_device.cuh"
#include "bcc_kernels.h"
#include "bcc_mlp.h"

namespace bcc {

extern const RobotOps kPandaOps;
extern const RobotOps kFetchOps;
extern const RobotOps kBaxterOps;

const RobotOps* robot_ops(int robot) {
    switch (robot) {
        case 0: return &kPandaOps;
        case 1: return &kFetchOps;
        case 2: return &kBaxterOps;
        default: return nullptr;
    }
}

// ------------------------------------------------------------------ scan
// Single-CTA exclusive scan of 32*steps[e] into offs[e], offs[E] = total, four
// consecutive edges a thread (50 000 edges: 13 rounds of loads and barriers
// instead of 49).  Sums run in 64 bits and every offset saturates at INT32_MAX, so
// a total too large for the sample table can never wrap into a small,
// valid-looking one; the host rejects any total above its limit.
__global__ void __launch_bounds__(1024) scan_kernel(const int* __restrict__ steps, int E, int* __restrict__ offs,
                                                    int* __restrict__ host_total) {
    __shared__ long long warp_sums[32];
    long long carry = 0;
    for (int base = 0; base < E; base += 4096) {
        const int i = base + 4 * threadIdx.x;
        long long v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = i + k < E ? (long long)kLanes * steps[i + k] : 0;
        const long long sum = v[0] + v[1] + v[2] + v[3];
        long long all;
        long long at = carry + block_scan_exclusive(sum, warp_sums, all);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (i + k < E) offs[i + k] = (int)min(at, 2147483647ll);
            at += v[k];
        }
        carry += all;
    }
    if (threadIdx.x == 0) {
        offs[E] = (int)min(carry, 2147483647ll);
        if (host_total) *host_total = (int)min(carry, 2147483647ll);
    }
}

cudaError_t launch_scan(const int* steps, int E, int* offs, int* host_total, cudaStream_t st) {
    scan_kernel<<<1, 1024, 0, st>>>(steps, E, offs, host_total);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ sizing
// Dynamic shared memory of a check CTA: the largest environment's records plus,
// per warp, a (primitive, link) pair list of max_prims x groups entries, at
// most kPairCap.
size_t check_smem_bytes(int max_prims, int groups, size_t blob_smem, int warps) {
    const size_t ppw = (size_t)std::min((max_prims * groups + 7) & ~7, kPairCap);
    return blob_smem + (size_t)warps * ppw * sizeof(uint16_t);
}

size_t records_smem_bytes(int max_prims, int groups, int warps) {
    const size_t ppw = (size_t)((max_prims * groups + 7) & ~7);
    return (size_t)max_prims * kPrimF4 * 16 + (size_t)warps * ppw * sizeof(uint16_t);
}

// ------------------------------------------------------------------ arena
// Largest slab s in [0, kGridSlabs) whose lower boundary is <= x (0 below the
// first); b increases.
__device__ __forceinline__ int slab_below(const float* b, double x) {
    int s = 0;
#pragma unroll
    for (int step = kGridSlabs / 2; step; step >>= 1)
        if ((double)b[s + step] <= x) s += step;
    return s;
}

// One CTA per environment: its records into the blob, then one warp per (axis,
// 64-primitive word) of the mask tables.  A primitive meets slabs [s0, s1] (its
// AABB widened by 1e-5 m, in FP64, so that the FP32 swept boxes can only
// over-include) and slab range [i0, i1] meets it when s0 <= i1 and s1 >= i0: the
// range's mask is A[i1] & B[i0] with A[i] the primitives that start at or below
// slab i and B[i] those that end at or above it.  Lane i holds A[i] and B[i]
// (ballots over the word's primitives), row i0 of the triangle is one shuffle,
// an AND and a coalesced store.  Bound by the table's stores (12.7 KB per 64
// primitives); built on the host it cost 528 tests a primitive and axis, 16 of
// the 21 ms of an upload and check of 211 environments x 997 edges.
constexpr int kArenaThreads = 128;

__global__ void __launch_bounds__(kArenaThreads) build_arena_kernel(const float4* __restrict__ records,
                                                                    const float4* __restrict__ hdr,
                                                                    const float* __restrict__ bounds,
                                                                    float4* __restrict__ blobs) {
    static_assert(kGridSlabs == 32, "lane i holds slab i's masks");
    __shared__ float b[3 * (kGridSlabs + 1)];
    const float4 h0 = hdr[2 * blockIdx.x], h1 = hdr[2 * blockIdx.x + 1];
    const uint32_t shape = __float_as_uint(h1.w);
    const int np = (int)(shape & 0xffffu), W = (int)(shape >> 16);
    const float4* src = records + (size_t)__float_as_uint(h1.x) * kPrimF4;
    float4* dst = blobs + (size_t)__float_as_uint(h0.w);
    for (int i = threadIdx.x; i < 3 * (kGridSlabs + 1); i += kArenaThreads) b[i] = bounds[i];
    for (int i = threadIdx.x; i < np * kPrimF4; i += kArenaThreads) dst[i] = src[i];
    __syncthreads();
    uint64_t* masks = reinterpret_cast<uint64_t*>(dst + (size_t)np * kPrimF4);
    const int lane = threadIdx.x & 31;
    for (int t = threadIdx.x >> 5; t < 3 * W; t += kArenaThreads / 32) {
        const int a = t / W, w = t - a * W;
        const float* ba = b + a * (kGridSlabs + 1);
        int s0[2], s1[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int p = w * 64 + k * 32 + lane;
            s0[k] = kGridSlabs;  // past the last primitive: in no slab
            s1[k] = -1;
            if (p < np) {
                const float* r = reinterpret_cast<const float*>(src + (size_t)p * kPrimF4);
                const double c = (double)r[a], h = (double)r[16 + a];
                s0[k] = slab_below(ba, __dsub_rn(__dsub_rn(c, h), 1e-5));
                s1[k] = slab_below(ba, __dadd_rn(__dadd_rn(c, h), 1e-5));
            }
        }
        uint64_t A = 0, B = 0;
        for (int i = 0; i < kGridSlabs; ++i) {
            const uint64_t x = __ballot_sync(0xffffffffu, s0[0] <= i) |
                               ((uint64_t)__ballot_sync(0xffffffffu, s0[1] <= i) << 32);
            const uint64_t y = __ballot_sync(0xffffffffu, s1[0] >= i) |
                               ((uint64_t)__ballot_sync(0xffffffffu, s1[1] >= i) << 32);
            if (lane == i) {
                A = x;
                B = y;
            }
        }
        for (int i0 = 0; i0 < kGridSlabs; ++i0) {
            const uint64_t m = A & __shfl_sync(0xffffffffu, B, i0);
            if (lane >= i0) masks[(size_t)(a * kGridTri + tri_index(i0, lane)) * W + w] = m;
        }
    }
}

cudaError_t launch_build_arena(const float4* records, const float4* env_hdr, const float* bounds, int num_envs,
                               float4* blobs, cudaStream_t st) {
    if (num_envs <= 0) return cudaSuccess;
    build_arena_kernel<<<(unsigned)num_envs, kArenaThreads, 0, st>>>(records, env_hdr, bounds, blobs);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ probe grid
// Per voxel the signed distance of its centre to every primitive (outside: to the
// rounded box; inside: minus the depth), the nearest one and its quantised distance.
// One warp per brick of 4 x 4 x 2 voxels.  Distances are 1-Lipschitz (where they are
// not, kEnvIrregular, the grid is not read): lanes over the primitives, those within
// twice the brick's radius of the nearest one to its centre can be nearest to a
// voxel, and only they are tested by the lanes as voxels.
// Bound by FP32 issue, ~35 instructions a test, the record read as a shared-memory
// broadcast: 0.37 ms for 1000 environments of 8 .. 64 primitives, 0.53 for 500 of 16 .. 256,
// against 0.76 and 1.48 for every voxel against every primitive.
constexpr int kGridThreads = 256;
constexpr int kGridChunk = 128;  // records staged at a time
constexpr int kBrickX = 4, kBrickY = 4, kBrickZ = 2;
static_assert(kBrickX * kBrickY * kBrickZ == 32, "a lane a voxel");

__device__ __forceinline__ float prim_signed_dist(const float4* rec, float x, float y, float z) {
    const float4 w0 = rec[0], w1 = rec[1], w2 = rec[2], w3 = rec[3];
    const float dx = x - w0.x, dy = y - w0.y, dz = z - w0.z;
    const float p1 = fabsf(fmaf(w1.x, dx, fmaf(w1.y, dy, w1.z * dz))) - w1.w;
    const float p2 = fabsf(fmaf(w2.x, dx, fmaf(w2.y, dy, w2.z * dz))) - w2.w;
    const float p3 = fabsf(fmaf(w3.x, dx, fmaf(w3.y, dy, w3.z * dz))) - w3.w;
    const float e1 = fmaxf(p1, 0.0f), e2 = fmaxf(p2, 0.0f), e3 = fmaxf(p3, 0.0f);
    const float in = fminf(fmaxf(p1, fmaxf(p2, p3)), 0.0f);
    return sqrtf(fmaf(e1, e1, fmaf(e2, e2, e3 * e3))) + in - w0.w;
}

__device__ __host__ __forceinline__ int grid_bricks(const ProbeGrid& p) {
    return (p.nx + kBrickX - 1) / kBrickX * ((p.ny + kBrickY - 1) / kBrickY) * ((p.nz + kBrickZ - 1) / kBrickZ);
}

__global__ void __launch_bounds__(kGridThreads) probe_grid_kernel(const float4* __restrict__ blobs,
                                                                  const float4* __restrict__ hdr, ProbeGrid p,
                                                                  uint16_t* __restrict__ vox) {
    __shared__ float4 rec[kGridChunk * 4];
    constexpr int kSteps = kGridChunk / 32;
    const int env = blockIdx.x, lane = threadIdx.x & 31;
    const int brick = blockIdx.y * (kGridThreads / 32) + (threadIdx.x >> 5);
    const float4 h0 = hdr[2 * env], h1 = hdr[2 * env + 1];
    const float4* src = blobs + __float_as_uint(h0.w);
    const int np = (int)(__float_as_uint(h1.w) & 0xffffu);
    const int bx = (p.nx + kBrickX - 1) / kBrickX, by = (p.ny + kBrickY - 1) / kBrickY;
    const int x0 = brick % bx * kBrickX, y0 = brick / bx % by * kBrickY, z0 = brick / (bx * by) * kBrickZ;
    const int ix = x0 + lane % kBrickX, iy = y0 + lane / kBrickX % kBrickY, iz = z0 + lane / (kBrickX * kBrickY);
    const float x = fmaf((float)ix, p.h, p.ox), y = fmaf((float)iy, p.h, p.oy), z = fmaf((float)iz, p.h, p.oz);
    const float cx = fmaf((float)x0 + 0.5f * (kBrickX - 1), p.h, p.ox);
    const float cy = fmaf((float)y0 + 0.5f * (kBrickY - 1), p.h, p.oy);
    const float cz = fmaf((float)z0 + 0.5f * (kBrickZ - 1), p.h, p.oz);
    // twice half a brick's diagonal, from voxel centre to voxel centre
    const float span = p.h * sqrtf((kBrickX - 1) * (kBrickX - 1) + (kBrickY - 1) * (kBrickY - 1) +
                                   (kBrickZ - 1) * (kBrickZ - 1));
    float best = INFINITY, near = INFINITY;
    unsigned id = 0u;
    for (int p0 = 0; p0 < np; p0 += kGridChunk) {
        const int m = min(kGridChunk, np - p0);
        __syncthreads();
        for (int i = threadIdx.x; i < m * 4; i += kGridThreads) rec[i] = src[(size_t)(p0 + i / 4) * kPrimF4 + (i & 3)];
        __syncthreads();
        float d[kSteps];
#pragma unroll
        for (int s = 0; s < kSteps; ++s) {
            d[s] = INFINITY;
            if (32 * s + lane < m) d[s] = prim_signed_dist(rec + 4 * (32 * s + lane), cx, cy, cz);
            near = fminf(near, d[s]);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) near = fminf(near, __shfl_xor_sync(0xffffffffu, near, o));
        // (a margin over FP32 rounding of the distances)
        const float reach = near + span + 1e-4f + 1e-5f * fabsf(near);
#pragma unroll
        for (int s = 0; s < kSteps; ++s) {
            unsigned todo = __ballot_sync(0xffffffffu, 32 * s + lane < m && d[s] <= reach);
            for (; todo; todo &= todo - 1u) {
                const int k = 32 * s + __ffs(todo) - 1;
                const float v = prim_signed_dist(rec + 4 * k, x, y, z);
                if (v < best) {
                    best = v;
                    id = (unsigned)(p0 + k);
                }
            }
        }
    }
    if (ix >= p.nx || iy >= p.ny || iz >= p.nz) return;
    const float q = (best - kVoxMin) * (1.0f / kVoxStep);
    const unsigned code = (unsigned)(int)fminf(fmaxf(floorf(q), 0.0f), 255.0f);
    vox[(size_t)env * (p.stride / 2) + ((size_t)iz * p.ny + iy) * p.nx + ix] =
        (uint16_t)(min(id, kVoxUnknown) << 8 | code);
}

cudaError_t launch_probe_grid(const float4* blobs, const float4* env_hdr, int num_envs, const ProbeGrid& p,
                              uint16_t* vox, cudaStream_t st) {
    if (num_envs <= 0) return cudaSuccess;
    const dim3 grid((unsigned)num_envs, (unsigned)((grid_bricks(p) + kGridThreads / 32 - 1) / (kGridThreads / 32)));
    probe_grid_kernel<<<grid, kGridThreads, 0, st>>>(blobs, env_hdr, p, vox);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ environment code
// 32-value environment code (one warp per environment): [0..3] counts of
// sphere-like, capsule-like and box-like primitives and the total, / 64;
// [4..27] for 8 fixed anchor points the distance from the anchor to the
// nearest primitive of each of the three kinds (clamped to [-0.5, 1.5] m);
// [28..31] mean primitive centre xyz and mean extent.
__device__ __forceinline__ float prim_point_dist(const float4* rec, float x, float y, float z) {
    const float4 w0 = rec[0], w1 = rec[1], w2 = rec[2], w3 = rec[3];
    const float dx = x - w0.x, dy = y - w0.y, dz = z - w0.z;
    const float e1 = fmaxf(fabsf(w1.x * dx + w1.y * dy + w1.z * dz) - w1.w, 0.0f);
    const float e2 = fmaxf(fabsf(w2.x * dx + w2.y * dy + w2.z * dz) - w2.w, 0.0f);
    const float e3 = fmaxf(fabsf(w3.x * dx + w3.y * dy + w3.z * dz) - w3.w, 0.0f);
    return sqrtf(e1 * e1 + e2 * e2 + e3 * e3) - w0.w;
}

__global__ void env_encode_kernel(const float4* __restrict__ blobs, const float4* __restrict__ hdr, int N,
                                  float* __restrict__ code) {
    const int env = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (env >= N) return;
    const float4 h0 = hdr[2 * env], h1 = hdr[2 * env + 1];
    const float4* rec = blobs + __float_as_uint(h0.w);
    const int np = (int)(__float_as_uint(h1.w) & 0xffffu);
    float cnt[3] = {0, 0, 0}, best[8][3], mean[4] = {0, 0, 0, 0};
#pragma unroll
    for (int a = 0; a < 8; ++a) best[a][0] = best[a][1] = best[a][2] = 1.5f;
    for (int p = lane; p < np; p += 32) {
        const float4* r = rec + p * kPrimF4;
        const float4 w0 = r[0];
        const float hsum = r[1].w + r[2].w + r[3].w;
        const int kind = w0.w > 0.0f ? (hsum > 0.0f ? 1 : 0) : 2;  // sphere, capsule, box
        cnt[kind] += 1.0f;
        mean[0] += w0.x;
        mean[1] += w0.y;
        mean[2] += w0.z;
        mean[3] += w0.w + hsum;
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const float ax = (a & 1) ? 0.35f : -0.35f, ay = (a & 2) ? 0.35f : -0.35f, az = (a & 4) ? 0.8f : 0.3f;
            best[a][kind] = fminf(best[a][kind], prim_point_dist(r, ax, ay, az));
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
#pragma unroll
        for (int k = 0; k < 3; ++k) cnt[k] += __shfl_xor_sync(0xffffffffu, cnt[k], o);
#pragma unroll
        for (int k = 0; k < 4; ++k) mean[k] += __shfl_xor_sync(0xffffffffu, mean[k], o);
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int k = 0; k < 3; ++k) best[a][k] = fminf(best[a][k], __shfl_xor_sync(0xffffffffu, best[a][k], o));
    }
    if (lane == 0) {
        float* c = code + (size_t)env * kEnvCode;
        c[0] = cnt[0] / 64.0f;
        c[1] = cnt[1] / 64.0f;
        c[2] = cnt[2] / 64.0f;
        c[3] = (float)np / 64.0f;
        for (int a = 0; a < 8; ++a)
            for (int k = 0; k < 3; ++k) c[4 + a * 3 + k] = fminf(fmaxf(best[a][k], -0.5f), 1.5f);
        const float inv = np > 0 ? 1.0f / (float)np : 0.0f;
        for (int k = 0; k < 4; ++k) c[28 + k] = mean[k] * inv;
    }
}

cudaError_t launch_env_encode(const float4* blobs, const float4* env_hdr, int num_envs, float* code, cudaStream_t st) {
    if (num_envs <= 0) return cudaSuccess;
    env_encode_kernel<<<(num_envs * 32 + 255) / 256, 256, 0, st>>>(blobs, env_hdr, num_envs, code);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ training rows
__global__ void gather_rows_kernel(const uint4* __restrict__ x, const uint8_t* __restrict__ y,
                                   const int* __restrict__ perm, int rows, uint4* __restrict__ x2,
                                   uint8_t* __restrict__ y2) {
    constexpr int W = kMlpIn * 2 / 16;  // uint4 words per row
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows) return;
    const int src = perm[i];
#pragma unroll
    for (int w = 0; w < W; ++w) x2[(size_t)i * W + w] = x[(size_t)src * W + w];
    y2[i] = y[src];
}

cudaError_t launch_gather_rows(const uint16_t* x, const uint8_t* y, const int* perm, int rows, uint16_t* x2,
                               uint8_t* y2, cudaStream_t st) {
    static_assert(kMlpIn * 2 % 16 == 0, "feature rows are whole 16-byte words");
    if (rows <= 0) return cudaSuccess;
    gather_rows_kernel<<<(rows + 255) / 256, 256, 0, st>>>(reinterpret_cast<const uint4*>(x), y, perm, rows,
                                                           reinterpret_cast<uint4*>(x2), y2);
    return cudaGetLastError();
}

}  // namespace bcc
