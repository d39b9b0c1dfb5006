// bcc_mlp.cu -- the collision-likelihood MLP on 5th-generation tensor cores.
//
// Network (per sample configuration in one environment):
//     x (48: normalised joints, 32 environment code, zeros, position along the edge,
//     bias input) -> 128 -> 128 -> 128 -> 1
// ReLU between layers, logit output.  Weights are BF16 in shared memory (core-matrix
// images, see bcc_tc.cuh), products accumulate in FP32 tensor memory via tcgen05.mma
// (M = 128 rows per tile, N = 128).  Activations are BF16, in tensor memory in the
// forward kernel (biases and the last layer are MMAs too, the epilogue is a ReLU), in
// shared memory in the training kernel (bias, ReLU and the last dot product in FP32
// registers).
//
// Parameters (FP32 masters, flat, kMlpParams floats):
//     W1 [48][128] (in x out), b1 [128], W2 [128][128], b2 [128],
//     W3 [128][128], b3 [128], w4 [128], b4 [1]
#include <cstdint>
#include <cstring>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/bcc.h"
#include "bcc_ctx.h"
#include "bcc_device.cuh"
#include "bcc_mlp.h"
#include "bcc_tc.cuh"

namespace bcc {

// Offsets of the parameter blocks in the flat FP32 vector.
constexpr int kOffW1 = 0;
constexpr int kOffB1 = kOffW1 + kMlpIn * kMlpHidden;
constexpr int kOffW2 = kOffB1 + kMlpHidden;
constexpr int kOffB2 = kOffW2 + kMlpHidden * kMlpHidden;
constexpr int kOffW3 = kOffB2 + kMlpHidden;
constexpr int kOffB3 = kOffW3 + kMlpHidden * kMlpHidden;
constexpr int kOffW4 = kOffB3 + kMlpHidden;
constexpr int kOffB4 = kOffW4 + kMlpHidden;
static_assert(kOffB4 + 1 == kMlpParams, "parameter layout");

// Images (BF16 core-matrix layouts, bcc_tc.cuh): W1^T [128][48] -- its column
// 47 carries b1, the forward kernel reads feature 47 as 1 --, W2^T, W3^T
// [128][128] (the training kernel uses these three), then for the forward
// kernel only: W4 [16][128] (row 0 = w4, the last layer as an N = 16 MMA) and
// B2, B3 [128][16] (column 0 = b2 / b3, added by one K = 16 MMA against a
// ones column).
constexpr uint32_t kImgW1 = kMlpHidden * kMlpIn * 2;       // 12288
constexpr uint32_t kImgW = kMlpHidden * kMlpHidden * 2;    // 32768
constexpr uint32_t kImgSmall = kMlpHidden * 16 * 2;         // 4096: W4, B2, B3 and the ones image
constexpr uint32_t kImagesW = kImgW1 + 2 * kImgW;           // W1T | W2T | W3T
constexpr uint32_t kImagesBytes = kImagesW + 3 * kImgSmall;  // ... | W4 | B2 | B3
constexpr int kBiasCol = kMlpIn - 1;                        // feature 47: reserved, read as 1 by the forward kernel

// Shared-memory map of the forward kernel (bytes): the images, the ones image
// (A operand of the bias MMAs), then per row group its X tile (128 x 48), b4, the
// groups' mbarriers and the TMEM address slot.
constexpr uint32_t kSmW1 = 0;
constexpr uint32_t kSmW2 = kSmW1 + kImgW1;
constexpr uint32_t kSmW3 = kSmW2 + kImgW;
constexpr uint32_t kSmW4 = kSmW3 + kImgW;
constexpr uint32_t kSmB2 = kSmW4 + kImgSmall;
constexpr uint32_t kSmB3 = kSmB2 + kImgSmall;
constexpr uint32_t kSmOnes = kSmB3 + kImgSmall;
constexpr int kFwdGroups = 2;                              // independent 128-row tile streams per CTA
constexpr int kFwdGroupThreads = 256;                      // two threads a row
// Tensor memory of group g, columns 256 g ..: the accumulator (128), H as the next
// layer's A operand (64, two BF16 values a column), the logits' accumulator (16).
constexpr uint32_t kFwdTmemCols = 512;
constexpr uint32_t kFwdH = kMlpHidden;
constexpr uint32_t kFwdC = kFwdH + kMlpHidden / 2;
constexpr uint32_t kSmGroup0 = kSmOnes + kImgSmall;
constexpr uint32_t kSmGroupStride = kImgW1;
constexpr uint32_t kSmVec = kSmGroup0 + kFwdGroups * kSmGroupStride;  // b4
constexpr uint32_t kSmBar = kSmVec + 16;
constexpr uint32_t kSmTmem = kSmBar + 8 * kFwdGroups;
constexpr uint32_t kFwdSmem = kSmTmem + 8;
static_assert(kSmGroup0 % 16 == 0 && kSmGroupStride % 16 == 0, "core-matrix images are 16-byte aligned");
static_assert(kSmW4 == kImagesW && kSmOnes == kImagesBytes, "forward images are copied as one block");
static_assert(kFwdSmem <= 227 * 1024, "forward kernel shared memory");

// ---------------------------------------------------------------- images
// FP32 masters -> BF16 core-matrix images of W1^T [128][48], W2^T, W3^T.
// Feature 47 is zero in every input row, so W1's row 47 never contributes;
// the image's column 47 holds b1 instead, which the forward kernel adds by
// reading feature 47 as 1 (the training kernel reads it as the 0 it is and
// adds b1 in its epilogue).
__global__ void mlp_pack_kernel(const float* __restrict__ params, uint8_t* __restrict__ images) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n1 = kMlpHidden * kMlpIn, n2 = kMlpHidden * kMlpHidden, ns = kMlpHidden * 16;
    if (i < n1) {
        const int out = i / kMlpIn, in = i % kMlpIn;
        const float w = in == kBiasCol ? params[kOffB1 + out] : params[kOffW1 + in * kMlpHidden + out];
        *reinterpret_cast<__nv_bfloat16*>(images + tc::cm_offset(out, in, kMlpIn)) = __float2bfloat16_rn(w);
    } else if (i < n1 + 2 * n2) {
        const int j = i - n1;
        const int layer = j / n2, r = j % n2;
        const int out = r / kMlpHidden, in = r % kMlpHidden;
        const float w = params[(layer ? kOffW3 : kOffW2) + in * kMlpHidden + out];
        *reinterpret_cast<__nv_bfloat16*>(images + kImgW1 + layer * kImgW + tc::cm_offset(out, in, kMlpHidden)) =
            __float2bfloat16_rn(w);
    } else if (i < n1 + 2 * n2 + ns) {  // W4 [16][128]: row 0 = w4
        const int j = i - n1 - 2 * n2;
        const int out = j / kMlpHidden, in = j % kMlpHidden;
        const float w = out == 0 ? params[kOffW4 + in] : 0.0f;
        *reinterpret_cast<__nv_bfloat16*>(images + kImagesW + tc::cm_offset(out, in, kMlpHidden)) =
            __float2bfloat16_rn(w);
    } else if (i < n1 + 2 * n2 + 3 * ns) {  // B2, B3 [128][16]: column 0 = bias
        const int j = i - n1 - 2 * n2 - ns;
        const int layer = j / ns, r = j % ns;
        const int out = r / 16, in = r % 16;
        const float w = in == 0 ? params[(layer ? kOffB3 : kOffB2) + out] : 0.0f;
        *reinterpret_cast<__nv_bfloat16*>(images + kImagesW + (1 + layer) * kImgSmall + tc::cm_offset(out, in, 16)) =
            __float2bfloat16_rn(w);
    }
}

// ---------------------------------------------------------------- forward
// ReLU of two FP32 values, rounded to BF16 and packed (lo in the low half).
__device__ __forceinline__ uint32_t relu_bf16x2(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

// Forward epilogue of a hidden layer whose bias the MMAs already added: this
// thread's half (64 columns) of its accumulator row, ReLU, BF16 into the H columns
// (one conversion per two values).
__device__ __forceinline__ void epilogue_relu_only(uint32_t acc, uint32_t h) {
    float v[64];
    uint32_t w[32];
    tc::tmem_ld64(acc, v);
#pragma unroll
    for (int i = 0; i < 32; ++i) w[i] = relu_bf16x2(v[2 * i], v[2 * i + 1]);
    tc::tmem_st32(h, w);
    tc::wait_st();
}

// Barrier of one warp group (named barrier 1 + group) that also ORs a predicate
// over its threads.
__device__ __forceinline__ bool group_sync_or(bool pred, int grp) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)pred), "r"(1 + grp), "n"(kFwdGroupThreads)
        : "memory");
    return r != 0;
}

// Persistent: each CTA loads the weights once; its two warp groups (8 warps, two
// threads a row) run independent streams of 128-row tiles, each with its own X
// buffer, TMEM columns and mbarrier, so one group's MMAs overlap the other's
// epilogues.  The biases ride in the MMAs (b1 as column 47 of W1^T against feature
// 47 read as 1; b2, b3 by a K = 16 MMA of a ones column against B2 / B3) and the
// output layer is an N = 16 MMA against W4, issued together with the next tile's
// first layer, so a tile is three rounds of MMAs and epilogues.  x: BF16
// [rows][48] row-major (feature 47 zero); logits: FP32 [rows].
//
// H lives in tensor memory as the A operand of layers 2 to 4.  With H in shared
// memory a 128 x 128 x 16 MMA read 8 KB of operands, and with the epilogue's
// stores a tile took 2500 cycles of the shared memory's 128 B a cycle: 109 us for
// 1 000 003 rows.  Without, it takes 960 of a stream's 3 x 1800, and 89 us; the
// MMAs alone would take 1400 a tile.  A stage's chain bounds it: 440 cycles around
// its MMAs, 160 of epilogue, 130 of barrier, and the other stream's MMAs.  So the
// logits and the next X are written behind the second layer's MMAs (98 us before
// them).  Four streams of 128 columns, layers in two halves of 64 outputs, spilled
// and took 113 us.
__global__ void __launch_bounds__(kFwdGroupThreads * kFwdGroups, 1)
    mlp_forward_kernel(const uint16_t* __restrict__ x, int rows, const int* __restrict__ rows_dev,
                       const uint4* __restrict__ images, const float* __restrict__ params, float* __restrict__ logits,
                       int* __restrict__ err) {
    // rows_dev (optional): the row count produced on the device, capped by rows.
    if (rows_dev) rows = min(rows, *rows_dev);
    // The grid is sized for the host's row bound; CTAs without a tile of the
    // device count leave before loading the weights.
    if ((long long)blockIdx.x * kFwdGroups * 128 >= (long long)rows) return;
    extern __shared__ __align__(1024) uint8_t sm[];
    const int t = threadIdx.x, warp = t >> 5, grp = t / kFwdGroupThreads, gt = t % kFwdGroupThreads;
    const int r = gt & 127, half = gt >> 7;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kSmBar) + grp;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + kSmTmem);
    float* vec = reinterpret_cast<float*>(sm + kSmVec);
    uint8_t* xs = sm + kSmGroup0 + grp * kSmGroupStride;

    for (uint32_t i = t; i < kImagesBytes / 16; i += blockDim.x) reinterpret_cast<uint4*>(sm)[i] = images[i];
    if (t < 128) {  // ones image [128][16]: column 0 = 1 (BF16 0x3f80), the rest 0
        *reinterpret_cast<uint4*>(sm + kSmOnes + tc::cm_offset(t, 0, 16)) = make_uint4(0x3f80u, 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(sm + kSmOnes + tc::cm_offset(t, 8, 16)) = make_uint4(0u, 0u, 0u, 0u);
    }
    if (t == 0) {
        vec[0] = params[kOffB4];
        for (int g = 0; g < kFwdGroups; ++g) mbar_init(reinterpret_cast<uint64_t*>(sm + kSmBar) + g, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tc::tmem_alloc(tmem_slot, kFwdTmemCols);
    tc::fence_async_smem();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tmem_slot + 256u * grp;
    const uint32_t taddr = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    const uint32_t idesc = tc::make_idesc_bf16(128, kMlpHidden, 0, 0);
    const uint32_t idesc16 = tc::make_idesc_bf16(128, 16, 0, 0);
    const uint32_t sbase = tc::smem_addr(sm);
    const float b4 = vec[0];
    uint32_t phase = 0;
    bool bad = false;

    const int tiles = (rows + 127) / 128;
    const int tile_step = gridDim.x * kFwdGroups;
    // X rows are loaded one tile ahead into registers, so their latency overlaps
    // the current tile's layers: half a row a thread, three 16-byte chunks.
    constexpr int kChunks = kMlpIn / 16;
    static_assert(kMlpIn % 16 == 0 && kBiasCol == kMlpIn - 1, "the bias feature is the last of the row's last chunk");
    uint4 xv[kChunks];
    auto load_x = [&](int tile) {
        const int row = tile * 128 + r;
        const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)row * kMlpIn) + kChunks * half;
#pragma unroll
        for (int j = 0; j < kChunks; ++j) xv[j] = (tile < tiles && row < rows) ? src[j] : make_uint4(0, 0, 0, 0);
    };
    // ... into the X buffer; feature 47 (zero in the input) is read as 1 to pick up
    // b1 from W1^T's column 47.
    auto store_x = [&] {
        if (half) xv[kChunks - 1].w = (xv[kChunks - 1].w & 0xffffu) | 0x3f800000u;
#pragma unroll
        for (int j = 0; j < kChunks; ++j)
            *reinterpret_cast<uint4*>(xs + tc::cm_offset(r, 8 * (kChunks * half + j), kMlpIn)) = xv[j];
        tc::fence_async_smem();
    };
    // MMAs of a stage, by the group's first thread.
    auto first_layer = [&] {
        const uint32_t a0 = tc::smem_addr(xs), b0 = sbase + kSmW1;
        constexpr uint32_t sbo = (uint32_t)(kMlpIn / 8) * 128u;
        for (int s = 0; s < kMlpIn / 16; ++s)
            tc::mma_bf16(tmem, tc::make_desc(a0 + 256u * s, 128u, sbo), tc::make_desc(b0 + 256u * s, 128u, sbo), idesc,
                         s > 0 ? 1u : 0u);
    };
    auto h_layer = [&](uint32_t d, uint32_t b0, uint32_t id) {
        constexpr uint32_t sbo = (uint32_t)(kMlpHidden / 8) * 128u;
        for (int s = 0; s < kMlpHidden / 16; ++s)
            tc::mma_bf16_ts(d, tmem + kFwdH + 8u * s, tc::make_desc(b0 + 256u * s, 128u, sbo), id, s > 0 ? 1u : 0u);
    };
    // Waits for the stage in flight (once a wait has run out, for none).
    auto await = [&] {
        if (!bad) bad = !mbar_wait_bounded(bar, phase, 1u << 22);
        if (!bad) phase ^= 1u;
        tc::fence_after();
    };
    auto write_logits = [&](int tile) {
        if (half) return;  // whole warps
        const float z = tc::tmem_ld1(taddr + kFwdC);
        tc::wait_ld();
        const int row = tile * 128 + r;
        if (!bad && row < rows) logits[row] = z + b4;
    };

    int tile = blockIdx.x * kFwdGroups + grp, done = -1;  // done: the tile whose logits are in flight
    bool stop = tile >= tiles;
    if (!stop) {
        load_x(tile);
        store_x();
        load_x(tile + tile_step);
        tc::fence_before();
        group_sync_or(false, grp);
        if (gt == 0) {
            tc::fence_after();
            first_layer();
            tc::commit(bar);
        }
    }
    for (; !stop && tile < tiles; tile += tile_step) {
        const int next = tile + tile_step;
#pragma unroll 1
        for (int layer = 1; layer < 4; ++layer) {
            await();
            epilogue_relu_only(taddr + 64u * half, taddr + kFwdH + 32u * half);
            tc::fence_before();
            if (group_sync_or(bad, grp)) {  // group-uniform decision
                bad = stop = true;
                break;
            }
            if (gt == 0) {
                tc::fence_after();
                if (layer < 3) {
                    h_layer(tmem, sbase + (layer == 1 ? kSmW2 : kSmW3), idesc);
                    // + bias: ones [128][16] x B [128][16]^T
                    tc::mma_bf16(tmem, tc::make_desc(sbase + kSmOnes, 128u, 256u),
                                 tc::make_desc(sbase + (layer == 1 ? kSmB2 : kSmB3), 128u, 256u), idesc, 1u);
                } else {
                    h_layer(tmem + kFwdC, sbase + kSmW4, idesc16);
                    if (next < tiles) first_layer();
                }
                tc::commit(bar);
            }
            if (layer == 1) {  // behind these MMAs: the last tile's logits, the next tile's X
                if (done >= 0) write_logits(done);
                store_x();
                load_x(next + tile_step);
            }
        }
        done = tile;
    }
    if (done >= 0 && !stop) {
        await();
        write_logits(done);
    }
    if (bad) {
        atomicOr(err, 1);
        mbar_wait_bounded(bar, phase, 1u << 22);  // let in-flight MMAs finish before freeing TMEM
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (warp == 0) tc::tmem_free(*tmem_slot, kFwdTmemCols);
}

// ---------------------------------------------------------------- training
// One CTA runs forward and backward over its 128-row tiles.  Activations stay in shared memory as BF16 images; the three
// weight-gradient accumulators stay in tensor memory across tiles and are
// added to the global FP32 gradient once at the end.  Loss: mean binary
// cross-entropy of the logit against the 0/1 label (scale = 1 / total rows).
//
// GEMMs (M = 128 unless noted; "K" / "MN" = operand read K- or MN-major):
//   forward   z1 = X W1 (A=X K, B=W1T K), z2 = H1 W2, z3 = H2 W3
//   backward  dW3 += H2^T dZ3   (A=H2 MN, B=dZ3 MN, K = rows)
//             dH2  = dZ3 W3^T   (A=dZ3 K, B=W3T MN)
//             dW2 += H1^T dZ2,  dH1 = dZ2 W2^T
//             dW1^T += dZ1^T X  (A=dZ1 MN, B=X MN, N = 48)
constexpr uint32_t kTrW1 = 0;
constexpr uint32_t kTrW2 = kTrW1 + kImgW1;
constexpr uint32_t kTrW3 = kTrW2 + kImgW;
constexpr uint32_t kTrX = kTrW3 + kImgW;
constexpr uint32_t kTrH1 = kTrX + kImgW1;
constexpr uint32_t kTrH2 = kTrH1 + kImgW;
constexpr uint32_t kTrD = kTrH2 + kImgW;
constexpr uint32_t kTrVec = kTrD + kImgW;                 // b1 b2 b3 w4 b4 (params)
constexpr uint32_t kTrGrad = kTrVec + 5 * kMlpHidden * 4;  // db1 db2 db3 dw4 db4 loss
constexpr uint32_t kTrPart = kTrGrad + 5 * kMlpHidden * 4 + 16;
constexpr uint32_t kTrBar = kTrPart + 128 * 4;             // MMAs, weights
constexpr uint32_t kTrTmem = kTrBar + 16;
constexpr uint32_t kTrainSmem = kTrTmem + 8;
static_assert(kOffW2 % 4 == 0 && kOffW3 % 4 == 0 && kTrBar % 8 == 0 && kTrainSmem <= 227 * 1024, "training kernel layout");
// TMEM columns: forward / backward-data accumulator, dW3, dW2, dW1^T.
constexpr uint32_t kColAcc = 0, kColW3 = 128, kColW2 = 256, kColW1 = 384;

__device__ __forceinline__ void gemm_issue(uint32_t d, uint32_t a0, uint32_t a_lbo, uint32_t a_sbo, uint32_t a_step,
                                           uint32_t b0, uint32_t b_lbo, uint32_t b_sbo, uint32_t b_step, int ksteps,
                                           uint32_t idesc, bool accumulate) {
    for (int s = 0; s < ksteps; ++s)
        tc::mma_bf16(d, tc::make_desc(a0 + a_step * s, a_lbo, a_sbo), tc::make_desc(b0 + b_step * s, b_lbo, b_sbo),
                     idesc, (accumulate || s > 0) ? 1u : 0u);
}

// Sum over the warp's 32 lanes of each of 32 per-lane values: lane i returns the
// sum of v[i].  Halves the values with the lanes: 31 shuffles where a butterfly
// per value takes 160.
__device__ __forceinline__ float warp_colsum32(float (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const float send = up ? v[i] : v[i + o];
            const float keep = up ? v[i + o] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0];
}

// 32 values as BF16 into columns c0 .. c0 + 31 of row r of a 128-column image.
__device__ __forceinline__ void store_bf16x32(uint8_t* img, int r, int c0, const float* v) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            __nv_bfloat162 h = __floats2bfloat162_rn(v[8 * q + 2 * i], v[8 * q + 2 * i + 1]);
            w[i] = *reinterpret_cast<uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(img + tc::cm_offset(r, c0 + 8 * q, kMlpHidden)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Zero the values whose activation (BF16 image, >= 0) is zero.
__device__ __forceinline__ void mask_by_activation(const uint8_t* img, int r, int c0, float* v) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint4 h = *reinterpret_cast<const uint4*>(img + tc::cm_offset(r, c0 + 8 * q, kMlpHidden));
        const uint32_t w[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if ((int16_t)(w[i] & 0xffffu) <= 0) v[8 * q + 2 * i] = 0.0f;
            if ((int16_t)(w[i] >> 16) <= 0) v[8 * q + 2 * i + 1] = 0.0f;
        }
    }
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    tc::tmem_ld16(taddr, v);
    tc::tmem_ld16(taddr + 16, v + 16);
    tc::wait_ld();
}

__device__ __forceinline__ void red_add4(float* p, float a, float b, float c, float d) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}

// Two threads per row: thread t holds row t % 128 and column half t / 128, so
// each of the six epilogues is 64 columns of one row deep.  A batch of up to
// 148 x 128 rows is one tile per CTA and the kernel is that tile's serial chain:
// with one thread a row, a butterfly of five shuffles per column sum, 2-byte
// reads of the activations, word-by-word weight loads and scalar atomics it took
// 150 us for 16 384 rows; 27 us now.
constexpr int kTrainThreads = 256;

__global__ void __launch_bounds__(kTrainThreads, 1)
    mlp_train_kernel(const uint16_t* __restrict__ x, const uint8_t* __restrict__ y, int rows,
                     const uint4* __restrict__ images, const float* __restrict__ params, float* __restrict__ grads,
                     float* __restrict__ loss_sum, int* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t sm[];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int r = t & 127, half = t >> 7, col0 = half * (kMlpHidden / 2);
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kTrBar);
    uint64_t* bar_w = bar + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + kTrTmem);
    float* vec = reinterpret_cast<float*>(sm + kTrVec);    // b1 | b2 | b3 | w4 | b4
    float* gv = reinterpret_cast<float*>(sm + kTrGrad);    // db1 | db2 | db3 | dw4 | db4, loss
    float* part = reinterpret_cast<float*>(sm + kTrPart);  // [128] logits half way, then whole
    const float inv_rows = 1.0f / (float)rows;

    if (t == 0) {
        mbar_init(bar, 1);
        mbar_init(bar_w, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        bulk_copy_g2s(sm + kTrW1, images, kImagesW, bar_w);
    }
    for (int i = t; i < kMlpHidden; i += kTrainThreads) {
        vec[i] = params[kOffB1 + i];
        vec[kMlpHidden + i] = params[kOffB2 + i];
        vec[2 * kMlpHidden + i] = params[kOffB3 + i];
        vec[3 * kMlpHidden + i] = params[kOffW4 + i];
    }
    for (int i = t; i < 5 * kMlpHidden + 4; i += kTrainThreads) gv[i] = 0.0f;
    if (t == 0) vec[4 * kMlpHidden] = params[kOffB4];
    if (warp == 0) tc::tmem_alloc(tmem_slot, 512);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t lane_off = (uint32_t)(32 * (warp & 3)) << 16;
    const uint32_t acc = tmem + lane_off + kColAcc + (uint32_t)col0;  // this thread's half row of the accumulator
    const uint32_t sb = tc::smem_addr(sm);
    const uint32_t id_fwd = tc::make_idesc_bf16(128, 128, 0, 0);   // A K-major, B K-major
    const uint32_t id_dw = tc::make_idesc_bf16(128, 128, 1, 1);    // A MN, B MN
    const uint32_t id_dh = tc::make_idesc_bf16(128, 128, 0, 1);    // A K, B MN
    const uint32_t id_dw1 = tc::make_idesc_bf16(128, 48, 1, 1);    // dW1^T: N = 48
    uint32_t phase = 0;
    bool first = true;
    // The weights' copy; waited for again (bounded) before the CTA may leave.
    const bool ok_w = mbar_wait_bounded(bar_w, 0u, 1u << 22);
    bool bad = __syncthreads_or(!ok_w) != 0;
    if (bad) mbar_wait_bounded(bar_w, 0u, 1u << 22);
    const bool issued_any = !bad;
    float* db1 = gv;
    float* db2 = gv + kMlpHidden;
    float* db3 = gv + 2 * kMlpHidden;
    float* dw4 = gv + 3 * kMlpHidden;

    // Issue (thread 0) + wait (all): returns false on a timed-out wait.
    auto sync_issue = [&](auto&& issue) -> bool {
        tc::fence_async_smem();
        tc::fence_before();
        __syncthreads();
        if (t == 0) {
            tc::fence_after();
            issue();
            tc::commit(bar);
        }
        const bool ok = mbar_wait_bounded(bar, phase, 1u << 22);
        if (__syncthreads_or(!ok)) return false;
        phase ^= 1u;
        tc::fence_after();
        return true;
    };
    // Hidden layer's epilogue: accumulator + bias, ReLU, BF16 into an H image.
    auto relu_to = [&](const float* bias, uint8_t* himg) {
#pragma unroll 1
        for (int c = 0; c < kMlpHidden / 2; c += 32) {
            float v[32];
            tmem_ld32(acc + c, v);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = fmaxf(v[i] + bias[col0 + c + i], 0.0f);
            store_bf16x32(himg, r, col0 + c, v);
        }
    };
    // A hidden layer's dZ: the accumulator where the activation is positive, its
    // column sums added to db and its BF16 image written.
    auto dz_to = [&](const uint8_t* himg, float* db) {
#pragma unroll 1
        for (int c = 0; c < kMlpHidden / 2; c += 32) {
            float v[32];
            tmem_ld32(acc + c, v);
            mask_by_activation(himg, r, col0 + c, v);
            store_bf16x32(sm + kTrD, r, col0 + c, v);
            const float s = warp_colsum32(v);
            atomicAdd(db + col0 + c + lane, s);
        }
    };

    const int tiles = (rows + 127) / 128;
    for (int tile = blockIdx.x; tile < tiles && !bad; tile += gridDim.x) {
        const int row = tile * 128 + r;
        const bool live = row < rows;
        const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)row * kMlpIn);
#pragma unroll
        for (int j = 0; j < kMlpIn / 16; ++j) {
            const int c = half * (kMlpIn / 16) + j;
            *reinterpret_cast<uint4*>(sm + kTrX + tc::cm_offset(r, 8 * c, kMlpIn)) = live ? src[c] : make_uint4(0, 0, 0, 0);
        }
        const float label = live ? (float)y[row] : 0.0f;

        // ---- forward
        if (!sync_issue([&] { gemm_issue(tmem + kColAcc, sb + kTrX, 128, 768, 256, sb + kTrW1, 128, 768, 256, 3, id_fwd, false); })) { bad = true; break; }
        relu_to(vec, sm + kTrH1);
        if (!sync_issue([&] { gemm_issue(tmem + kColAcc, sb + kTrH1, 128, 2048, 256, sb + kTrW2, 128, 2048, 256, 8, id_fwd, false); })) { bad = true; break; }
        relu_to(vec + kMlpHidden, sm + kTrH2);
        if (!sync_issue([&] { gemm_issue(tmem + kColAcc, sb + kTrH2, 128, 2048, 256, sb + kTrW3, 128, 2048, 256, 8, id_fwd, false); })) { bad = true; break; }
        // The logit is one chain over the 128 columns in order (its last bits decide
        // roundings of every gradient): the lower half's threads, then the upper's.
        float logit = vec[4 * kMlpHidden];
        for (int h = 0; h < 2; ++h) {
            if (half == h) {
                if (h) logit = part[r];
#pragma unroll 1
                for (int c = 0; c < kMlpHidden / 2; c += 32) {
                    float v[32];
                    tmem_ld32(acc + c, v);
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        logit = fmaf(fmaxf(v[i] + vec[2 * kMlpHidden + col0 + c + i], 0.0f), vec[3 * kMlpHidden + col0 + c + i], logit);
                }
                part[r] = logit;
            }
            __syncthreads();
        }
        logit = part[r];
        // ---- loss and dlogit (mean BCE)
        const float prob = 1.0f / (1.0f + __expf(-logit));
        const float dlogit = live ? (prob - label) * inv_rows : 0.0f;
        if (half == 0) {
            const float l = live ? (fmaxf(logit, 0.0f) - logit * label + log1pf(__expf(-fabsf(logit)))) : 0.0f;
            float s1 = l, s2 = dlogit;
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                s1 += __shfl_xor_sync(0xffffffffu, s1, o);
                s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            }
            if (lane == 0) {
                atomicAdd(gv + 5 * kMlpHidden + 1, s1);
                atomicAdd(gv + 4 * kMlpHidden, s2);
            }
        }
        // dz3 = dlogit * w4 * (h3 > 0); dw4 += dlogit * h3; db3 += dz3
#pragma unroll 1
        for (int c = 0; c < kMlpHidden / 2; c += 32) {
            float v[32], g3[32];
            tmem_ld32(acc + c, v);
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const float h3 = fmaxf(v[i] + vec[2 * kMlpHidden + col0 + c + i], 0.0f);
                g3[i] = h3 > 0.0f ? dlogit * vec[3 * kMlpHidden + col0 + c + i] : 0.0f;
                v[i] = dlogit * h3;
            }
            store_bf16x32(sm + kTrD, r, col0 + c, g3);
            const float s3 = warp_colsum32(g3), s4 = warp_colsum32(v);
            atomicAdd(db3 + col0 + c + lane, s3);
            atomicAdd(dw4 + col0 + c + lane, s4);
        }
        // ---- dW3 += H2^T dZ3 ; dH2 = dZ3 W3^T
        const bool acc_w = !first;
        if (!sync_issue([&] {
                gemm_issue(tmem + kColW3, sb + kTrH2, 2048, 128, 4096, sb + kTrD, 2048, 128, 4096, 8, id_dw, acc_w);
                gemm_issue(tmem + kColAcc, sb + kTrD, 128, 2048, 256, sb + kTrW3, 2048, 128, 4096, 8, id_dh, false);
            })) { bad = true; break; }
        dz_to(sm + kTrH2, db2);
        // ---- dW2 += H1^T dZ2 ; dH1 = dZ2 W2^T
        if (!sync_issue([&] {
                gemm_issue(tmem + kColW2, sb + kTrH1, 2048, 128, 4096, sb + kTrD, 2048, 128, 4096, 8, id_dw, acc_w);
                gemm_issue(tmem + kColAcc, sb + kTrD, 128, 2048, 256, sb + kTrW2, 2048, 128, 4096, 8, id_dh, false);
            })) { bad = true; break; }
        dz_to(sm + kTrH1, db1);
        // ---- dW1^T += dZ1^T X
        if (!sync_issue([&] {
                gemm_issue(tmem + kColW1, sb + kTrD, 2048, 128, 4096, sb + kTrX, 768, 128, 1536, 8, id_dw1, acc_w);
            })) { bad = true; break; }
        first = false;
    }
    if (bad) {
        if (t == 0) atomicOr(err, 1);
        if (issued_any) mbar_wait_bounded(bar, phase, 1u << 22);
    }
    // ---- write gradients: a thread owns its row's half of each accumulator.
    if (!bad && !first) {
        const uint32_t lanes = tmem + lane_off;
#pragma unroll 1
        for (int c = col0; c < col0 + kMlpHidden / 2; c += 32) {
            float v[32];
            tmem_ld32(lanes + kColW3 + c, v);
#pragma unroll
            for (int i = 0; i < 32; i += 4) red_add4(grads + kOffW3 + r * kMlpHidden + c + i, v[i], v[i + 1], v[i + 2], v[i + 3]);
            tmem_ld32(lanes + kColW2 + c, v);
#pragma unroll
            for (int i = 0; i < 32; i += 4) red_add4(grads + kOffW2 + r * kMlpHidden + c + i, v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
#pragma unroll 1
        for (int c = half * 32; c < (half ? kMlpIn : 32); c += 16) {
            float v[16];
            tc::tmem_ld16(lanes + kColW1 + c, v);
            tc::wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) atomicAdd(grads + kOffW1 + (c + i) * kMlpHidden + r, v[i]);
        }
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (!bad && t < 128) {
        atomicAdd(grads + kOffB1 + t, db1[t]);
        atomicAdd(grads + kOffB2 + t, db2[t]);
        atomicAdd(grads + kOffB3 + t, db3[t]);
        atomicAdd(grads + kOffW4 + t, dw4[t]);
        if (t == 0) {
            atomicAdd(grads + kOffB4, gv[4 * kMlpHidden]);
            atomicAdd(loss_sum, gv[5 * kMlpHidden + 1]);
        }
    }
    if (warp == 0) tc::tmem_free(tmem, 512);
}

// Byte offset of parameter i's BF16 copy in the images, or -1 (b4, and W1's row of
// the bias feature, have none).  The inverse of mlp_pack_kernel's map.
__device__ __forceinline__ int image_offset(int i) {
    if (i < kOffB1) {
        const int in = i / kMlpHidden, out = i - in * kMlpHidden;
        return in == kBiasCol ? -1 : (int)tc::cm_offset(out, in, kMlpIn);
    }
    if (i < kOffW2) return (int)tc::cm_offset(i - kOffB1, kBiasCol, kMlpIn);
    if (i < kOffW4) {  // W2 b2 W3 b3
        const int layer = i >= kOffW3, j = i - (layer ? kOffW3 : kOffW2);
        const int in = j / kMlpHidden, out = j - in * kMlpHidden;
        return in < kMlpHidden ? (int)(kImgW1 + layer * kImgW + tc::cm_offset(out, in, kMlpHidden))
                               : (int)(kImagesW + (1 + layer) * kImgSmall + tc::cm_offset(out, 0, 16));
    }
    return i < kOffB4 ? (int)(kImagesW + tc::cm_offset(0, i - kOffW4, kMlpHidden)) : -1;
}

// Adam on the FP32 masters (bias-corrected) and each parameter's BF16 copy, in
// one pass; does nothing once the gradient kernel has flagged an error.
__global__ void mlp_adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                                float* __restrict__ v, uint8_t* __restrict__ images, const int* __restrict__ err, int n,
                                float lr, float b1, float b2, float eps, float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || *err) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float w = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = w;
    const int at = image_offset(i);
    if (at >= 0) *reinterpret_cast<__nv_bfloat16*>(images + at) = __float2bfloat16_rn(w);
}

cudaError_t mlp_train_grads(const uint16_t* d_x, const uint8_t* d_y, int rows, const uint8_t* d_images,
                            const float* d_params, float* d_grads, int num_sms, cudaStream_t st) {
    float* d_loss = d_grads + kMlpParams;
    int* d_err = reinterpret_cast<int*>(d_loss + 1);
    cudaError_t e = cudaMemsetAsync(d_grads, 0, kMlpGradBytes, st);
    if (e != cudaSuccess) return e;
    if (rows <= 0) return cudaSuccess;
    e = cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem);
    if (e != cudaSuccess) return e;
    const int tiles = (rows + 127) / 128;
    const int grid = tiles < num_sms ? tiles : num_sms;
    mlp_train_kernel<<<grid, kTrainThreads, kTrainSmem, st>>>(d_x, d_y, rows, reinterpret_cast<const uint4*>(d_images), d_params,
                                                    d_grads, d_loss, d_err);
    return cudaGetLastError();
}

cudaError_t mlp_adam(float* d_params, const float* d_grads, float* d_m, float* d_v, uint8_t* d_images, long long step,
                     float lr, cudaStream_t st) {
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
    mlp_adam_kernel<<<(kMlpParams + 255) / 256, 256, 0, st>>>(d_params, d_grads, d_m, d_v, d_images,
                                                              reinterpret_cast<const int*>(d_grads + kMlpParams + 1),
                                                              kMlpParams, lr, b1, b2, 1e-8f, c1, c2);
    return cudaGetLastError();
}

cudaError_t mlp_pack(const float* d_params, uint8_t* d_images, cudaStream_t st) {
    const int n = kMlpHidden * kMlpIn + 2 * kMlpHidden * kMlpHidden + 3 * kMlpHidden * 16;
    mlp_pack_kernel<<<(n + 255) / 256, 256, 0, st>>>(d_params, d_images);
    return cudaGetLastError();
}

cudaError_t mlp_forward(const uint16_t* d_x, int rows, const uint8_t* d_images, const float* d_params,
                        float* d_logits, int* d_err, int num_sms, cudaStream_t st, const int* d_rows) {
    if (rows <= 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwdSmem);
    if (e != cudaSuccess) return e;
    const int tiles = (rows + 127) / 128;
    const int ctas = (tiles + kFwdGroups - 1) / kFwdGroups;
    const int grid = ctas < num_sms ? ctas : num_sms;
    mlp_forward_kernel<<<grid, kFwdGroupThreads * kFwdGroups, kFwdSmem, st>>>(d_x, rows, d_rows,
                                                                 reinterpret_cast<const uint4*>(d_images), d_params,
                                                                 d_logits, d_err);
    return cudaGetLastError();
}

}  // namespace bcc

// ====================================================================== C ABI
namespace {

bcc_status mlp_fail(bcc_ctx* c, bcc_status s, const char* msg) {
    if (c) c->err = msg;
    return s;
}

int sm_count(int dev) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

// Up to kMlpGradBytes of device memory into the context's pinned buffer
// (mlp.host), after everything queued on st.
bool to_host(bcc_ctx* ctx, const void* src, size_t bytes, cudaStream_t st) {
    if (!ctx->mlp.host && cudaMallocHost(&ctx->mlp.host, bcc::kMlpGradBytes) != cudaSuccess) return false;
    return cudaMemcpyAsync(ctx->mlp.host, src, bytes, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
           cudaStreamSynchronize(st) == cudaSuccess;
}

}  // namespace

extern "C" {

int32_t bcc_mlp_num_params(void) { return bcc::kMlpParams; }

bcc_status bcc_mlp_set_params(bcc_ctx* ctx, const float* params, int32_t n) {
    if (!ctx || !params || n != bcc::kMlpParams) return mlp_fail(ctx, BCC_ERR_INVALID_ARGUMENT, "bad MLP parameters");
    if (cudaSetDevice(ctx->device) != cudaSuccess) return BCC_ERR_CUDA;
    bcc::MlpState& m = ctx->mlp;
    const size_t pb = sizeof(float) * bcc::kMlpParams;
    if (m.params.ensure(pb) != cudaSuccess || m.grads.ensure(bcc::kMlpGradBytes) != cudaSuccess || m.adam_m.ensure(pb) != cudaSuccess ||
        m.adam_v.ensure(pb) != cudaSuccess || m.images.ensure(bcc::kImagesBytes) != cudaSuccess)
        return mlp_fail(ctx, BCC_ERR_CUDA, "MLP allocation failed");
    if (cudaMemcpy(m.params.p, params, pb, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(m.adam_m.p, 0, pb) != cudaSuccess || cudaMemset(m.adam_v.p, 0, pb) != cudaSuccess ||
        cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess)  // (see copy_in, bcc_api.cu)
        return mlp_fail(ctx, BCC_ERR_CUDA, "MLP upload failed");
    if (bcc::mlp_pack(m.params.as<float>(), m.images.as<uint8_t>(), ctx->stream) != cudaSuccess ||
        cudaStreamSynchronize(ctx->stream) != cudaSuccess)
        return mlp_fail(ctx, BCC_ERR_CUDA, "MLP pack failed");
    m.step = 0;
    m.ready = true;
    return BCC_OK;
}

bcc_status bcc_mlp_get_params(bcc_ctx* ctx, float* params, int32_t n) {
    if (!ctx || !params || n != bcc::kMlpParams || !ctx->mlp.ready) return BCC_ERR_INVALID_ARGUMENT;
    if (cudaSetDevice(ctx->device) != cudaSuccess ||
        !to_host(ctx, ctx->mlp.params.p, sizeof(float) * n, ctx->stream))
        return BCC_ERR_CUDA;
    std::memcpy(params, ctx->mlp.host, sizeof(float) * n);
    return BCC_OK;
}

bcc_status bcc_mlp_forward(bcc_ctx* ctx, const void* d_x_bf16, int32_t rows, float* d_logits, void* stream) {
    if (!ctx || !ctx->mlp.ready) return mlp_fail(ctx, BCC_ERR_INVALID_ARGUMENT, "MLP parameters not set");
    if (rows < 0 || (rows > 0 && (!d_x_bf16 || !d_logits))) return mlp_fail(ctx, BCC_ERR_INVALID_ARGUMENT, "bad MLP input");
    if (cudaSetDevice(ctx->device) != cudaSuccess) return BCC_ERR_CUDA;
    if (ctx->error_flag.ensure(sizeof(int)) != cudaSuccess) return BCC_ERR_CUDA;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(ctx->error_flag.p, 0, sizeof(int), st) != cudaSuccess) return BCC_ERR_CUDA;
    if (bcc::mlp_forward(static_cast<const uint16_t*>(d_x_bf16), rows, ctx->mlp.images.as<uint8_t>(),
                         ctx->mlp.params.as<float>(), d_logits, ctx->error_flag.as<int>(), sm_count(ctx->device),
                         st) != cudaSuccess)
        return mlp_fail(ctx, BCC_ERR_CUDA, "MLP forward launch failed");
    return BCC_OK;
}

// Gradients (and summed loss) of the mean BCE over `rows` labelled rows,
// computed by the tensor-core training kernel; written to host arrays.
bcc_status bcc_mlp_gradients(bcc_ctx* ctx, const void* d_x_bf16, const uint8_t* d_labels, int32_t rows,
                             float* h_grads, float* h_loss) {
    if (!ctx || !ctx->mlp.ready) return mlp_fail(ctx, BCC_ERR_INVALID_ARGUMENT, "MLP parameters not set");
    if (rows < 0 || (rows > 0 && (!d_x_bf16 || !d_labels))) return BCC_ERR_INVALID_ARGUMENT;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return BCC_ERR_CUDA;
    bcc::MlpState& m = ctx->mlp;
    cudaStream_t st = ctx->stream;
    if (bcc::mlp_train_grads(static_cast<const uint16_t*>(d_x_bf16), d_labels, rows, m.images.as<uint8_t>(),
                             m.params.as<float>(), m.grads.as<float>(), sm_count(ctx->device), st) != cudaSuccess)
        return mlp_fail(ctx, BCC_ERR_CUDA, "MLP training kernel launch failed");
    // loss and error behind the gradients: one copy, one wait
    const size_t first = h_grads ? 0 : bcc::kMlpParams;
    if (!to_host(ctx, m.grads.as<float>() + first, bcc::kMlpGradBytes - sizeof(float) * first, st)) return BCC_ERR_CUDA;
    const float* tail = m.host + (bcc::kMlpParams - first);
    int flag = 0;
    std::memcpy(&flag, tail + 1, sizeof(int));
    if (flag) return mlp_fail(ctx, BCC_ERR_TIMEOUT, "MLP training kernel wait timed out");
    if (h_grads) std::memcpy(h_grads, m.host, sizeof(float) * bcc::kMlpParams);
    if (h_loss) *h_loss = *tail;
    return BCC_OK;
}

// One optimisation step: gradients of the batch, Adam update (lr) and the BF16
// copies, queued together; the host waits once, for the loss.
bcc_status bcc_mlp_train_step(bcc_ctx* ctx, const void* d_x_bf16, const uint8_t* d_labels, int32_t rows, float lr,
                              float* h_loss) {
    if (!ctx || !ctx->mlp.ready) return mlp_fail(ctx, BCC_ERR_INVALID_ARGUMENT, "MLP parameters not set");
    if (rows < 0 || (rows > 0 && (!d_x_bf16 || !d_labels))) return BCC_ERR_INVALID_ARGUMENT;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return BCC_ERR_CUDA;
    bcc::MlpState& m = ctx->mlp;
    cudaStream_t st = ctx->stream;
    if (bcc::mlp_train_grads(static_cast<const uint16_t*>(d_x_bf16), d_labels, rows, m.images.as<uint8_t>(),
                             m.params.as<float>(), m.grads.as<float>(), sm_count(ctx->device), st) != cudaSuccess)
        return mlp_fail(ctx, BCC_ERR_CUDA, "MLP training kernel launch failed");
    if (bcc::mlp_adam(m.params.as<float>(), m.grads.as<float>(), m.adam_m.as<float>(), m.adam_v.as<float>(),
                      m.images.as<uint8_t>(), m.step + 1, lr, st) != cudaSuccess ||
        !to_host(ctx, m.grads.as<float>() + bcc::kMlpParams, 2 * sizeof(float), st))
        return mlp_fail(ctx, BCC_ERR_CUDA, "MLP update failed");
    int flag = 0;
    std::memcpy(&flag, m.host + 1, sizeof(int));
    if (flag) return mlp_fail(ctx, BCC_ERR_TIMEOUT, "MLP training kernel wait timed out");
    m.step += 1;
    if (h_loss) *h_loss = m.host[0];
    return BCC_OK;
}

}  // extern "C"
