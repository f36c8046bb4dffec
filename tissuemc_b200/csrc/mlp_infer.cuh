// Fused inference of the surrogate ensemble: one persistent kernel runs every member's five layers
// (64 -> 512 -> 512 -> 512 -> 512 -> 128, GELU between) for tiles of 128 queries and applies the
// disagreement gate, without writing an activation to global memory.
//
// Per CTA (one per SM, 20 warps, two of them idle: registers move between groups of four):
//   warp 0             producer: streams the members' weights, pre-packed in the order they are
//                      consumed (tmc_b200_nn_pack), through three 32 KB shared-memory stages with
//                      bulk copies (cp.async.bulk, completion counted on the stage's mbarrier);
//   warp 1             tensor-core issuer: for each layer, tcgen05.mma of the 128 x K activation
//                      tile (shared memory) by each weight tile into the TMEM accumulator (128 lanes x
//                      up to 512 FP32 columns), in two halves of 256 columns, committing each stage
//                      back to the producer and each finished half to the epilogue;
//   warps 4-19         epilogue: read the accumulator with tcgen05.ld (warp w owns TMEM lanes
//                      32 (w % 4) .. + 31, i.e. query rows, and a quarter of each half's columns),
//                      add the bias, apply GELU, and write the BF16 activations back into the
//                      activation tile in the 128-byte-swizzled K-major layout the next layer's MMA
//                      reads; after the output layer they de-normalise, accumulate the members'
//                      mean, sum each member's R_d on the grid (sum of 10^y * annulus area) and
//                      finally write the mean outputs, the mean R_d, the spread (sample standard
//                      deviation over the mean) and the route flag. They also encode the raw features
//                      (z-score, BF16, zero padding to 64) into the activation tile before each member.
//
// The tensor pipe bounds the kernel (a 128 x 512 x 512 layer is 8,192 cycles of it), the epilogue
// comes next (65,536 tanh on 16 SFU lanes a cycle: 4,096 cycles), and there is room for one
// activation tile (128 KB) and one accumulator (all of TMEM), so the two are overlapped by halves:
// while the second half of a layer's columns is multiplied, the epilogue turns the first half into
// activations and leaves them, packed, in the accumulator columns they came from; when the second
// half is done, nothing reads the activation tile any more, the first half moves there, and the next
// layer starts on it, chunk by chunk (64 columns of its K range), while the epilogue works on the
// second half. Measured against the two taking turns (and
// with an issuer whose branch on the lane number cost 850 cycles per 64-wide K slice of 512 tensor
// cycles): 131,072 queries of four members 1,500 -> 759 us, 619 -> 1,223 TFLOP/s of padded layers.
//
// A single tile's members would follow one another on one SM. With few tiles (SPLIT) a cluster of
// as many CTAs as members takes each tile, one member per CTA; each CTA leaves its member's outputs
// in its shared memory and every CTA sums a share of the rows over the members, in member order,
// through distributed shared memory: the same sums in the same order (100 queries of four members:
// 36 us against 210 us before both changes).
//
// Hand-offs are mbarriers: full[s] / empty[s] between producer and issuer, acc_full[h] (issuer ->
// epilogue, one phase per half), act_ready[c] (epilogue -> issuer, one arrival per warp: chunk c of
// the activation tile is written and the accumulator columns that the chunk lets the issuer overwrite
// are read), rdx (the warps holding R_d
// bins 32-63 hand their partial sums to those holding bins 0-31, once per member) and, with SPLIT,
// xch / xch_done (the members' outputs of a tile are in place / have been read). Every wait is
// bounded: a wait that gives up raises the device status word and a shared abort flag, every role
// leaves its loop (warp-uniformly), the producer waits (bounded) for its copies in flight, the issuer
// for its MMAs in flight, and the CTA frees its TMEM and returns (after the cluster's other CTAs).
#pragma once

#include <cuda_bf16.h>

#include "umma.cuh"

namespace tmc {

constexpr int kInferThreads = 640;        // 20 warps: producer, issuer, two idle, 16 of the epilogue
// Registers per thread after the split (setmaxnreg): 128 x 32 + 512 x 112 = 61,440 = 640 x 96, what the
// block is launched with.
constexpr int kInferFrontRegs = 32, kInferEpiRegs = 112;
static_assert(128 * kInferFrontRegs + 512 * kInferEpiRegs <= 640 * 96, "the split cannot exceed the launch's registers");
constexpr int kInferStages = 3;
constexpr int kInferStageBytes = 32768;   // 256 rows x 64 bf16
constexpr int kInferChunkBytes = 16384;   // 128 rows x 64 bf16
constexpr int kInferLayers = 5;
constexpr int kInferHidden = 512, kInferIn = 64, kInferOut = 128;
constexpr int kInferBiasPerMember = 4 * kInferHidden + kInferOut;  // 2176
// tiles per member in stream order: layer 0 (2 halves x 1 K chunk), layers 1-3 (2 x 8), layer 4 (1 x 8)
constexpr int kInferTilesPerMember = 2 + 3 * 16 + 8;
constexpr int kInferBigTiles = 2 + 3 * 16;  // 32 KB each; the last 8 are 16 KB
constexpr uint32_t kInferMemberBytes = kInferBigTiles * 32768u + 8u * 16384u;  // 1,769,472
constexpr int kInferMaxMembers = 8;
constexpr uint32_t kInferWaitLimit = 1u << 24;

struct InferSmem {
    static constexpr int a = 0;                                          // 8 chunks x 16 KB
    static constexpr int stages = a + 8 * kInferChunkBytes;              // 131072
    static constexpr int rdx = stages + kInferStages * kInferStageBytes; // 229376: 2 x 128 floats
    static constexpr int bars = rdx + 2 * 128 * 4;                       // 230400: 20 mbarriers
    static constexpr int tmem_slot = bars + 20 * 8;
    static constexpr int abort_flag = tmem_slot + 4;
    static constexpr int bytes = abort_flag + 4 + 1024;  // + alignment slack
};

struct InferParams {
    const unsigned char *packed;  // members x kInferMemberBytes
    const float *bias;            // members x 2176: b0[512] b1[512] b2[512] b3[512] b4[128]
    const float *feats;           // n x n_feat raw features
    const float *x_mean, *x_std;  // n_feat
    const float *y_mean, *y_std;  // n_out
    const float *areas;           // nbins
    float *out;                   // n x n_out, optional
    float *rd_mean, *spread;      // n, optional
    unsigned char *route;         // n, optional
    int n, n_feat, n_out, nbins, members;
    float threshold;
    int *status;
};

// ------------------------------------------------------------------------------ weight packing
// Packed tile (rows x 64 bf16 of W[row0 + r][k0 + k]): byte r * 128 + ((k / 8) ^ (r % 8)) * 16 + (k % 8) * 2.
struct PackParams {
    const __nv_bfloat16 *w[kInferMaxMembers * kInferLayers];  // per member: 512x64, 512x512 x3, 128x512
    int members;
};

__global__ void pack_kernel(const __grid_constant__ PackParams P, unsigned char *__restrict__ packed) {
    const size_t units_per_member = kInferMemberBytes / 16;
    const size_t u = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (u >= units_per_member * P.members) return;
    const int m = static_cast<int>(u / units_per_member);
    uint32_t off = static_cast<uint32_t>(u % units_per_member) * 16u;  // byte offset inside the member
    // locate the tile
    int layer, half, kc;
    uint32_t in_tile;
    if (off < 2u * 32768u) {
        layer = 0;
        half = static_cast<int>(off / 32768u);
        kc = 0;
        in_tile = off % 32768u;
    } else if (off < static_cast<uint32_t>(kInferBigTiles) * 32768u) {
        const uint32_t t = (off - 2u * 32768u) / 32768u;  // 0..47
        layer = 1 + static_cast<int>(t / 16u);
        half = static_cast<int>((t % 16u) / 8u);
        kc = static_cast<int>(t % 8u);
        in_tile = (off - 2u * 32768u) % 32768u;
    } else {
        const uint32_t o = off - static_cast<uint32_t>(kInferBigTiles) * 32768u;
        layer = 4;
        half = 0;
        kc = static_cast<int>(o / 16384u);
        in_tile = o % 16384u;
    }
    const int r = static_cast<int>(in_tile / 128u);
    const int unit = static_cast<int>((in_tile % 128u) / 16u) ^ (r & 7);  // logical 8-element group
    const int K = layer == 0 ? kInferIn : kInferHidden;
    const __nv_bfloat16 *W = P.w[m * kInferLayers + layer];
    const uint4 v = *reinterpret_cast<const uint4 *>(W + static_cast<size_t>(half * 256 + r) * K + kc * 64 + unit * 8);
    *reinterpret_cast<uint4 *>(packed + static_cast<size_t>(m) * kInferMemberBytes + off) = v;
}

// ------------------------------------------------------------------------------ the fused kernel
__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}

// Byte address of columns [c, c + 8) of row r in the swizzled activation tile (c a multiple of 8).
__device__ __forceinline__ unsigned char *act_unit(unsigned char *A, int r, int c) {
    return A + (c >> 6) * kInferChunkBytes + r * 128 + ((((c & 63) >> 3) ^ (r & 7)) << 4);
}

// The abort flag is looked at only while the wait has to wait.
__device__ __forceinline__ bool infer_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int *status) {
    if (mbar_wait(bar, parity, 1)) return true;
    for (uint32_t i = 0; i < kInferWaitLimit / 64; ++i) {
        if (mbar_wait(bar, parity, 64)) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    atomicExch(status, 1);
    return false;
}

// Columns [16 part, 16 part + 16) of row (row0 + r) of the raw features as network inputs: z-scored,
// BF16, zero beyond the features (512 epilogue threads: r = et / 4, part = et % 4).
__device__ __forceinline__ void infer_encode(const InferParams &P, int row0, int et, uint4 (&u)[2]) {
    const int g = row0 + (et >> 2), c_first = (et & 3) * 16;
    u[0] = u[1] = make_uint4(0u, 0u, 0u, 0u);
    if (g >= P.n || c_first >= P.n_feat) return;
    const float *f = P.feats + static_cast<size_t>(g) * P.n_feat;
    float v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int c = c_first + i;
        v[i] = c < P.n_feat ? (__ldg(f + c) - __ldg(P.x_mean + c)) / __ldg(P.x_std + c) : 0.0f;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
        u[h] = make_uint4(pack_bf16x2(v[8 * h], v[8 * h + 1]), pack_bf16x2(v[8 * h + 2], v[8 * h + 3]),
                          pack_bf16x2(v[8 * h + 4], v[8 * h + 5]), pack_bf16x2(v[8 * h + 6], v[8 * h + 7]));
}

// One arrival of a warp that has written its part of an activation chunk and read its accumulator.
__device__ __forceinline__ void epi_release(uint64_t *bar) {
    fence_async_smem();  // activation writes visible to the tensor core's async proxy
    tc_fence_before();   // accumulator reads ordered before the hand-off
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

// This warp's 16 columns of each of a half's four chunks (accumulator columns taddr + 64 i, biases
// b4 + 16 i), plus their biases, through GELU into eight packed BF16 pairs: put(i, pairs). The next
// biases are on their way while one set is worked on (from L2, since shared memory is full: waiting for
// them took a fifth of the epilogue); the other warps' work covers the accumulator's shorter latency.
template <class Put> __device__ __forceinline__ void infer_hidden(uint32_t taddr, const float4 *b4, const float4 (&first)[4], Put put) {
    float4 bb[2][4];
#pragma unroll
    for (int k = 0; k < 4; ++k) bb[0][k] = first[k];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t v[16];
        tmem_ld16_async(taddr + 64u * i, v);
        if (i < 3) {
#pragma unroll
            for (int k = 0; k < 4; ++k) bb[(i + 1) & 1][k] = __ldg(b4 + 16 * (i + 1) + k);  // one address across the warp
        }
        tmem_ld_wait16(v);
        const auto x = [&](int c) { return __uint_as_float(v[c]); };
        uint32_t w[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float4 b = bb[i & 1][k];
            const float2 p = gelu_tanh2(__fadd2_rn(make_float2(x(4 * k), x(4 * k + 1)), make_float2(b.x, b.y)));
            const float2 q = gelu_tanh2(__fadd2_rn(make_float2(x(4 * k + 2), x(4 * k + 3)), make_float2(b.z, b.w)));
            w[2 * k] = pack_bf16x2(p.x, p.y);
            w[2 * k + 1] = pack_bf16x2(q.x, q.y);
        }
        put(i, w);
    }
}

// SPLIT: a cluster of P.members CTAs per tile, one member each; otherwise a CTA runs every member.
template <bool SPLIT>
__global__ void __launch_bounds__(kInferThreads, 1) ensemble_infer_kernel(const __grid_constant__ InferParams P) {
    extern __shared__ unsigned char ism_raw[];
    unsigned char *base = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(ism_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    unsigned char *A = base + InferSmem::a;
    unsigned char *stages = base + InferSmem::stages;
    float *rdx = reinterpret_cast<float *>(base + InferSmem::rdx);
    uint64_t *bars = reinterpret_cast<uint64_t *>(base + InferSmem::bars);
    uint64_t *full = bars, *empty = bars + kInferStages, *acc_full = bars + 6, *act_ready = bars + 8;
    uint64_t *rdx_bar = bars + 16, *drain = bars + 17, *xch = bars + 18, *xch_done = bars + 19;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(base + InferSmem::tmem_slot);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(base + InferSmem::abort_flag);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles = (P.n + 127) / 128;
    // this CTA's tiles and members
    const int rank = SPLIT ? static_cast<int>(cluster_rank()) : 0;
    const int tile0 = SPLIT ? static_cast<int>(blockIdx.x) / P.members : static_cast<int>(blockIdx.x);
    const int tile_step = SPLIT ? static_cast<int>(gridDim.x) / P.members : static_cast<int>(gridDim.x);
    const int m_first = SPLIT ? rank : 0, m_end = SPLIT ? rank + 1 : P.members;
    if (warp == 1) tmem_alloc(tmem_slot, 512);
    if (threadIdx.x == 0) {
        for (int s = 0; s < kInferStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int h = 0; h < 2; ++h) mbar_init(&acc_full[h], 1);
        for (int c = 0; c < 8; ++c) mbar_init(&act_ready[c], 16);
        mbar_init(rdx_bar, 128);
        mbar_init(drain, 1);
        mbar_init(xch, 16 * P.members);
        mbar_init(xch_done, 16 * P.members);
        *abort_flag = 0;
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (SPLIT) cluster_barrier();  // every CTA's barriers exist before a peer arrives on them
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp < 4) {
        reg_shrink<kInferFrontRegs>();
        if (warp == 0) {
            // ---------------------------------------------------------------- producer (whole warp, one lane issues)
            uint32_t it = 0, s = 0, parity = 1u;  // the parity of a stage's last hand-back
            bool ok = true;
            for (int t = tile0; ok && t < tiles; t += tile_step) {
                for (int m = m_first; ok && m < m_end; ++m) {
                    const unsigned char *src = P.packed + static_cast<size_t>(m) * kInferMemberBytes;
                    for (int i = 0; i < kInferTilesPerMember; ++i, ++it) {
                        const uint32_t bytes = i < kInferBigTiles ? 32768u : 16384u;
                        if (it >= static_cast<uint32_t>(kInferStages) &&
                            !__all_sync(0xffffffffu, infer_wait(&empty[s], parity, abort_flag, P.status))) {
                            ok = false;
                            break;
                        }
                        if (elect_one()) {
                            mbar_arrive_expect_tx(&full[s], bytes);
                            bulk_g2s(stages + s * kInferStageBytes, src, bytes, &full[s]);
                        }
                        src += bytes;
                        if (++s == static_cast<uint32_t>(kInferStages)) {
                            s = 0;
                            parity ^= 1u;
                        }
                    }
                }
            }
            // copies still in flight when a wait gave up: wait (bounded) until they have landed
            if (!ok) {
                const uint32_t first = it > static_cast<uint32_t>(kInferStages) ? it - kInferStages : 0u;
                for (uint32_t j = first; j < it; ++j)
                    mbar_wait(&full[j % kInferStages], (j / kInferStages) & 1u, kInferWaitLimit);
            }
            __syncwarp();
        } else if (warp == 1) {
            // ---------------------------------------------------------------- tensor-core issuer (one lane)
            if (elect_one()) {
                const auto wait = [&](uint64_t *bar, uint32_t parity) {
                    const bool done = infer_wait(bar, parity, abort_flag, P.status);
                    tc_fence_after();
                    return done;
                };
                const uint64_t a_desc = umma_desc_sw128(smem_u32(A)), b_desc = umma_desc_sw128(smem_u32(stages));
                uint32_t s = 0, full_parity = 0u, inputs = 0, layers = 0;  // phases of act_ready[0] and of the others
                // one K chunk of a layer's half: its weights have landed, four MMAs, hand the stage back
                const auto chunk = [&](int h, int kc, uint32_t idesc) {
                    if (!wait(&full[s], full_parity)) return false;
                    umma_bf16_k64(tmem + static_cast<uint32_t>(h * 256), a_desc + static_cast<uint32_t>(kc * (kInferChunkBytes >> 4)),
                                  b_desc + s * (kInferStageBytes >> 4), idesc, kc > 0 ? 1u : 0u);
                    umma_commit(&empty[s]);
                    if (++s == static_cast<uint32_t>(kInferStages)) {
                        s = 0;
                        full_parity ^= 1u;
                    }
                    return true;
                };
                bool ok = true;
                for (int t = tile0; ok && t < tiles; t += tile_step) {
                    for (int m = m_first; ok && m < m_end; ++m) {
                        // layer 0: one K chunk
                        const uint32_t wide = umma_idesc_bf16(128, 256);
                        ok = wait(&act_ready[0], inputs++ & 1u) && chunk(0, 0, wide);
                        if (ok) umma_commit(&acc_full[0]);
                        ok = ok && chunk(1, 0, wide);
                        if (ok) umma_commit(&acc_full[1]);
                        for (int l = 1; ok && l < kInferLayers; ++l, ++layers) {
                            const uint32_t idesc = l == 4 ? umma_idesc_bf16(128, 128) : wide;
                            // the first half's columns follow the epilogue chunk by chunk; when the last
                            // chunk is ready the accumulator's second half has been read too
                            ok = wait(&act_ready[0], inputs++ & 1u) && chunk(0, 0, idesc);
#pragma unroll
                            for (int kc = 1; kc < 8; ++kc) ok = ok && wait(&act_ready[kc], layers & 1u) && chunk(0, kc, idesc);
                            if (ok) umma_commit(&acc_full[0]);
                            if (l == 4) continue;
#pragma unroll
                            for (int kc = 0; kc < 8; ++kc) ok = ok && chunk(1, kc, idesc);
                            if (ok) umma_commit(&acc_full[1]);
                        }
                    }
                }
                if (!ok) {  // let the MMAs already issued finish before the tile memory goes away
                    umma_commit(drain);
                    mbar_wait(drain, 0u, kInferWaitLimit);
                }
            }
            __syncwarp();
        }
    } else {
        reg_grow<kInferEpiRegs>();
        // ---------------------------------------------------------------- epilogue (512 threads)
        const int et = threadIdx.x - 128;
        const int q = warp & 3;            // TMEM lane quarter this warp may read
        const int j = (warp - 4) >> 2;     // column quarter (of each half of a hidden layer)
        const int r = q * 32 + lane;       // query row inside the tile
        const uint32_t lane_addr = tmem + (static_cast<uint32_t>(q * 32) << 16);
        uint32_t full0 = 0, full1 = 0;     // phases of acc_full[0] (every layer) and [1] (hidden layers)
        uint32_t member_no = 0, tile_no = 0;
        bool ok = true;
        // the decision to go on is warp-uniform: tcgen05.ld is a warp-collective
        const auto wait = [&](uint64_t *bar, uint32_t parity) {
            return __all_sync(0xffffffffu, infer_wait(bar, parity, abort_flag, P.status)) != 0;
        };
        int t = tile0;
        uint4 enc[2] = {};  // this thread's 16 columns of the tile's encoded inputs, written before every member
        const auto put_inputs = [&]() {
            *reinterpret_cast<uint4 *>(act_unit(A, et >> 2, (et & 3) * 16)) = enc[0];
            *reinterpret_cast<uint4 *>(act_unit(A, et >> 2, (et & 3) * 16 + 8)) = enc[1];
            epi_release(&act_ready[0]);
        };
        if (t < tiles) {
            infer_encode(P, t * 128, et, enc);
            put_inputs();
        }
        // lane i holds the output constants of column 32 j + i
        const int oc = j * 32 + lane;
        const float o_std = oc < P.n_out ? __ldg(P.y_std + oc) : 0.0f, o_mean = oc < P.n_out ? __ldg(P.y_mean + oc) : 0.0f;
        const float o_area = oc < P.nbins ? __ldg(P.areas + oc) : 0.0f;
        const int n_cols = min(32, P.n_out - j * 32), n_bins = min(32, P.nbins - j * 32);  // of this warp's 32
        for (; ok && t < tiles; t += tile_step, ++tile_no) {
            float acc[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[i] = 0.0f;
            float s1 = 0.0f, s2 = 0.0f;  // members' R_d on the grid: sum and sum of squares
            for (int m = m_first; ok && m < m_end; ++m) {
                const float *bias = P.bias + static_cast<size_t>(m) * kInferBiasPerMember;
                for (int l = 0; l < kInferLayers - 1; ++l) {
                    // hidden layer: this warp has columns 16 j .. + 15 of each 64-column chunk
                    const float4 *b4 = reinterpret_cast<const float4 *>(bias + l * kInferHidden + j * 16);
                    const uint32_t d0 = lane_addr + static_cast<uint32_t>(j * 16), d1 = d0 + 256u;
                    const auto put_act = [&](int c, const uint32_t (&w)[8]) {
                        *reinterpret_cast<uint4 *>(act_unit(A, r, c * 64 + j * 16)) = make_uint4(w[0], w[1], w[2], w[3]);
                        *reinterpret_cast<uint4 *>(act_unit(A, r, c * 64 + j * 16 + 8)) = make_uint4(w[4], w[5], w[6], w[7]);
                        epi_release(&act_ready[c]);
                    };
                    float4 b_first[4];  // fetched while the products run
#pragma unroll
                    for (int k = 0; k < 4; ++k) b_first[k] = __ldg(b4 + k);
                    if (!wait(&acc_full[0], full0++ & 1u)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    infer_hidden(d0, b4, b_first, [&](int i, const uint32_t (&w)[8]) { tmem_st8(d0 + 64u * i, w); });
#pragma unroll
                    for (int k = 0; k < 4; ++k) b_first[k] = __ldg(b4 + 64 + k);
                    tmem_st_wait();
                    if (!wait(&acc_full[1], full1++ & 1u)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    if constexpr (SPLIT) {
                        // the last tile's outputs (in this tile's place) have been read by every CTA
                        if (l == 0 && tile_no > 0 &&
                            !__all_sync(0xffffffffu, mbar_wait_cluster(xch_done, (tile_no - 1u) & 1u, kInferWaitLimit))) {
                            *abort_flag = 1;
                            atomicExch(P.status, 1);
                            ok = false;
                            break;
                        }
                    }
                    {
                        uint32_t w[4][8];
#pragma unroll
                        for (int i = 0; i < 4; ++i) tmem_ld8_async(d0 + 64u * i, w[i]);
#pragma unroll
                        for (int i = 0; i < 4; ++i) tmem_ld_wait8(w[i]);
#pragma unroll
                        for (int i = 0; i < 4; ++i) put_act(i, w[i]);
                    }
                    infer_hidden(d1, b4 + 64, b_first, [&](int i, const uint32_t (&w)[8]) { put_act(4 + i, w); });
                }
                if (!ok) break;
                // output layer: columns [32 j, 32 j + 32) of 128; its bias, and the inputs of the next
                // member (or tile), are fetched while its products run
                const float o_bias = __ldg(bias + 4 * kInferHidden + oc);
                const bool last_member = m == m_end - 1;
                const int next_t = last_member ? t + tile_step : t;
                if (last_member && next_t < tiles) infer_encode(P, next_t * 128, et, enc);
                if (!wait(&acc_full[0], full0++ & 1u)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                uint32_t v[2][16];
                tmem_ld16_async(lane_addr + static_cast<uint32_t>(j * 32), v[0]);
                tmem_ld16_async(lane_addr + static_cast<uint32_t>(j * 32 + 16), v[1]);
                tmem_ld_wait16(v[0]);
                tmem_ld_wait16(v[1]);
                // this member's MMAs are done and its accumulator is read: hand the next inputs over before
                // working on the outputs
                if (next_t < tiles) put_inputs();
                float rd = 0.0f;
#pragma unroll
                for (int i0 = 0; i0 < 32; i0 += 8) {  // eight columns without a branch between them
                    if (i0 >= n_cols) break;           // warp-uniform
                    float y[8], e[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int c = i0 + i;
                        y[i] = fmaf(__uint_as_float(v[c >> 4][c & 15]) + __shfl_sync(0xffffffffu, o_bias, c),
                                    __shfl_sync(0xffffffffu, o_std, c), __shfl_sync(0xffffffffu, o_mean, c));
                        acc[c] += y[i];
                    }
                    if (i0 >= n_bins) continue;
#pragma unroll
                    for (int i = 0; i < 8; ++i) e[i] = exp10f(y[i]);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float sum = fmaf(e[i], __shfl_sync(0xffffffffu, o_area, i0 + i), rd);
                        rd = i0 + i < n_bins ? sum : rd;
                    }
                }
                // the R_d bins are columns 0..63: quarter 1 hands its partial sums to quarter 0 (two
                // buffers by member parity: a buffer is rewritten two members later, which takes
                // quarter 0's activations of the member in between, written after it has read)
                const uint32_t slot = (member_no & 1u) * 128u + static_cast<uint32_t>(r);
                if (j == 1) {
                    rdx[slot] = rd;
                    mbar_arrive(rdx_bar);
                } else if (j == 0) {
                    if (!wait(rdx_bar, member_no & 1u)) {
                        ok = false;
                        break;
                    }
                    rd += rdx[slot];
                    s1 += rd;
                    s2 = fmaf(rd, rd, s2);
                }
                ++member_no;
            }
            if (!ok) break;
            const float M = static_cast<float>(P.members), inv = 1.0f / M;
            const auto gate = [&](int g, float sum, float squares) {
                const float mean = sum / M;
                const float var = P.members > 1 ? fmaxf(fmaf(-sum, mean, squares), 0.0f) / (M - 1.0f) : 0.0f;
                const float sp = sqrtf(var) / fmaxf(mean, 1e-12f);
                if (P.rd_mean) P.rd_mean[g] = mean;
                if (P.spread) P.spread[g] = sp;
                if (P.route) P.route[g] = sp > P.threshold ? 1 : 0;
            };
            if constexpr (!SPLIT) {
                const int g = t * 128 + r;
                if (g < P.n) {
                    if (P.out) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const int c = j * 32 + i;
                            if (c < P.n_out) P.out[static_cast<size_t>(g) * P.n_out + c] = acc[i] * inv;
                        }
                    }
                    if (j == 0) gate(g, s1, s2);
                }
            } else {
                // this member's outputs (row-major, at most 64 KB) and R_d, in activation chunks 1-5: free
                // until the next tile's first hidden layer is written
                float *ys = reinterpret_cast<float *>(A + kInferChunkBytes);
                float *rds = reinterpret_cast<float *>(A + 5 * kInferChunkBytes);
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (j * 32 + i < P.n_out) ys[r * P.n_out + j * 32 + i] = acc[i];
                if (j == 0) rds[r] = s1;
                __syncwarp();
                for (uint32_t c = lane; c < static_cast<uint32_t>(P.members); c += 32) mbar_arrive_cluster(xch, c);
                if (!__all_sync(0xffffffffu, mbar_wait_cluster(xch, tile_no & 1u, kInferWaitLimit))) {
                    *abort_flag = 1;
                    atomicExch(P.status, 1);
                    ok = false;
                    break;
                }
                // this CTA's share of the rows, summed over the members in member order
                const int share = (128 + P.members - 1) / P.members;
                const int row0 = rank * share;
                const int rows = min(min(share, 128 - row0), P.n - t * 128 - row0);
                if (P.out) {
                    float *out = P.out + static_cast<size_t>(t * 128 + row0) * P.n_out;
                    for (int e = et; e < rows * P.n_out; e += 512) {
                        float y = 0.0f;
                        for (int c = 0; c < P.members; ++c) y += ld_cluster_f32(ys + row0 * P.n_out + e, static_cast<uint32_t>(c));
                        out[e] = y * inv;
                    }
                }
                if (et < rows) {
                    float sum = 0.0f, squares = 0.0f;
                    for (int c = 0; c < P.members; ++c) {
                        const float rd = ld_cluster_f32(rds + row0 + et, static_cast<uint32_t>(c));
                        sum += rd;
                        squares = fmaf(rd, rd, squares);
                    }
                    gate(t * 128 + row0 + et, sum, squares);
                }
                __syncwarp();
                for (uint32_t c = lane; c < static_cast<uint32_t>(P.members); c += 32) mbar_arrive_cluster(xch_done, c);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
    if constexpr (SPLIT) {
        __syncwarp();
        cluster_barrier();  // no CTA leaves while a peer may still read its shared memory or arrive on it
    }
}

}  // namespace tmc
