// D = A * B^T on the 5th-generation tensor cores (tcgen05), BF16 operands, FP32 accumulation in
// tensor memory, with a fused epilogue. A is M x K and B is N x K, both row-major with K
// contiguous (K-major), 16-byte aligned; K is a multiple of 64. One CTA of eight warps computes a
// 128 x BN tile over the K range of its blockIdx.z (split-K: each z covers K / gridDim.z, a
// multiple of 64):
//
//   warp 0 (the producer) streams 64-wide K slices of A and B into a ring of kGemmStages
//   shared-memory stages with tiled TMA loads (cp.async.bulk.tensor, 128-byte swizzle: the layout
//   the MMA descriptors read, umma.cuh), each stage's mbarrier counting the bytes in; warp 1 (the
//   issuer) waits for a stage, issues its four tcgen05.mma (K = 16 each) into the TMEM accumulator
//   and commits them to the stage's "empty" mbarrier, which hands the stage back to the producer;
//   a last commit marks the accumulator complete. Rows past M or N arrive as zeros. Every wait is
//   bounded: one that runs out records an error in *status (the host discards the results) and
//   the CTA skips its epilogue. Nothing is released while this CTA's own asynchronous work may
//   still be in flight: the issuer commits the accumulator barrier after whatever MMAs it issued
//   (also when it gave up), every warp waits for that barrier before TMEM is read or freed, and
//   the producer waits for every load it issued; these drain waits have a longer limit of their
//   own (issued copies and MMAs finish without help from any other party). Only if a drain wait
//   runs out too does the CTA free TMEM regardless (so that a later CTA can allocate it) and
//   report status 2.
//   The epilogue reads the accumulator with tcgen05.ld, 32 columns per load: warp w owns TMEM lanes
//   32 (w % 4) .. + 31, i.e. output rows, and half w / 4 of the columns. A lane then holds one row,
//   so storing straight from its registers would touch 32 rows per instruction (it made a
//   4096 x 512 x 512 layer 18.3 us instead of 10.1). The warp therefore stages each 32 x 32 piece in its 8 KB
//   of the finished operand ring (16-byte units, swizzled: no bank conflicts) and moves it between
//   shared and global memory in whole rows of 64 or 128 bytes (EpiTile in mlp.cu).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include "umma.cuh"

namespace tmc {

constexpr int kGemmBM = 128, kGemmBK = 64, kGemmThreads = 256, kGemmStages = 3;
constexpr int kGemmWarpStage = 8192;            // bytes of the ring one warp's epilogue stages through
constexpr uint32_t kGemmWaitLimit = 1u << 24;   // mbarrier polls before a wait gives up
constexpr uint32_t kGemmDrainLimit = 1u << 26;  // polls of a wait for this CTA's own issued work

template <int BN> struct GemmSmem {
    static constexpr int a_bytes = kGemmBM * 128;  // 128 rows x 64 bf16
    static constexpr int b_bytes = BN * 128;
    static constexpr int stage_bytes = a_bytes + b_bytes;
    // alignment slack, the stages, then 2 x kGemmStages + 1 mbarriers, the TMEM address and the
    // CTA's abort flag (128 bytes), and the bias of the tile's columns
    static constexpr int bytes = 1024 + kGemmStages * stage_bytes + 128 + BN * 4;
};

// One CTA's shared memory and accumulator.
template <int BN> struct GemmCta {
    unsigned char *base;  // the ring, 1024-byte aligned
    uint64_t *full, *empty, *acc_bar;
    volatile int *abort_flag;
    float *sbias;
    uint32_t tmem_d;
};

// A whole warp's bounded wait: true when every lane saw the phase complete. Lanes poll, and give up, at their
// own times; the warp goes on, or gives up, as one (its next elect.sync names all 32 lanes).
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, uint32_t limit) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, limit)) != 0;
}

// Barriers, TMEM and the bias of columns n0 .. (zeros past N or without one). Whole CTA.
template <int BN>
__device__ __forceinline__ GemmCta<BN> gemm_begin(unsigned char *raw, const float *bias, int n0, int N) {
    static_assert(GemmSmem<BN>::a_bytes % 1024 == 0 && GemmSmem<BN>::b_bytes % 1024 == 0, "1024-byte tiles");
    GemmCta<BN> g;
    g.base = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~static_cast<uintptr_t>(1023));
    g.full = reinterpret_cast<uint64_t *>(g.base + kGemmStages * GemmSmem<BN>::stage_bytes);
    g.empty = g.full + kGemmStages;
    g.acc_bar = g.empty + kGemmStages;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(g.acc_bar + 1);
    g.abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    g.sbias = reinterpret_cast<float *>(g.base + kGemmStages * GemmSmem<BN>::stage_bytes + 128);
    if (threadIdx.x < 32) tmem_alloc(tmem_slot, BN);
    if (threadIdx.x == 0) {
        for (int s = 0; s < kGemmStages; ++s) {
            mbar_init(&g.full[s], 1);
            mbar_init(&g.empty[s], 1);
        }
        mbar_init(g.acc_bar, 1);
        *g.abort_flag = 0;
    }
    wait_for_inputs();
    for (int i = threadIdx.x; i < BN; i += kGemmThreads) g.sbias[i] = bias && n0 + i < N ? bias[n0 + i] : 0.0f;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    g.tmem_d = *tmem_slot;
    return g;
}

// The products of K slices kt0 .. kt0 + kt_n - 1 of the tile at (m0, n0): warp 0 loads, warp 1 issues, the
// other warps pass through.
template <int BN>
__device__ __forceinline__ void gemm_products(const GemmCta<BN> &g, const CUtensorMap *tma_a, const CUtensorMap *tma_b,
                                              int m0, int n0, int kt0, int kt_n, int *status, uint32_t wait_limit,
                                              int withhold) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr uint32_t idesc = umma_idesc_bf16(kGemmBM, BN);
    bool ok = true;
    if (warp == 0) {
        // ---- producer: the whole warp walks the ring, one lane issues
        int issued = 0;
        for (int kt = 0; kt < (withhold ? 0 : kt_n); ++kt) {
            const int s = kt % kGemmStages;
            // the stage was last read by the MMAs of slice kt - kGemmStages
            if (kt >= kGemmStages &&
                !warp_wait(&g.empty[s], static_cast<uint32_t>((kt / kGemmStages - 1) & 1), wait_limit)) {
                ok = false;
                break;
            }
            if (elect_one()) {
                unsigned char *sa = g.base + s * GemmSmem<BN>::stage_bytes;
                mbar_arrive_expect_tx(&g.full[s], GemmSmem<BN>::stage_bytes);
                tma_load_2d(sa, tma_a, (kt0 + kt) * kGemmBK, m0, &g.full[s]);
                tma_load_2d(sa + GemmSmem<BN>::a_bytes, tma_b, (kt0 + kt) * kGemmBK, n0, &g.full[s]);
            }
            __syncwarp();
            issued = kt + 1;
        }
        // every load issued has landed before the CTA can end (the last phase of each stage)
        for (int kt = issued > kGemmStages ? issued - kGemmStages : 0; kt < issued; ++kt)
            if (!warp_wait(&g.full[kt % kGemmStages], static_cast<uint32_t>((kt / kGemmStages) & 1), kGemmDrainLimit)) {
                ok = false;
                if (lane == 0) atomicExch(status, 2);
            }
    } else if (warp == 1) {
        // ---- issuer: the whole warp waits, one lane issues the MMAs and the commits
        for (int kt = 0; kt < kt_n; ++kt) {
            const int s = kt % kGemmStages;
            if (!warp_wait(&g.full[s], static_cast<uint32_t>((kt / kGemmStages) & 1), wait_limit)) {
                ok = false;
                break;
            }
            tc_fence_after();
            if (elect_one()) {
                const uint32_t a0 = smem_u32(g.base + s * GemmSmem<BN>::stage_bytes);
                umma_bf16_k64(g.tmem_d, umma_desc_sw128(a0), umma_desc_sw128(a0 + GemmSmem<BN>::a_bytes), idesc,
                              kt > 0 ? 1u : 0u);
                umma_commit(&g.empty[s]);
            }
            __syncwarp();
        }
        // arrives when every MMA issued above has completed, also after a give-up
        if (elect_one()) umma_commit(g.acc_bar);
        __syncwarp();
    }
    if (!ok) {
        if (lane == 0) atomicCAS(status, 0, 1);
        *g.abort_flag = 1;
    }
}

// Whole CTA: every MMA issued has completed (before TMEM is read or released); false when a wait gave up.
template <int BN> __device__ __forceinline__ bool gemm_done(const GemmCta<BN> &g, int *status, uint32_t wait_limit) {
    const int lane = threadIdx.x & 31;
    if (!warp_wait(g.acc_bar, 0u, wait_limit)) {
        if (lane == 0) atomicCAS(status, 0, 1);
        *g.abort_flag = 1;
        if (!warp_wait(g.acc_bar, 0u, kGemmDrainLimit) && lane == 0) atomicExch(status, 2);
    }
    tc_fence_after();
    __syncthreads();  // orders the abort flag: the epilogue runs in every warp or none
    return *g.abort_flag == 0;
}
template <int BN> __device__ __forceinline__ void gemm_end(const GemmCta<BN> &g) {
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) tmem_dealloc(g.tmem_d, BN);
}

// Epilogue functor interface. `bias` (device pointer or NULL) is added by the functor from the
// tile's copy in shared memory (zeros where there is none). prefetch(row0, col0, regs) starts
// loading what the piece at (row0, col0) needs from global memory; piece(split, row0, col0, v,
// bias, stage, regs) takes 32 consecutive columns of lane's row (row0 + lane) and writes the
// piece's outputs, ignoring rows >= M and columns >= N. Both are called by whole warps.
// wait_limit bounds the waits on the other roles (kGemmWaitLimit in production). withhold = 1 is
// a test of the give-up path: the producer issues no loads, so the issuer's first wait runs out
// with no copy and no MMA outstanding.
template <int BN, class Epi>
__global__ void __launch_bounds__(kGemmThreads, 2) gemm_tc_kernel(const __grid_constant__ CUtensorMap tma_a,
                                                              const __grid_constant__ CUtensorMap tma_b, int M, int N,
                                                              int K, Epi epi, int *status, uint32_t wait_limit,
                                                              int withhold) {
    extern __shared__ unsigned char gsm_raw[];
    const int warp = threadIdx.x >> 5;
    const int m0 = blockIdx.y * kGemmBM, n0 = blockIdx.x * BN;
    const GemmCta<BN> g = gemm_begin<BN>(gsm_raw, epi.bias, n0, N);
    const int kt_n = K / kGemmBK / static_cast<int>(gridDim.z);  // K slices of this split
    gemm_products<BN>(g, &tma_a, &tma_b, m0, n0, static_cast<int>(blockIdx.z) * kt_n, kt_n, status, wait_limit, withhold);
    // the warp's part of the tile: 32 rows, half of the columns
    const int row0 = m0 + (warp & 3) * 32, c_first = (warp >> 2) * (BN / 2);
    typename Epi::Regs regs;
    epi.prefetch(row0, n0 + c_first, regs);
    if (gemm_done<BN>(g, status, wait_limit)) {
        // the ring is free: its last bytes were read by the MMAs that acc_bar waited for
        unsigned char *stage = g.base + warp * kGemmWarpStage;
        static_assert((kGemmThreads / 32) * kGemmWarpStage <= kGemmStages * GemmSmem<BN>::stage_bytes, "staging");
        static_assert(BN % 64 == 0 && kGemmThreads == 256, "eight warps: four row groups x two column halves");
        const uint32_t lane_addr = g.tmem_d + (static_cast<uint32_t>((warp & 3) * 32) << 16);
#pragma unroll 1
        for (int c = c_first; c < c_first + BN / 2; c += 32) {
            float v[32];
            tmem_ld32(lane_addr + static_cast<uint32_t>(c), v);
            if (row0 < M && n0 + c < N) {  // warp-uniform
                epi.piece(static_cast<int>(blockIdx.z), row0, n0 + c, v, g.sbias + c, stage, regs);
                if (c + 32 < c_first + BN / 2) epi.prefetch(row0, n0 + c + 32, regs);
            }
        }
    }
    gemm_end<BN>(g);
}

// ------------------------------------------------------------------------------ weight gradients
// Several products D = A B^T that contract over the same long K (a network's weight gradients, K the
// batch), in one launch: a cluster of `splits` CTAs per 128 x 128 tile, each over its share of K. The CTAs
// leave their float32 partial tiles in shared memory and each sums a share of the rows over the splits, in
// split order, through distributed shared memory (the sums and their order are those of a split-K product
// with its partials in global memory). Bound by the launch and the latency of short products: against one
// product and one summing launch per layer, five layers of a network at batch 4096 in
// 8 splits 43 -> 23.5 us.
constexpr int kWgradMost = 8;
struct WgradProblems {
    CUtensorMap a[kWgradMost], b[kWgradMost];
    float *D[kWgradMost];
    int M[kWgradMost], N[kWgradMost];
    int first[kWgradMost + 1];  // first tile of each problem
    int count;
};

template <int BN>
__global__ void __launch_bounds__(kGemmThreads, 2) wgrad_kernel(const __grid_constant__ WgradProblems P, int K, int splits,
                                                                int *status) {
    extern __shared__ unsigned char gsm_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = static_cast<int>(blockIdx.x) / splits, split = static_cast<int>(cluster_rank());
    int q = 0;
    while (q + 1 < P.count && tile >= P.first[q + 1]) ++q;
    const int M = P.M[q], N = P.N[q], across = (N + BN - 1) / BN;
    const int m0 = (tile - P.first[q]) / across * kGemmBM, n0 = (tile - P.first[q]) % across * BN;
    const GemmCta<BN> g = gemm_begin<BN>(gsm_raw, nullptr, 0, 0);
    const int kt_n = K / kGemmBK / splits;
    gemm_products<BN>(g, &P.a[q], &P.b[q], m0, n0, split * kt_n, kt_n, status, kGemmWaitLimit, 0);
    const bool ok = gemm_done<BN>(g, status, kGemmWaitLimit);
    dependents_may_start();
    // the partial tile in the finished ring: row r at 512 r, its 16-byte unit u at place u ^ (r % 8)
    static_assert(kGemmBM * BN * 4 <= kGemmStages * GemmSmem<BN>::stage_bytes, "the tile fits the ring");
    const auto unit = [&](int r, int u) { return reinterpret_cast<float4 *>(g.base + r * (BN * 4) + ((u ^ (r & 7)) << 4)); };
    if (ok) {
        const int r = (warp & 3) * 32 + lane;
        const uint32_t lane_addr = g.tmem_d + (static_cast<uint32_t>((warp & 3) * 32) << 16);
#pragma unroll 1
        for (int c = (warp >> 2) * (BN / 2); c < (warp >> 2) * (BN / 2) + BN / 2; c += 32) {
            float v[32];
            tmem_ld32(lane_addr + static_cast<uint32_t>(c), v);
#pragma unroll
            for (int u = 0; u < 8; ++u) *unit(r, c / 4 + u) = make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
        }
    }
    __syncwarp();
    cluster_barrier();  // every split's partial tile is in place
    if (ok) {
        const int share = (kGemmBM + splits - 1) / splits, r_end = min(min((split + 1) * share, kGemmBM), M - m0);
        const bool vec = N % 4 == 0 && reinterpret_cast<uintptr_t>(P.D[q]) % 16 == 0;
        for (int i = split * share * (BN / 4) + static_cast<int>(threadIdx.x); i < r_end * (BN / 4); i += kGemmThreads) {
            const int r = i / (BN / 4), u = i % (BN / 4), col = n0 + 4 * u;
            if (col >= N) continue;
            float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            for (int z = 0; z < splits; ++z) {
                const float4 w = ld_cluster_f32x4(unit(r, u), static_cast<uint32_t>(z));
                s.x += w.x;
                s.y += w.y;
                s.z += w.z;
                s.w += w.w;
            }
            float *d = P.D[q] + static_cast<size_t>(m0 + r) * N + col;
            if (vec) {
                *reinterpret_cast<float4 *>(d) = s;
            } else {
                d[0] = s.x;
                if (col + 1 < N) d[1] = s.y;
                if (col + 2 < N) d[2] = s.z;
                if (col + 3 < N) d[3] = s.w;
            }
        }
    }
    __syncwarp();
    cluster_barrier();  // no CTA leaves while another may still read its partial tile
    gemm_end<BN>(g);
}

}  // namespace tmc
