// The surrogate's neural-network kernels and their C ABI (no counterpart in the reference: the
// learned surrogate is an addition of this engine). Every matrix product runs on the tcgen05
// tensor cores through gemm_tc.cuh (BF16 operands, FP32 accumulation in tensor memory) with the
// bias, GELU and GELU-derivative work fused into its epilogue; the element-wise kernels (transpose,
// bias gradient, loss, Adam) are plain CUDA. Entry points take device pointers and a stream and
// do not synchronise (so a training step can be captured in a CUDA graph); a bounded tensor-core
// wait that gives up sets a per-device status word read by tmc_b200_nn_status.

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>
#include <utility>

#include "../../include/tissuemc_b200.h"
#include "gemm_tc.cuh"
#include "mlp_infer.cuh"

namespace tmc {
namespace {

// Columns of a product's tiles (launch_gemm chooses) and of the weight gradients' (the wide ones).
constexpr int kWide = 128, kNarrow = 64;
// three stages of 32 KB plus slack: two CTAs per SM, i.e. 2 x 128 of the 512 TMEM columns
static_assert(2 * GemmSmem<kWide>::bytes <= 227 * 1024, "two GEMM CTAs per SM");

__device__ __forceinline__ float gelu(float x) { return gelu_tanh(x); }
__device__ __forceinline__ float gelu_grad(float x) { return gelu_tanh_grad(x); }

__device__ __forceinline__ uint32_t pack2_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ uint4 pack8_bf16(const float (&x)[8]) {
    return make_uint4(pack2_bf16(x[0], x[1]), pack2_bf16(x[2], x[3]), pack2_bf16(x[4], x[5]), pack2_bf16(x[6], x[7]));
}

// A warp's 32 x 32 piece of an output tile between the lanes' registers (lane = row) and global
// memory, through the warp's staging bytes: the lanes write their rows in 16-byte units, the warp
// then moves whole rows (or, transposed, whole columns). A unit's place is swizzled by its row, so
// neither side meets a bank conflict. `vec`: rows start on 16-byte boundaries and hold whole units,
// else the same piece goes element by element, still a row at a time. Against storing each lane's
// row straight from registers (32 rows per instruction, 16 of every 32-byte sector), launches back to
// back in one graph: a 4096 x 512 x 512 layer with Z, H and its transpose 18.3 -> 10.1 us, the
// backward product 14.9 -> 10.4 us, the split-K weight gradient (8 splits and their sum) 10.8 -> 9.6 us.
struct EpiTile {
    static constexpr int f32_at = 0, b16_at = 4096, tr_at = 6144;  // 4 KB, 2 KB, 2 KB

    // 16-byte unit u (0..7) of row r of the float32 piece, u (0..3) of row r of the bf16 piece
    static __device__ __forceinline__ float4 *f32_unit(unsigned char *st, int r, int u) {
        return reinterpret_cast<float4 *>(st + f32_at + r * 128 + ((u ^ (r & 7)) << 4));
    }
    static __device__ __forceinline__ uint4 *b16_unit(unsigned char *st, int r, int u) {
        return reinterpret_cast<uint4 *>(st + b16_at + r * 64 + ((u ^ ((r >> 1) & 3)) << 4));
    }
    // row r of the transposed piece's column c (64 bytes per column)
    static __device__ __forceinline__ __nv_bfloat16 *tr_elem(unsigned char *st, int c, int r) {
        return reinterpret_cast<__nv_bfloat16 *>(st + tr_at + c * 64) + r;
    }

    static __device__ __forceinline__ void store_f32(unsigned char *st, float *D, int M, int N, int row0, int col0, bool vec) {
        const int lane = threadIdx.x & 31;
        if (vec) {
            const int u = lane & 7, col = col0 + u * 4;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = i * 4 + (lane >> 3);
                if (row0 + r < M && col < N)
                    *reinterpret_cast<float4 *>(D + static_cast<size_t>(row0 + r) * N + col) = *f32_unit(st, r, u);
            }
        } else if (col0 + lane < N) {
            for (int r = 0; r < 32 && row0 + r < M; ++r)
                D[static_cast<size_t>(row0 + r) * N + col0 + lane] =
                    reinterpret_cast<const float *>(f32_unit(st, r, lane >> 2))[lane & 3];
        }
    }
    static __device__ __forceinline__ void store_b16(unsigned char *st, __nv_bfloat16 *H, int M, int N, int row0, int col0,
                                                     bool vec) {
        const int lane = threadIdx.x & 31;
        if (vec) {
            const int u = lane & 3, col = col0 + u * 8;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = i * 8 + (lane >> 2);
                if (row0 + r < M && col < N)
                    *reinterpret_cast<uint4 *>(H + static_cast<size_t>(row0 + r) * N + col) = *b16_unit(st, r, u);
            }
        } else if (col0 + lane < N) {
            for (int r = 0; r < 32 && row0 + r < M; ++r)
                H[static_cast<size_t>(row0 + r) * N + col0 + lane] =
                    reinterpret_cast<const __nv_bfloat16 *>(b16_unit(st, r, lane >> 3))[lane & 7];
        }
    }
    // the transposed piece into HT (N x M)
    static __device__ __forceinline__ void store_tr(unsigned char *st, __nv_bfloat16 *HT, int M, int N, int row0, int col0,
                                                    bool vec) {
        const int lane = threadIdx.x & 31;
        if (vec) {
            const int u = lane & 3, row = row0 + u * 8;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int c = i * 8 + (lane >> 2);
                if (col0 + c < N && row < M)
                    *reinterpret_cast<uint4 *>(HT + static_cast<size_t>(col0 + c) * M + row) =
                        *reinterpret_cast<const uint4 *>(tr_elem(st, c, u * 8));
            }
        } else if (row0 + lane < M) {
            for (int c = 0; c < 32 && col0 + c < N; ++c)
                HT[static_cast<size_t>(col0 + c) * M + row0 + lane] = *tr_elem(st, c, lane);
        }
    }
};

// Whether the rows of a matrix of `ld` elements of `size` bytes per row, starting at p, can be moved
// in 16-byte units.
bool unit_rows(const void *p, int ld, int size) {
    return reinterpret_cast<uintptr_t>(p) % 16 == 0 && (static_cast<size_t>(ld) * size) % 16 == 0;
}

// D (float32) = acc (+ bias); split z of a split-K product writes its partial at D + z * split_stride
struct EpiF32 {
    float *D;
    const float *bias;
    int M, N;
    size_t split_stride;
    bool vec;
    struct Regs {};
    EpiF32(float *D_, const float *bias_, int M_, int N_, size_t stride)
        : D(D_), bias(bias_), M(M_), N(N_), split_stride(stride), vec(unit_rows(D_, N_, 4) && stride % 4 == 0) {}
    __device__ __forceinline__ void prefetch(int, int, Regs &) const {}
    __device__ __forceinline__ void piece(int split, int row0, int col0, const float (&v)[32], const float *sbias,
                                          unsigned char *st, Regs &) const {
        const int lane = threadIdx.x & 31;
        const float4 *b4 = reinterpret_cast<const float4 *>(sbias);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const float4 b = b4[u];
            *EpiTile::f32_unit(st, lane, u) = make_float4(v[4 * u] + b.x, v[4 * u + 1] + b.y, v[4 * u + 2] + b.z, v[4 * u + 3] + b.w);
        }
        __syncwarp();
        EpiTile::store_f32(st, D + split * split_stride, M, N, row0, col0, vec);
        __syncwarp();
    }
};

// Forward linear layer: z = acc + bias (stored as float32 if Z), h = act(z) (stored as bf16 if H,
// and transposed as bf16 if HT, an N x M matrix).
struct EpiFwd {
    const float *bias;
    float *Z;
    __nv_bfloat16 *H;
    int N, act;
    __nv_bfloat16 *HT;
    int M;
    bool vec_z, vec_h, vec_t;
    struct Regs {};
    EpiFwd(const float *bias_, float *Z_, void *H_, void *HT_, int M_, int N_, int act_)
        : bias(bias_), Z(Z_), H(static_cast<__nv_bfloat16 *>(H_)), N(N_), act(act_), HT(static_cast<__nv_bfloat16 *>(HT_)),
          M(M_), vec_z(unit_rows(Z_, N_, 4)), vec_h(unit_rows(H_, N_, 2)), vec_t(unit_rows(HT_, M_, 2)) {}
    __device__ __forceinline__ void prefetch(int, int, Regs &) const {}
    __device__ __forceinline__ void piece(int, int row0, int col0, const float (&v)[32], const float *sbias,
                                          unsigned char *st, Regs &) const {
        const int lane = threadIdx.x & 31;
        const float4 *b4 = reinterpret_cast<const float4 *>(sbias);
#pragma unroll
        for (int u = 0; u < 4; ++u) {  // eight columns at a time
            const float4 b0 = b4[2 * u], b1 = b4[2 * u + 1];
            const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
            float z[8], h[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                z[i] = v[8 * u + i] + b[i];
                h[i] = act ? gelu(z[i]) : z[i];
            }
            if (Z) {
                *EpiTile::f32_unit(st, lane, 2 * u) = make_float4(z[0], z[1], z[2], z[3]);
                *EpiTile::f32_unit(st, lane, 2 * u + 1) = make_float4(z[4], z[5], z[6], z[7]);
            }
            if (H) *EpiTile::b16_unit(st, lane, u) = pack8_bf16(h);
            if (HT) {
#pragma unroll
                for (int i = 0; i < 8; ++i) *EpiTile::tr_elem(st, 8 * u + i, lane) = __float2bfloat16_rn(h[i]);
            }
        }
        __syncwarp();
        if (Z) EpiTile::store_f32(st, Z, M, N, row0, col0, vec_z);
        if (H) EpiTile::store_b16(st, H, M, N, row0, col0, vec_h);
        if (HT) EpiTile::store_tr(st, HT, M, N, row0, col0, vec_t);
        __syncwarp();
    }
};

// Backward through a linear layer into the previous GELU: dx = acc * gelu'(z_prev), bf16 (and
// transposed into dXT, an N x M matrix, if given). The first piece of z_prev is loaded while the
// products still run, the next one while the warp finishes the piece before it.
struct EpiBwd {
    const float *Zprev;
    __nv_bfloat16 *dX;
    int N;
    __nv_bfloat16 *dXT;
    int M;
    bool vec_z, vec_x, vec_t;
    static constexpr const float *bias = nullptr;
    struct Regs {
        float4 z[8];  // units lane % 8 of rows 4 i + lane / 8
    };
    EpiBwd(const float *Z_, void *dX_, void *dXT_, int M_, int N_)
        : Zprev(Z_), dX(static_cast<__nv_bfloat16 *>(dX_)), N(N_), dXT(static_cast<__nv_bfloat16 *>(dXT_)), M(M_),
          vec_z(unit_rows(Z_, N_, 4)), vec_x(unit_rows(dX_, N_, 2)), vec_t(unit_rows(dXT_, M_, 2)) {}
    __device__ __forceinline__ void prefetch(int row0, int col0, Regs &R) const {
        const int lane = threadIdx.x & 31, col = col0 + (lane & 7) * 4;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int row = row0 + i * 4 + (lane >> 3);
            float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (row < M) {
                const float *p = Zprev + static_cast<size_t>(row) * N + col;
                if (vec_z) {
                    if (col < N) z = *reinterpret_cast<const float4 *>(p);
                } else {
                    if (col < N) z.x = p[0];
                    if (col + 1 < N) z.y = p[1];
                    if (col + 2 < N) z.z = p[2];
                    if (col + 3 < N) z.w = p[3];
                }
            }
            R.z[i] = z;
        }
    }
    __device__ __forceinline__ void piece(int, int row0, int col0, const float (&v)[32], const float *, unsigned char *st,
                                          Regs &R) const {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int i = 0; i < 8; ++i) *EpiTile::f32_unit(st, i * 4 + (lane >> 3), lane & 7) = R.z[i];
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float4 z0 = *EpiTile::f32_unit(st, lane, 2 * u), z1 = *EpiTile::f32_unit(st, lane, 2 * u + 1);
            const float z[8] = {z0.x, z0.y, z0.z, z0.w, z1.x, z1.y, z1.z, z1.w};
            float d[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) d[i] = v[8 * u + i] * gelu_grad(z[i]);
            *EpiTile::b16_unit(st, lane, u) = pack8_bf16(d);
            if (dXT) {
#pragma unroll
                for (int i = 0; i < 8; ++i) *EpiTile::tr_elem(st, 8 * u + i, lane) = __float2bfloat16_rn(d[i]);
            }
        }
        __syncwarp();
        EpiTile::store_b16(st, dX, M, N, row0, col0, vec_x);
        if (dXT) EpiTile::store_tr(st, dXT, M, N, row0, col0, vec_t);
        __syncwarp();
    }
};

__global__ void transpose_bf16_kernel(const __nv_bfloat16 *__restrict__ X, __nv_bfloat16 *__restrict__ Y, int rows,
                                      int cols) {
    __shared__ __nv_bfloat16 tile[32][33];
    const int c = blockIdx.x * 32 + threadIdx.x, r0 = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += blockDim.y)
        if (r0 + j < rows && c < cols) tile[j][threadIdx.x] = X[static_cast<size_t>(r0 + j) * cols + c];
    __syncthreads();
    const int r = blockIdx.y * 32 + threadIdx.x, c0 = blockIdx.x * 32;
    for (int j = threadIdx.y; j < 32; j += blockDim.y)
        if (c0 + j < cols && r < rows) Y[static_cast<size_t>(c0 + j) * rows + r] = tile[threadIdx.x][j];
}

// Bias gradient db[n] = sum over rows of dZ[row][n], deterministically in two passes: block row y
// of the first sums rows y, y + G, y + 2G, ... (G = kColsumGroups) of its 128 columns into
// part[y][n]; the second adds the G partial sums of each column in a fixed order. No atomics, so a
// training step gives the same bits every time it runs.
constexpr int kColsumGroups = 128;

__global__ void colsum_partial_kernel(const __nv_bfloat16 *__restrict__ dZ, float *__restrict__ part, int M, int N) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // four independent chains keep several loads in flight
    int m = blockIdx.y;
    for (; m + 3 * static_cast<int>(gridDim.y) < M; m += 4 * gridDim.y) {
#pragma unroll
        for (int u = 0; u < 4; ++u) s[u] += __bfloat162float(dZ[static_cast<size_t>(m + u * gridDim.y) * N + n]);
    }
    for (; m < M; m += gridDim.y) s[0] += __bfloat162float(dZ[static_cast<size_t>(m) * N + n]);
    part[static_cast<size_t>(blockIdx.y) * N + n] = (s[0] + s[1]) + (s[2] + s[3]);
}

// One warp per column: lane l adds partial rows l, l + 32, ... in order, then a fixed shuffle tree
// adds the lanes (deterministic, and 32 loads in flight per column instead of one).
__global__ void colsum_final_kernel(const float *__restrict__ part, float *__restrict__ db, int N, int groups) {
    const int n = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (n >= N) return;  // warp-uniform
    float acc = 0.0f;
    for (int y = lane; y < groups; y += 32) acc += part[static_cast<size_t>(y) * N + n];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) db[n] = acc;
}

// Several bias gradients in one launch, each with the sums of the two kernels above in their order: a block
// takes 16 columns of one matrix over all rows; thread (y, half) has the row group y = 0 .. G - 1 of 8
// columns (16-byte loads), then a warp adds each column's G partial sums. Five layers at batch 4096 (18 MB
// from L2): 26.7 us in ten launches, 5.7 us in one.
constexpr int kColsumMost = 8, kColsumCols = 16;
struct ColsumProblems {
    const __nv_bfloat16 *dZ[kColsumMost];
    float *db[kColsumMost];
    int N[kColsumMost];
    int first[kColsumMost + 1];  // first block of each
    int count;
};
__global__ void __launch_bounds__(2 * kColsumGroups) colsum_multi_kernel(const __grid_constant__ ColsumProblems P, int M) {
    __shared__ float part[kColsumGroups][kColsumCols + 1];
    wait_for_inputs();
    int q = 0;
    while (q + 1 < P.count && static_cast<int>(blockIdx.x) >= P.first[q + 1]) ++q;
    const int N = P.N[q], n0 = (static_cast<int>(blockIdx.x) - P.first[q]) * kColsumCols;
    const int groups = M < kColsumGroups ? M : kColsumGroups;
    const int y = threadIdx.x >> 1, c0 = (threadIdx.x & 1) * 8;
    if (y < groups && n0 + c0 < N) {
        const __nv_bfloat16 *z = P.dZ[q] + n0 + c0;
        float s[4][8];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int k = 0; k < 8; ++k) s[u][k] = 0.0f;
        const auto add = [&](int u, const uint4 &x) {
            const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {  // a bf16 is the upper half of its float
                s[u][2 * k] += __uint_as_float(w[k] << 16);
                s[u][2 * k + 1] += __uint_as_float(w[k] & 0xFFFF0000u);
            }
        };
        int m = y;
        for (; m + 3 * groups < M; m += 4 * groups) {
            uint4 x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = *reinterpret_cast<const uint4 *>(z + static_cast<size_t>(m + u * groups) * N);
#pragma unroll
            for (int u = 0; u < 4; ++u) add(u, x[u]);
        }
        for (; m < M; m += groups) add(0, *reinterpret_cast<const uint4 *>(z + static_cast<size_t>(m) * N));
#pragma unroll
        for (int k = 0; k < 8; ++k) part[y][c0 + k] = (s[0][k] + s[1][k]) + (s[2][k] + s[3][k]);
    }
    dependents_may_start();
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int c = warp; c < kColsumCols && n0 + c < N; c += 2 * kColsumGroups / 32) {
        float acc = 0.0f;
        for (int g = lane; g < groups; g += 32) acc += part[g][c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) P.db[q][n0 + c] = acc;
    }
}

// Mean-squared error over the first T of ld columns: loss += scale * sum (p - t)^2 and
// dZ = 2 * scale * (p - t) (bf16; zero in the padded columns). Grid-stride over the elements; each
// block adds its partial loss once (one atomic per block rather than per warp).
__global__ void mse_kernel(const float *__restrict__ pred, const float *__restrict__ target, __nv_bfloat16 *dZ,
                           float *loss, int M, int T, int ld, float scale) {
    __shared__ float warp_sum[32];
    const size_t n = static_cast<size_t>(M) * ld;
    float l = 0.0f;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int row = static_cast<int>(i / ld), col = static_cast<int>(i % ld);
        float g = 0.0f;
        if (col < T) {
            const float d = pred[i] - target[static_cast<size_t>(row) * T + col];
            l += d * d;
            g = 2.0f * scale * d;
        }
        if (dZ) dZ[i] = __float2bfloat16_rn(g);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = l;
    __syncthreads();
    if (threadIdx.x < 32) {
        l = threadIdx.x < (blockDim.x >> 5) ? warp_sum[threadIdx.x] : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (threadIdx.x == 0 && l != 0.0f) atomicAdd(loss, l * scale);
    }
}

// The loss of a training step with what its backward pass reads: blocks 0 .. row_blocks - 1 take 32 rows
// of the error each (dZ, its transpose, the loss), the others 32 rows of the network's inputs (their
// transpose). Three passes and launches in one: 8.0 -> 6.8 us at batch 4096. A cluster of eight blocks adds its
// part of the loss at once, in order: float32 atomics round at every sum, in whatever order they come, and
// with one per 32 rows an epoch's mean loss moved by up to two units in its last place from run to run.
constexpr uint32_t kMseCluster = 8;
__global__ void __launch_bounds__(256) mse_transposes_kernel(const float *__restrict__ pred, const float *__restrict__ target,
                                                             __nv_bfloat16 *__restrict__ dZ, __nv_bfloat16 *__restrict__ dZT,
                                                             float *loss, int M, int T, int ld, float scale,
                                                             const __nv_bfloat16 *__restrict__ X, __nv_bfloat16 *__restrict__ XT,
                                                             int k, int row_blocks) {
    extern __shared__ __nv_bfloat16 tile[];  // 32 rows of ld or k columns, one apart from a bank multiple
    __shared__ float warp_sum[8];
    __shared__ float4 part;  // x: the block's part of the loss
    const bool inputs = static_cast<int>(blockIdx.x) >= row_blocks;
    wait_for_inputs();
    const int row0 = (static_cast<int>(blockIdx.x) - (inputs ? row_blocks : 0)) * 32, rows = max(0, min(32, M - row0));
    const int cols = inputs ? k : ld, pitch = cols + 2;
    float l = 0.0f;
    for (int i = threadIdx.x; i < rows * cols; i += 256) {
        const int r = i / cols, c = i % cols;
        const size_t row = static_cast<size_t>(row0 + r);
        __nv_bfloat16 v;
        if (inputs) {
            v = X[row * cols + c];
        } else {
            float g = 0.0f;
            if (c < T) {
                const float d = pred[row * cols + c] - target[row * T + c];
                l += d * d;
                g = 2.0f * scale * d;
            }
            v = __float2bfloat16_rn(g);
            dZ[row * cols + c] = v;
        }
        tile[r * pitch + c] = v;
    }
    dependents_may_start();
    __syncthreads();
    __nv_bfloat16 *const out = inputs ? XT : dZT;
    const int lane = threadIdx.x & 31;
    if (lane < rows)
        for (int c = threadIdx.x >> 5; c < cols; c += 8) out[static_cast<size_t>(c) * M + row0 + lane] = tile[lane * pitch + c];
    if (inputs) return;  // uniform in a cluster: row_blocks is a multiple of kMseCluster
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (lane == 0) warp_sum[threadIdx.x >> 5] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
        float sum = 0.0f;
        for (int w = 0; w < 8; ++w) sum += warp_sum[w];
        part.x = sum;
    }
    __syncwarp();
    cluster_barrier();  // every block's part is in place
    if (threadIdx.x == 0 && cluster_rank() == 0) {
        float sum = 0.0f;
        for (uint32_t b = 0; b < kMseCluster; ++b) sum += ld_cluster_f32x4(&part, b).x;
        if (sum != 0.0f) atomicAdd(loss, sum * scale);
    }
    __syncwarp();
    cluster_barrier();  // no block leaves while its part may still be read
}

// Polyak averaging of one value: avg = beta avg + (1 - beta) w, with its rounding pinned so that
// the separate pass (ema_kernel) and the one fused into Adam give the same bits.
__device__ __forceinline__ float polyak(float avg, float w, float beta) {
    return __fmaf_rn(beta, avg, __fmul_rn(__fsub_rn(1.0f, beta), w));
}

// One Adam step of element i of a rows x cols float32 parameter (row-major): the moments, the
// weight, its Polyak average (if avg), its bf16 copy (if wb) and transpose (if wt). Shared by the
// one-tensor and the many-tensor kernels, so both give the same bits. Returns the bf16 value.
__device__ __forceinline__ __nv_bfloat16 adam_element(size_t i, float *__restrict__ w, const float *__restrict__ g,
                                             float *__restrict__ m, float *__restrict__ v, int rows, int cols,
                                             float lr, float b1, float b2, float eps, float weight_decay,
                                             __nv_bfloat16 *wb, __nv_bfloat16 *wt, float *__restrict__ avg,
                                             float avg_beta) {
    const float gi = g[i] + weight_decay * w[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * mi / (sqrtf(vi) + eps);
    w[i] = wi;
    if (avg) avg[i] = polyak(avg[i], wi, avg_beta);
    const __nv_bfloat16 b = __float2bfloat16_rn(wi);
    if (wb) wb[i] = b;
    if (wt) {
        const int r = static_cast<int>(i / cols), c = static_cast<int>(i % cols);
        wt[static_cast<size_t>(c) * rows + r] = b;
    }
    return b;
}

// Adam on float32 master weights (rows x cols, row-major), writing the bf16 copy and its transpose.
// The step size is lr_dev[0] when lr_dev is given (so that a captured graph reads the current
// step's value), else lr_t; with avg given, the averaged weights are updated from the new ones.
__global__ void adam_kernel(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, int rows, int cols, float lr_t, const float *__restrict__ lr_dev,
                            float b1, float b2, float eps, float weight_decay, __nv_bfloat16 *wb,
                            __nv_bfloat16 *wt, float *__restrict__ avg, float avg_beta) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= static_cast<size_t>(rows) * cols) return;
    const float lr = lr_dev ? __ldg(lr_dev) : lr_t;
    adam_element(i, w, g, m, v, rows, cols, lr, b1, b2, eps, weight_decay, wb, wt, avg, avg_beta);
}

constexpr int kAdamThreads = 256;

// The same step for every tensor of a table (one launch for all of a network's parameters): block b
// belongs to the tensor whose first_block range holds it. A block's 256 elements are consecutive, or, where
// a transpose is written and the sides are multiples of 16, a 16 x 16 tile: element by element the
// transpose touched a sector per element (a network of 0.9 M parameters 14.2 -> 8.6 us, 36 MB).
__global__ void adam_multi_kernel(const tmc_adam_tensor *__restrict__ tab, int count, float lr_t,
                                  const float *__restrict__ lr_dev, float b1, float b2, float eps, float avg_beta) {
    __shared__ tmc_adam_tensor T;
    wait_for_inputs();
    dependents_may_start();
    if (threadIdx.x == 0) {
        int t = 0;
        while (t + 1 < count && static_cast<int>(blockIdx.x) >= tab[t + 1].first_block) ++t;
        T = tab[t];
    }
    __syncthreads();
    const int block = static_cast<int>(blockIdx.x) - T.first_block;
    const float lr = lr_dev ? __ldg(lr_dev) : lr_t;
    __nv_bfloat16 *const wb = reinterpret_cast<__nv_bfloat16 *>(T.wb), *const wt = reinterpret_cast<__nv_bfloat16 *>(T.wt);
    if (wt && T.rows % 16 == 0 && T.cols % 16 == 0) {  // block-uniform: a 16 x 16 tile, its transpose through shared memory
        __shared__ __nv_bfloat16 tile[16][18];
        const int across = T.cols / 16, r0 = block / across * 16, c0 = block % across * 16;
        const int a = threadIdx.x >> 4, b = threadIdx.x & 15;
        tile[a][b] = adam_element(static_cast<size_t>(r0 + a) * T.cols + c0 + b, T.w, T.g, T.m, T.v, T.rows, T.cols, lr, b1, b2,
                                  eps, T.weight_decay, wb, nullptr, T.avg, avg_beta);
        __syncthreads();
        wt[static_cast<size_t>(c0 + a) * T.rows + r0 + b] = tile[b][a];
        return;
    }
    const size_t i = static_cast<size_t>(block) * kAdamThreads + threadIdx.x;
    if (i >= static_cast<size_t>(T.rows) * T.cols) return;
    adam_element(i, T.w, T.g, T.m, T.v, T.rows, T.cols, lr, b1, b2, eps, T.weight_decay, wb, wt, T.avg, avg_beta);
}

// D = sum over the splits of a split-K product's partials (fixed order: deterministic)
__global__ void sum_splits_kernel(const float *__restrict__ work, float *__restrict__ D, size_t n, int splits) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float acc = 0.0f;
    for (int z = 0; z < splits; ++z) acc += work[z * n + i];
    D[i] = acc;
}

__global__ void ema_kernel(const float *__restrict__ w, float *__restrict__ avg, size_t n, float beta) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) avg[i] = polyak(avg[i], w[i], beta);
}

__global__ void to_bf16_kernel(const float *__restrict__ w, int rows, int cols, __nv_bfloat16 *wb,
                               __nv_bfloat16 *wt) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= static_cast<size_t>(rows) * cols) return;
    const __nv_bfloat16 b = __float2bfloat16_rn(w[i]);
    if (wb) wb[i] = b;
    if (wt) wt[static_cast<size_t>(i % cols) * rows + i / cols] = b;
}

// Network inputs from raw features: z-score the first nf of n_feat columns, zero-pad to ld, bf16.
__global__ void encode_kernel(const float *__restrict__ feats, const float *__restrict__ mean,
                              const float *__restrict__ stdv, __nv_bfloat16 *__restrict__ X, int n, int nf, int ld) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= static_cast<size_t>(n) * ld) return;
    const int row = static_cast<int>(i / ld), col = static_cast<int>(i % ld);
    const float v = col < nf ? (feats[static_cast<size_t>(row) * nf + col] - mean[col]) / stdv[col] : 0.0f;
    X[i] = __float2bfloat16_rn(v);
}

// The same from float64 features with float64 statistics: the z-score rounded to float32, then to bf16.
// One thread per column: bound by the launch and the features' copy (8,000 rows: 4 us).
__global__ void encode_f64_kernel(const double *__restrict__ feats, const double *__restrict__ mean,
                                  const double *__restrict__ stdv, __nv_bfloat16 *__restrict__ X, int n, int nf, int ld) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= static_cast<size_t>(n) * ld) return;
    const int row = static_cast<int>(i / ld), col = static_cast<int>(i % ld);
    const float v = col < nf ? static_cast<float>(__ddiv_rn(__dsub_rn(feats[static_cast<size_t>(row) * nf + col], mean[col]), stdv[col])) : 0.0f;
    X[i] = __float2bfloat16_rn(v);
}

// Raw outputs in float64 from the members' float32 outputs: y = z * std + mean, product and sum rounded
// apart, per member (out_members, members x n x n_out) and / or their mean (out_mean: the sum in member
// order, divided by the count). The host's arithmetic for four members of 8,000 queries took 7 ms of a
// predict call; this takes 8 us, its 17 MB of inputs and 4 MB of results through memory.
__global__ void denormalise_kernel(const float *__restrict__ Z, int members, size_t member_stride, int ld, int n, int n_out,
                                   const double *__restrict__ mean, const double *__restrict__ stdv,
                                   double *__restrict__ out_members, double *__restrict__ out_mean) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x, total = static_cast<size_t>(n) * n_out;
    if (i >= total) return;
    const int col = static_cast<int>(i % n_out);
    const float *z = Z + i / n_out * ld + col;
    double sum = 0.0;
    for (int m = 0; m < members; ++m) {
        const double y = __dadd_rn(__dmul_rn(static_cast<double>(z[m * member_stride]), stdv[col]), mean[col]);
        if (out_members) out_members[m * total + i] = y;
        sum = m ? __dadd_rn(sum, y) : y;
    }
    if (out_mean) out_mean[i] = __ddiv_rn(sum, static_cast<double>(members));
}

// The ensemble gate: for each query, every member's diffuse reflectance on the grid
// (sum over bins of 10^(z * std + mean) * area), their mean, their spread (sample standard
// deviation over the mean) and whether the spread exceeds the threshold (route the query to Monte
// Carlo).
__global__ void gate_kernel(const float *__restrict__ Z, int members, size_t member_stride, int ld,
                            const float *__restrict__ ymean, const float *__restrict__ ystd,
                            const float *__restrict__ areas, int nbins, int n, float threshold, float *rd_mean,
                            float *spread, unsigned char *route) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    float s1 = 0.0f, s2 = 0.0f;
    for (int m = 0; m < members; ++m) {
        const float *z = Z + m * member_stride + static_cast<size_t>(q) * ld;
        float rd = 0.0f;
        for (int b = 0; b < nbins; ++b) rd += exp10f(z[b] * ystd[b] + ymean[b]) * areas[b];
        s1 += rd;
        s2 += rd * rd;
    }
    const float mean = s1 / members;
    const float var = members > 1 ? fmaxf(s2 - s1 * mean, 0.0f) / (members - 1) : 0.0f;
    const float sp = sqrtf(var) / fmaxf(mean, 1e-12f);
    if (rd_mean) rd_mean[q] = mean;
    if (spread) spread[q] = sp;
    route[q] = sp > threshold ? 1 : 0;
}

std::mutex g_mu;
int *g_status[64] = {};
int g_gemm_sms[64] = {};  // SMs of a device whose GEMM kernels are ready to launch
bool g_infer_attr[64] = {};
int g_infer_clusters[64][kInferMaxMembers + 1] = {};  // clusters of that many CTAs resident at once (-1: none)

// The launch of the fused ensemble kernel on `blocks` CTAs in clusters of `members`.
cudaLaunchConfig_t infer_config(int blocks, int members, cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(blocks / members * members));
    cfg.blockDim = dim3(kInferThreads);
    cfg.dynamicSmemBytes = InferSmem::bytes;
    cfg.stream = s;
    return cfg;
}
cudaLaunchAttribute cluster_attr(int ctas) {
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = static_cast<unsigned>(ctas);
    a.val.clusterDim.y = a.val.clusterDim.z = 1;
    return a;
}

void put(tmc_status *st, int code, const std::string &m) {
    if (!st) return;
    st->code = code;
    std::snprintf(st->message, sizeof st->message, "%s", m.c_str());
}

int current_device() {
    int d = -1;
    if (cudaGetDevice(&d) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    return d;
}

// The per-device status word (allocated at the first call on a device, before any capture).
int *status_word(int dev) {
    if (dev < 0 || dev >= 64) return nullptr;
    if (!g_status[dev]) {
        if (cudaMalloc(&g_status[dev], sizeof(int)) != cudaSuccess) return nullptr;
        if (cudaMemset(g_status[dev], 0, sizeof(int)) != cudaSuccess) return nullptr;
    }
    return g_status[dev];
}

template <class Epi> void set_smem_attr() {
    cudaFuncSetAttribute(gemm_tc_kernel<kWide, Epi>, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmSmem<kWide>::bytes);
    cudaFuncSetAttribute(gemm_tc_kernel<kNarrow, Epi>, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmSmem<kNarrow>::bytes);
}

// cuTensorMapEncodeTiled, from the driver through the runtime (no link against libcuda).
PFN_cuTensorMapEncodeTiled_v12000 g_encode_tiled = nullptr;

// Tensor map of a rows x K bf16 matrix (K contiguous) read in boxes of 64 (K) x box_rows, with the
// 128-byte swizzle of the MMA operand tiles; rows past the end read as zeros.
bool encode_operand(CUtensorMap *map, const void *ptr, int rows, int K, int box_rows) {
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K) * 2u};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(kGemmBK), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t elem[2] = {1u, 1u};
    return g_encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, elem,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A launch that may start under the kernel before it in its stream (umma.cuh, wait_for_inputs): the kernels
// of a training step are a few microseconds long, a good part of it their start. With it one
// network's gradients at batch 4096 165 -> 146 us, an ensemble step (in epochs of 16 steps) at batch 1024
// 0.244 -> 0.234 ms, at 4096 0.415 -> 0.412 ms.
template <class... Params, class... Args>
void launch_chained(void (*kernel)(Params...), dim3 grid, int threads, int smem, cudaStream_t s, int cluster, Args &&...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = static_cast<size_t>(smem);
    cfg.stream = s;
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1] = cluster_attr(cluster);
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 0 ? 2 : 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// What a GEMM launch needs on the current device, under g_mu: the status word, the number of SMs, the
// driver's tensor-map encoder, the kernels' shared memory.
int gemm_ready(int **status, int *sms, tmc_status *st) {
    const int dev = current_device();
    *status = status_word(dev);
    if (!*status) {
        put(st, TMC_NO_DEVICE, "no usable CUDA device found");
        return TMC_NO_DEVICE;
    }
    if (!g_encode_tiled) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !fn) {
            cudaGetLastError();
            put(st, TMC_CUDA_ERROR, "the CUDA driver does not provide cuTensorMapEncodeTiled");
            return TMC_CUDA_ERROR;
        }
        g_encode_tiled = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    if (!g_gemm_sms[dev]) {
        set_smem_attr<EpiF32>();
        set_smem_attr<EpiFwd>();
        set_smem_attr<EpiBwd>();
        cudaFuncSetAttribute(wgrad_kernel<kWide>, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmSmem<kWide>::bytes);
        cudaDeviceGetAttribute(&g_gemm_sms[dev], cudaDevAttrMultiProcessorCount, dev);
    }
    *sms = g_gemm_sms[dev];
    return TMC_OK;
}

// Whether a product's tiles are 64 columns wide instead of 128: while all tiles are on the device at once a
// product lasts as long as one tile's loads, MMAs and epilogue, and half a tile's are shorter; A is loaded
// twice as often, though. Up to half as many wide tiles as SMs, so that each narrow one has an SM to itself:
// last layer at batch 4096 (32 wide tiles) 6.4 -> 5.0 us, a network's gradients at batch 2304 112 -> 93 us, the
// ensemble's step at batch 1024 0.235 -> 0.209 ms, 2048 0.302 -> 0.290. With the hidden layers at batch 4096
// (128 tiles) narrow too, one network's gradients go from 147 to 134 us, but the ensemble's step, whose four
// members fill the device, from 0.412 to 0.434 ms (in epochs of 16 steps).
bool narrow_tiles(int M, int N, int splits, int sms) {
    const int64_t across = (static_cast<int64_t>(N) + kWide - 1) / kWide, down = (static_cast<int64_t>(M) + kGemmBM - 1) / kGemmBM;
    return 2 * across * down * splits <= sms;
}

// Common checks and the launch of one tensor-core GEMM (asynchronous).
template <class Epi>
int launch_gemm(const void *A, const void *B, int M, int N, int K, const Epi &epi, void *stream, tmc_status *st,
                int splits = 1, uint32_t wait_limit = kGemmWaitLimit, int withhold = 0) {
    if (!A || !B) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument");
        return TMC_BAD_ARGUMENT;
    }
    if (M < 1 || N < 1 || K < 64 || K % 64 != 0) {
        put(st, TMC_BAD_CONFIG, "tensor-core GEMM needs M, N >= 1 and K a positive multiple of 64");
        return TMC_BAD_CONFIG;
    }
    if (splits < 1 || (K / 64) % splits != 0) {
        put(st, TMC_BAD_CONFIG, "split-K needs K / 64 to be a multiple of the number of splits");
        return TMC_BAD_CONFIG;
    }
    if (reinterpret_cast<uintptr_t>(A) % 16 != 0 || reinterpret_cast<uintptr_t>(B) % 16 != 0) {
        put(st, TMC_BAD_ARGUMENT, "tensor-core GEMM operands must be 16-byte aligned");
        return TMC_BAD_ARGUMENT;
    }
    std::lock_guard<std::mutex> lock(g_mu);
    int *status = nullptr, sms = 0;
    if (const int rc = gemm_ready(&status, &sms, st); rc != TMC_OK) return rc;
    const bool narrow = narrow_tiles(M, N, splits, sms);
    CUtensorMap ta, tb;
    if (!encode_operand(&ta, A, M, K, kGemmBM) || !encode_operand(&tb, B, N, K, narrow ? kNarrow : kWide)) {
        put(st, TMC_BAD_ARGUMENT, "tensor-core GEMM operands do not fit a TMA tensor map");
        return TMC_BAD_ARGUMENT;
    }
    const auto run = [&](auto bn) {
        constexpr int BN = decltype(bn)::value;
        const dim3 grid((N + BN - 1) / BN, (M + kGemmBM - 1) / kGemmBM, splits);
        launch_chained(gemm_tc_kernel<BN, Epi>, grid, kGemmThreads, GemmSmem<BN>::bytes, static_cast<cudaStream_t>(stream), 0,
                       ta, tb, M, N, K, epi, status, wait_limit, withhold);
    };
    if (narrow) run(std::integral_constant<int, kNarrow>{});
    else run(std::integral_constant<int, kWide>{});
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        put(st, TMC_CUDA_ERROR, std::string("CUDA error launching the tensor-core GEMM: ") + cudaGetErrorString(e));
        return TMC_CUDA_ERROR;
    }
    return TMC_OK;
}

int launched(tmc_status *st) {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        put(st, TMC_CUDA_ERROR, std::string("CUDA error: ") + cudaGetErrorString(e));
        return TMC_CUDA_ERROR;
    }
    return TMC_OK;
}

}  // namespace
}  // namespace tmc

using namespace tmc;

extern "C" {

int tmc_b200_gemm_bf16(const uint16_t *A, const uint16_t *B, const float *bias, float *D, int32_t M, int32_t N,
                       int32_t K, void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!D) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument");
        return TMC_BAD_ARGUMENT;
    }
    const int dev = current_device();
    int *status = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        status = status_word(dev);
    }
    if (!status) {
        put(st, TMC_NO_DEVICE, "no usable CUDA device found");
        return TMC_NO_DEVICE;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaMemsetAsync(status, 0, sizeof(int), s);
    const int rc = launch_gemm(A, B, M, N, K, EpiF32(D, bias, M, N, 0), stream, st);
    if (rc != TMC_OK) return rc;
    const cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        put(st, TMC_CUDA_ERROR, std::string("CUDA error in the tensor-core GEMM: ") + cudaGetErrorString(e));
        return TMC_CUDA_ERROR;
    }
    int h = 0;
    cudaMemcpy(&h, status, sizeof(int), cudaMemcpyDeviceToHost);
    if (h) {
        put(st, TMC_DEVICE_TIMEOUT, "a tensor-core wait gave up (mbarrier poll limit)");
        return TMC_DEVICE_TIMEOUT;
    }
    return TMC_OK;
}

int tmc_b200_probe_wait_timeout(int32_t device, uint32_t wait_limit, tmc_status *st) {
    put(st, TMC_OK, "");
    if (wait_limit < 1 || wait_limit > kGemmWaitLimit) {
        put(st, TMC_BAD_ARGUMENT, "wait_limit must be between 1 and the production limit");
        return TMC_BAD_ARGUMENT;
    }
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) {
        cudaGetLastError();
        put(st, TMC_NO_DEVICE, "no usable CUDA device found");
        return TMC_NO_DEVICE;
    }
    int saved = 0;
    cudaGetDevice(&saved);
    cudaSetDevice(device);
    // one 128 x 128 x 64 product whose producer issues no loads: the issuer's wait runs out
    void *buf = nullptr;
    const size_t a_bytes = 128 * 64 * 2, d_bytes = 128 * 128 * 4;
    if (cudaMalloc(&buf, 2 * a_bytes + d_bytes) != cudaSuccess) {
        cudaGetLastError();
        cudaSetDevice(saved);
        put(st, TMC_CUDA_ERROR, "CUDA error: cannot allocate the probe's operands");
        return TMC_CUDA_ERROR;
    }
    cudaMemset(buf, 0, 2 * a_bytes + d_bytes);
    unsigned char *b = static_cast<unsigned char *>(buf);
    int *status = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        status = status_word(device);
    }
    int rc = TMC_OK;
    if (!status) {
        put(st, TMC_NO_DEVICE, "no usable CUDA device found");
        rc = TMC_NO_DEVICE;
    } else {
        cudaMemset(status, 0, sizeof(int));
        rc = launch_gemm(b, b + a_bytes, 128, 128, 64, EpiF32(reinterpret_cast<float *>(b + 2 * a_bytes), nullptr, 128, 128, 0),
                         nullptr, st, 1, wait_limit, 1);
        if (rc == TMC_OK) {
            const cudaError_t e = cudaDeviceSynchronize();
            int h = 0;
            if (e == cudaSuccess) cudaMemcpy(&h, status, sizeof(int), cudaMemcpyDeviceToHost);
            if (e != cudaSuccess) {
                put(st, TMC_CUDA_ERROR, std::string("CUDA error in the wait probe: ") + cudaGetErrorString(e));
                rc = TMC_CUDA_ERROR;
            } else if (h) {
                put(st, TMC_DEVICE_TIMEOUT, h == 1 ? "a tensor-core wait gave up (mbarrier poll limit)"
                                                   : "a tensor-core wait gave up and the CTA's own work did not drain");
                rc = TMC_DEVICE_TIMEOUT;
            }
            cudaMemset(status, 0, sizeof(int));
        }
    }
    cudaFree(buf);
    cudaSetDevice(saved);
    return rc;
}

int tmc_b200_nn_linear(const uint16_t *X, const uint16_t *W, const float *bias, float *Z, uint16_t *H, uint16_t *HT,
                       int32_t M, int32_t N, int32_t K, int32_t gelu_act, void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!bias || (!Z && !H && !HT)) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument");
        return TMC_BAD_ARGUMENT;
    }
    return launch_gemm(X, W, M, N, K,
                       EpiFwd(bias, Z, H, HT, M, N, gelu_act),
                       stream, st);
}

int tmc_b200_nn_backward_data(const uint16_t *dZ, const uint16_t *WT, const float *Zprev, uint16_t *dX, uint16_t *dXT,
                              int32_t M, int32_t N, int32_t K, void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!Zprev || !dX) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument");
        return TMC_BAD_ARGUMENT;
    }
    return launch_gemm(dZ, WT, M, N, K,
                       EpiBwd(Zprev, dX, dXT, M, N),
                       stream, st);
}

int tmc_b200_nn_matmul_f32(const uint16_t *A, const uint16_t *B, float *D, int32_t M, int32_t N, int32_t K,
                           void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!D) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument");
        return TMC_BAD_ARGUMENT;
    }
    return launch_gemm(A, B, M, N, K, EpiF32(D, nullptr, M, N, 0), stream, st);
}

int tmc_b200_nn_matmul_f32_splitk(const uint16_t *A, const uint16_t *B, float *D, float *work, int32_t M, int32_t N,
                                  int32_t K, int32_t splits, void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!D || !work) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument");
        return TMC_BAD_ARGUMENT;
    }
    const size_t mn = static_cast<size_t>(M) * N;
    const int rc = launch_gemm(A, B, M, N, K, EpiF32(work, nullptr, M, N, mn), stream, st, splits);
    if (rc != TMC_OK) return rc;
    sum_splits_kernel<<<static_cast<unsigned>((mn + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        work, D, mn, splits);
    return launched(st);
}

int tmc_b200_nn_weight_grads(const uint16_t *const *A, const uint16_t *const *B, float *const *D, const int32_t *M,
                             const int32_t *N, int32_t count, int32_t K, int32_t splits, void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!A || !B || !D || !M || !N || count < 1 || count > kWgradMost) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument, or not 1 to 8 products");
        return TMC_BAD_ARGUMENT;
    }
    if (K < 64 || K % 64 != 0 || splits < 1 || splits > 8 || (K / 64) % splits != 0) {
        put(st, TMC_BAD_CONFIG, "weight gradients need K a positive multiple of 64 and K / 64 a multiple of 1 to 8 splits");
        return TMC_BAD_CONFIG;
    }
    std::lock_guard<std::mutex> lock(g_mu);
    int *status = nullptr, sms = 0;
    if (const int rc = gemm_ready(&status, &sms, st); rc != TMC_OK) return rc;
    WgradProblems P{};
    P.count = count;
    for (int q = 0; q < count; ++q) {
        if (!A[q] || !B[q] || !D[q] || M[q] < 1 || N[q] < 1 || reinterpret_cast<uintptr_t>(A[q]) % 16 != 0 ||
            reinterpret_cast<uintptr_t>(B[q]) % 16 != 0 || !encode_operand(&P.a[q], A[q], M[q], K, kGemmBM) ||
            !encode_operand(&P.b[q], B[q], N[q], K, kWide)) {
            put(st, TMC_BAD_ARGUMENT, "weight-gradient operands must be 16-byte aligned and fit a TMA tensor map");
            return TMC_BAD_ARGUMENT;
        }
        P.D[q] = D[q];
        P.M[q] = M[q];
        P.N[q] = N[q];
        P.first[q + 1] = P.first[q] + (M[q] + kGemmBM - 1) / kGemmBM * ((N[q] + kWide - 1) / kWide);
    }
    launch_chained(wgrad_kernel<kWide>, dim3(static_cast<unsigned>(P.first[count] * splits)), kGemmThreads, GemmSmem<kWide>::bytes,
                   static_cast<cudaStream_t>(stream), splits, P, K, splits, status);
    return launched(st);
}

int tmc_b200_nn_transpose(const uint16_t *X, uint16_t *Y, int32_t rows, int32_t cols, void *stream,
                          tmc_status *st) {
    put(st, TMC_OK, "");
    if (!X || !Y || rows < 1 || cols < 1) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument or empty matrix");
        return TMC_BAD_ARGUMENT;
    }
    transpose_bf16_kernel<<<dim3((cols + 31) / 32, (rows + 31) / 32), dim3(32, 8), 0,
                            static_cast<cudaStream_t>(stream)>>>(reinterpret_cast<const __nv_bfloat16 *>(X),
                                                                 reinterpret_cast<__nv_bfloat16 *>(Y), rows, cols);
    return launched(st);
}

int tmc_b200_nn_colsum(const uint16_t *dZ, float *db, int32_t M, int32_t N, float *work, void *stream,
                       tmc_status *st) {
    put(st, TMC_OK, "");
    if (!dZ || !db || !work || M < 1 || N < 1) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument or empty matrix");
        return TMC_BAD_ARGUMENT;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int groups = M < kColsumGroups ? M : kColsumGroups;
    colsum_partial_kernel<<<dim3((N + 127) / 128, groups), 128, 0, s>>>(reinterpret_cast<const __nv_bfloat16 *>(dZ),
                                                                      work, M, N);
    colsum_final_kernel<<<(N + 7) / 8, 256, 0, s>>>(work, db, N, groups);  // 8 columns (warps) per block
    return launched(st);
}

int tmc_b200_nn_colsum_multi(const uint16_t *const *dZ, float *const *db, const int32_t *N, int32_t count, int32_t M,
                             void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!dZ || !db || !N || count < 1 || count > kColsumMost || M < 1) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument, no rows, or not 1 to 8 matrices");
        return TMC_BAD_ARGUMENT;
    }
    ColsumProblems P{};
    P.count = count;
    for (int q = 0; q < count; ++q) {
        if (!dZ[q] || !db[q] || N[q] < 8 || N[q] % 8 != 0 || reinterpret_cast<uintptr_t>(dZ[q]) % 16 != 0) {
            put(st, TMC_BAD_ARGUMENT, "every matrix must be 16-byte aligned with a multiple of 8 columns");
            return TMC_BAD_ARGUMENT;
        }
        P.dZ[q] = reinterpret_cast<const __nv_bfloat16 *>(dZ[q]);
        P.db[q] = db[q];
        P.N[q] = N[q];
        P.first[q + 1] = P.first[q] + (N[q] + kColsumCols - 1) / kColsumCols;
    }
    launch_chained(colsum_multi_kernel, dim3(static_cast<unsigned>(P.first[count])), 2 * kColsumGroups, 0,
                   static_cast<cudaStream_t>(stream), 0, P, M);
    return launched(st);
}

int32_t tmc_b200_nn_colsum_work(int32_t N) { return N < 1 ? 0 : kColsumGroups * N; }

int tmc_b200_nn_mse(const float *pred, const float *target, uint16_t *dZ, float *loss, int32_t M, int32_t T,
                    int32_t ld, float scale, void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!pred || !target || !loss || M < 1 || T < 1 || ld < T) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument or bad shape");
        return TMC_BAD_ARGUMENT;
    }
    const size_t n = static_cast<size_t>(M) * ld;
    const size_t blocks = std::min<size_t>((n + 255) / 256, 1184);  // at most 8 blocks per SM of a B200
    mse_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        pred, target, reinterpret_cast<__nv_bfloat16 *>(dZ), loss, M, T, ld, scale);
    return launched(st);
}

int tmc_b200_nn_mse_transposes(const float *pred, const float *target, uint16_t *dZ, uint16_t *dZT, float *loss, int32_t M,
                               int32_t T, int32_t ld, float scale, const uint16_t *X, uint16_t *XT, int32_t k, void *stream,
                               tmc_status *st) {
    put(st, TMC_OK, "");
    if (!pred || !target || !dZ || !dZT || !loss || !X || !XT || M < 1 || T < 1 || ld < T || k < 1 || std::max(ld, k) > 512) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument or bad shape (at most 512 columns)");
        return TMC_BAD_ARGUMENT;
    }
    const int clusters = ((M + 31) / 32 + kMseCluster - 1) / kMseCluster, blocks = clusters * kMseCluster;
    launch_chained(mse_transposes_kernel, dim3(static_cast<unsigned>(2 * blocks)), 256,
                   static_cast<int>(32 * (std::max(ld, k) + 2) * sizeof(__nv_bfloat16)), static_cast<cudaStream_t>(stream), kMseCluster,
                   pred, target, reinterpret_cast<__nv_bfloat16 *>(dZ), reinterpret_cast<__nv_bfloat16 *>(dZT), loss, M, T, ld,
                   scale, reinterpret_cast<const __nv_bfloat16 *>(X), reinterpret_cast<__nv_bfloat16 *>(XT), k, blocks);
    return launched(st);
}

int tmc_b200_nn_adam(float *w, const float *g, float *m, float *v, int32_t rows, int32_t cols, float lr_t,
                     const float *lr_dev, float b1, float b2, float eps, float weight_decay, uint16_t *wb, uint16_t *wt,
                     float *avg, float avg_beta, void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!w || !g || !m || !v || rows < 1 || cols < 1) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument or empty parameter");
        return TMC_BAD_ARGUMENT;
    }
    const size_t n = static_cast<size_t>(rows) * cols;
    adam_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        w, g, m, v, rows, cols, lr_t, lr_dev, b1, b2, eps, weight_decay, reinterpret_cast<__nv_bfloat16 *>(wb),
        reinterpret_cast<__nv_bfloat16 *>(wt), avg, avg_beta);
    return launched(st);
}

int32_t tmc_b200_nn_adam_plan(tmc_adam_tensor *tab, int32_t count) {
    if (!tab || count < 1) return -1;
    int64_t blocks = 0;
    for (int t = 0; t < count; ++t) {
        if (tab[t].rows < 1 || tab[t].cols < 1) return -1;
        tab[t].first_block = static_cast<int32_t>(blocks);
        blocks += (static_cast<int64_t>(tab[t].rows) * tab[t].cols + kAdamThreads - 1) / kAdamThreads;
        if (blocks > 0x7FFFFFFF) return -1;
    }
    return static_cast<int32_t>(blocks);
}

int tmc_b200_nn_adam_multi(const tmc_adam_tensor *tab, int32_t count, int32_t blocks, float lr_t, const float *lr_dev,
                           float b1, float b2, float eps, float avg_beta, void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!tab || count < 1 || blocks < 1) {
        put(st, TMC_BAD_ARGUMENT, "NULL table, no tensors or no blocks (plan the table first)");
        return TMC_BAD_ARGUMENT;
    }
    launch_chained(adam_multi_kernel, dim3(static_cast<unsigned>(blocks)), kAdamThreads, 0, static_cast<cudaStream_t>(stream), 0,
                   tab, count, lr_t, lr_dev, b1, b2, eps, avg_beta);
    return launched(st);
}

int tmc_b200_nn_ema(const float *w, float *avg, int64_t n, float beta, void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!w || !avg || n < 1) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument or empty parameter");
        return TMC_BAD_ARGUMENT;
    }
    ema_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        w, avg, static_cast<size_t>(n), beta);
    return launched(st);
}

int tmc_b200_nn_to_bf16(const float *w, int32_t rows, int32_t cols, uint16_t *wb, uint16_t *wt, void *stream,
                        tmc_status *st) {
    put(st, TMC_OK, "");
    if (!w || rows < 1 || cols < 1) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument or empty parameter");
        return TMC_BAD_ARGUMENT;
    }
    const size_t n = static_cast<size_t>(rows) * cols;
    to_bf16_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        w, rows, cols, reinterpret_cast<__nv_bfloat16 *>(wb), reinterpret_cast<__nv_bfloat16 *>(wt));
    return launched(st);
}

int tmc_b200_nn_encode(const float *feats, const float *mean, const float *stdv, uint16_t *X, int32_t n, int32_t nf,
                       int32_t ld, void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!feats || !mean || !stdv || !X || n < 1 || nf < 1 || ld < nf) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument or bad shape");
        return TMC_BAD_ARGUMENT;
    }
    const size_t total = static_cast<size_t>(n) * ld;
    encode_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        feats, mean, stdv, reinterpret_cast<__nv_bfloat16 *>(X), n, nf, ld);
    return launched(st);
}

int tmc_b200_nn_encode_f64(const double *feats, const double *mean, const double *stdv, uint16_t *X, int32_t n, int32_t nf,
                           int32_t ld, void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!feats || !mean || !stdv || !X || n < 1 || nf < 1 || ld < nf) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument or bad shape");
        return TMC_BAD_ARGUMENT;
    }
    const size_t total = static_cast<size_t>(n) * ld;
    encode_f64_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        feats, mean, stdv, reinterpret_cast<__nv_bfloat16 *>(X), n, nf, ld);
    return launched(st);
}

int tmc_b200_nn_denormalise(const float *Z, int32_t members, int64_t member_stride, int32_t ld, int32_t n, int32_t n_out,
                            const double *mean, const double *stdv, double *out_members, double *out_mean, void *stream,
                            tmc_status *st) {
    put(st, TMC_OK, "");
    if (!Z || !mean || !stdv || (!out_members && !out_mean) || members < 1 || n < 1 || n_out < 1 || ld < n_out ||
        member_stride < 0) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument or bad shape");
        return TMC_BAD_ARGUMENT;
    }
    const size_t total = static_cast<size_t>(n) * n_out;
    denormalise_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        Z, members, static_cast<size_t>(member_stride), ld, n, n_out, mean, stdv, out_members, out_mean);
    return launched(st);
}

int tmc_b200_nn_gate(const float *Z, int32_t members, int64_t member_stride, int32_t ld, const float *ymean,
                     const float *ystd, const float *areas, int32_t nbins, int32_t n, float threshold, float *rd_mean,
                     float *spread, uint8_t *route, void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!Z || !ymean || !ystd || !areas || !route || members < 1 || n < 1 || nbins < 1 || ld < nbins) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument or bad shape");
        return TMC_BAD_ARGUMENT;
    }
    gate_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        Z, members, static_cast<size_t>(member_stride), ld, ymean, ystd, areas, nbins, n, threshold, rd_mean, spread,
        route);
    return launched(st);
}

int64_t tmc_b200_nn_packed_bytes(int32_t members) {
    return members < 1 ? 0 : static_cast<int64_t>(members) * kInferMemberBytes;
}

int tmc_b200_nn_pack(const uint16_t *const *weights, int32_t members, uint8_t *packed, void *stream,
                     tmc_status *st) {
    put(st, TMC_OK, "");
    if (!weights || !packed) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument");
        return TMC_BAD_ARGUMENT;
    }
    if (members < 1 || members > kInferMaxMembers) {
        put(st, TMC_BAD_CONFIG, "the fused ensemble holds 1 to 8 members");
        return TMC_BAD_CONFIG;
    }
    PackParams P{};
    P.members = members;
    for (int i = 0; i < members * kInferLayers; ++i) {
        if (!weights[i] || reinterpret_cast<uintptr_t>(weights[i]) % 16 != 0) {
            put(st, TMC_BAD_ARGUMENT, "every weight matrix must be a non-NULL, 16-byte aligned device pointer");
            return TMC_BAD_ARGUMENT;
        }
        P.w[i] = reinterpret_cast<const __nv_bfloat16 *>(weights[i]);
    }
    const size_t units = static_cast<size_t>(members) * (kInferMemberBytes / 16);
    pack_kernel<<<static_cast<unsigned>((units + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(P, packed);
    return launched(st);
}

int tmc_b200_nn_ensemble_infer(const uint8_t *packed, const float *bias, int32_t members, const float *feats, int32_t n,
                               int32_t n_feat, const float *x_mean, const float *x_std, int32_t n_out,
                               const float *y_mean, const float *y_std, const float *areas, int32_t nbins,
                               float threshold, float *out, float *rd_mean, float *spread, uint8_t *route,
                               void *stream, tmc_status *st) {
    put(st, TMC_OK, "");
    if (!packed || !bias || !x_mean || !x_std || !y_mean || !y_std || (n > 0 && !feats) || (nbins > 0 && !areas)) {
        put(st, TMC_BAD_ARGUMENT, "NULL argument");
        return TMC_BAD_ARGUMENT;
    }
    if (members < 1 || members > kInferMaxMembers || n < 0 || n_feat < 1 || n_feat > kInferIn || n_out < 1 ||
        n_out > kInferOut || nbins < 0 || nbins > 64 || nbins > n_out) {
        put(st, TMC_BAD_CONFIG,
            "fused ensemble: 1-8 members, 1-64 input features, 1-128 outputs, 0-64 R_d bins among the outputs");
        return TMC_BAD_CONFIG;
    }
    if (n == 0) return TMC_OK;
    if (reinterpret_cast<uintptr_t>(packed) % 16 != 0) {
        put(st, TMC_BAD_ARGUMENT, "the packed weights must be 16-byte aligned");
        return TMC_BAD_ARGUMENT;
    }
    const int dev = current_device();
    int sms = 0, clusters = 0;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (!status_word(dev) || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
            cudaGetLastError();
            put(st, TMC_NO_DEVICE, "no usable CUDA device found");
            return TMC_NO_DEVICE;
        }
        if (!g_infer_attr[dev]) {
            if (cudaFuncSetAttribute(ensemble_infer_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     InferSmem::bytes) != cudaSuccess ||
                cudaFuncSetAttribute(ensemble_infer_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     InferSmem::bytes) != cudaSuccess)
                return launched(st);
            g_infer_attr[dev] = true;
        }
        if (members > 1) {
            if (!g_infer_clusters[dev][members]) {
                cudaLaunchConfig_t cfg = infer_config(members * sms, members, nullptr);
                cudaLaunchAttribute attr = cluster_attr(members);
                cfg.attrs = &attr;
                cfg.numAttrs = 1;
                int c = 0;
                if (cudaOccupancyMaxActiveClusters(&c, ensemble_infer_kernel<true>, &cfg) != cudaSuccess) {
                    cudaGetLastError();
                    c = 0;
                }
                g_infer_clusters[dev][members] = c > 0 ? c : -1;
            }
            clusters = g_infer_clusters[dev][members];
        }
    }
    InferParams P{};
    P.packed = packed;
    P.bias = bias;
    P.feats = feats;
    P.x_mean = x_mean;
    P.x_std = x_std;
    P.y_mean = y_mean;
    P.y_std = y_std;
    P.areas = areas;
    P.out = out;
    P.rd_mean = rd_mean;
    P.spread = spread;
    P.route = route;
    P.n = n;
    P.n_feat = n_feat;
    P.n_out = n_out;
    P.nbins = nbins;
    P.members = members;
    P.threshold = threshold;
    P.status = g_status[dev];
    // One CTA per SM (its shared memory allows no more). A CTA takes whole tiles, member after member,
    // or a cluster of `members` CTAs takes a tile, one member each. The first form has the higher rate
    // while it fills the device, so it gets the whole rounds of one tile per SM; the last, partial round
    // goes to whichever form needs less time. In units of one member on one tile the first takes
    // `members`, the second one per round of resident clusters and a tenth more for the exchange between
    // the CTAs (four members, 37 tiles: 66 us in clusters, 111 us whole; 71 tiles: 96 us against 111).
    const int tiles = (n + 127) / 128;
    const int whole = tiles / sms * sms, rest = tiles - whole;
    const int split_rounds = clusters > 0 ? (rest + clusters - 1) / clusters : members;
    const bool split = rest > 0 && split_rounds * 11 < members * 10;
    const int plain = split ? whole : tiles;  // tiles in the first form
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (plain > 0) {
        P.n = std::min(n, plain * 128);
        ensemble_infer_kernel<false><<<std::min(plain, sms), kInferThreads, InferSmem::bytes, s>>>(P);
        if (const int rc = launched(st); rc != TMC_OK) return rc;
    }
    if (split) {
        const size_t row0 = static_cast<size_t>(plain) * 128;
        P.n = n - static_cast<int>(row0);
        P.feats = feats + row0 * n_feat;
        P.out = out ? out + row0 * n_out : nullptr;
        P.rd_mean = rd_mean ? rd_mean + row0 : nullptr;
        P.spread = spread ? spread + row0 : nullptr;
        P.route = route ? route + row0 : nullptr;
        cudaLaunchConfig_t cfg = infer_config(members * std::min(rest, clusters), members, s);
        cudaLaunchAttribute attr = cluster_attr(members);
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, ensemble_infer_kernel<true>, P);
    }
    return launched(st);
}

int tmc_b200_nn_status(int32_t clear) {
    const int dev = current_device();
    std::lock_guard<std::mutex> lock(g_mu);
    if (dev < 0 || dev >= 64 || !g_status[dev]) return 0;
    int h = 0;
    cudaMemcpy(&h, g_status[dev], sizeof(int), cudaMemcpyDeviceToHost);
    if (clear) cudaMemset(g_status[dev], 0, sizeof(int));
    return h;
}

}  // extern "C"
