// The persistent photon-walk kernel of one run (see walk.cuh for the design and the reference
// citations; the step itself is walk_step.cuh).
#pragma once

#include "walk_step.cuh"
#include "work_queue.cuh"

namespace tmc {

// Shared-memory layout of one block, in 64-bit words (offsets computed identically on the host).
struct SmemLayout {
    int ring, batch, core_a, lastz_a, lastr_a, rd, tt, layers, alone, total;  // word offsets / total words
};

__host__ __device__ inline SmemLayout smem_layout(const WalkParams &P) {
    SmemLayout s;
    int off = 0;
    // each lane's random words: a ring of kRingWords 32-bit words
    s.ring = off;
    off += static_cast<int>(kRingWords / 2) * static_cast<int>(P.threads);
    s.batch = off;
    off += P.batch_smem ? P.nb * (4 + P.nl) : 0;
    s.core_a = off;
    off += P.tr_a * P.tz_a;
    // The clamped last depth bin and last radius bin of A(r,z) collect every deposit beyond the
    // grid; for a deep or wide stack they are the hottest bins, so a tile that does not cover the
    // whole grid carries them too (a "cross": core + last column + last row).
    const bool cross = P.profiles && P.cross;
    s.lastz_a = off;
    off += cross ? P.nr : 0;
    s.lastr_a = off;
    off += cross ? P.nz : 0;
    s.rd = off;
    off += P.tr_rd * P.na;
    s.tt = off;
    off += P.tr_tt * P.na;
    off = (off + 1) & ~1;  // 16-byte alignment for the layer table
    s.layers = off;
    off += (P.nl * static_cast<int>(sizeof(LayerC)) + 7) / 8;
    s.alone = off;
    off += static_cast<int>(sizeof(AloneState) / 8);
    s.total = off;
    return s;
}

// Where one run's walk keeps its layer table and tallies: a shared-memory layer table, per-batch
// totals and profile tiles privatised in shared memory (the rest in global memory).
// CORE: the plan has a shared core tile of A(r,z) (tr_a, tz_a > 0); without one the kernel is a
// separate instantiation that does not test for it.
// PROF: the run keeps the profile tallies (A(r,z), R_d(r,a), T_t(r,a)); a run of totals only is an
// instantiation of its own, so the step carries no test for it.
template <int FAST, bool CORE, bool PROF> struct PlainCtx {
    const WalkParams &P;
    Ring ring;  // refilled with the launch's precomputed Philox key schedule (P.round_keys)
    uint32_t step_cap;
    const LayerC *layers;
    unsigned long long *bt;
    int bstride;
    // The block's shared words through a generic address, and where the tiles start in them. (An atomic
    // whose address is known to be shared compiles into a compare-and-swap loop for 64-bit sums: 2,555
    // SM cycles for a warp on one word, 284 with four lanes on one, 29 with none; the generic form is
    // one instruction, 32, 14 and 14 cycles.)
    unsigned long long *words;
    int at_core, at_lastz, at_lastr, at_rd, at_tt;
    bool cross;
    static constexpr bool kPublishAtRelaunch = true;  // measured 2.4 % faster than in the step

    __device__ __forceinline__ void refill(Lane &L) const { ring.refill(L, P.round_keys); }
    __device__ __forceinline__ void refill2(Lane &L) const { ring.refill2(L, P.round_keys); }
    __device__ __forceinline__ void block(uint32_t id, uint32_t blk, uint32_t &w0, uint32_t &w1, uint32_t &w2, uint32_t &w3) const {
        philox4x32_10_rk(id, 0u, blk, P.round_keys, w0, w1, w2, w3);
    }
    __device__ __forceinline__ uint32_t tag() const { return 0u; }
    __device__ __forceinline__ void adopt(uint32_t) {}
    __device__ __forceinline__ float path(const Lane &L, const Hot &h) const { return step_length<FAST>(h, unit_open(ring.peek(L))); }
    __device__ __forceinline__ float unit(Lane &L) const { return unit_open(ring.draw(L)); }
    __device__ __forceinline__ void skip(Lane &L) const { ring.skip(L); }
    __device__ __forceinline__ void pass(Lane &L, uint32_t n) const { L.rp += n; }
    __device__ __forceinline__ void scatter(Lane &L, const Hot &h, float dwa) const { scatter_now<FAST>(L, *this, h, dwa); }
    __device__ __forceinline__ void leave_layer(Lane &) const {}
    __device__ __forceinline__ void enter_layer(Lane &) const {}
    __device__ __forceinline__ const LayerC &layer(const Lane &, int l) const { return layers[l]; }
    __device__ __forceinline__ int num_layers(const Lane &) const { return P.nl; }
    __device__ __forceinline__ void batch_add(const Lane &L, int slot, unsigned long long v) const {
        atomicAdd(&bt[L.batch * bstride + slot], v);
    }

    // Deposit into A(r,z) at bin (ir, iz): the shared core tile, the shared cross, or global memory, by
    // one generic-address atomic on the selected word (no divergent paths). The word is an index from
    // one of two bases: one 64-bit select and one address for whichever it is.
    __device__ __forceinline__ void deposit(int ir, int iz, unsigned long long v) const {
        int idx = ir * P.nz + iz;
        bool shared = false;
        if (cross) {
            if (ir == P.nr - 1) {
                idx = at_lastr + iz;
                shared = true;
            }
            if (iz == P.nz - 1) {
                idx = at_lastz + ir;
                shared = true;
            }
        }
        if (CORE && ir < P.tr_a && iz < P.tz_a) {
            idx = at_core + ir * P.tz_a + iz;
            shared = true;
        }
        atomicAdd((shared ? words : P.g_arz) + idx, v);
    }

    // Every deposit goes straight to its word (shared tile or global): a per-lane cache of the last
    // bin (merging consecutive deposits into one bin) measured 4 % slower on skin5, its branch
    // costing more than the atomics it saved.
    __device__ __forceinline__ void absorb(float2 xy, float z, unsigned long long v) const {
        if constexpr (!PROF) return;
        const float rr = radius<FAST>(xy);
        int ir, iz;
        bins_rz<FAST>(rr, z, P.dr, P.dz, P.inv_dr, P.inv_dz, P.nr, P.nz, ir, iz);
        deposit(ir, iz, v);
    }

    __device__ __forceinline__ void exit(const Lane &L, int kind, unsigned long long v) const {
        if constexpr (!PROF) return;
        const float rr = radius<FAST>(L.xy);
        const int ir = bin_of<FAST>(rr, P.dr, P.inv_dr, P.nr);
        const int ia = bin_of<FAST>(acosf(fminf(fabsf(L.uz), 1.0f)), P.da, P.inv_da, P.na);
        const bool top = kind == 1, shared = ir < (top ? P.tr_rd : P.tr_tt);
        unsigned long long *const base = shared ? words + (top ? at_rd : at_tt) : (top ? P.g_rd : P.g_tt);
        atomicAdd(base + ir * P.na + ia, v);
    }
};

// Minimum resident blocks per SM the compiler must allow for; 0 leaves the register budget to
// the compiler (which then uses 63 registers: four 256-thread blocks per SM).
#ifndef TMC_WALK_MIN_BLOCKS
#define TMC_WALK_MIN_BLOCKS 0
#endif
#if TMC_WALK_MIN_BLOCKS > 0
#define TMC_WALK_BOUNDS __launch_bounds__(256, TMC_WALK_MIN_BLOCKS)
#else
#define TMC_WALK_BOUNDS __launch_bounds__(256)
#endif

template <int FAST, bool CORE, bool PROF>
__device__ __forceinline__ PlainCtx<FAST, CORE, PROF> plain_ctx(const WalkParams &P, const SmemLayout &S, unsigned long long *smem) {
    return PlainCtx<FAST, CORE, PROF>{P,
                     Ring{reinterpret_cast<uint32_t *>(smem + S.ring) + ring_lane_offset()},
                     P.step_cap,
                     reinterpret_cast<const LayerC *>(smem + S.layers),
                     P.batch_smem ? smem + S.batch : P.g_batch,
                     4 + P.nl,
                     smem,
                     S.core_a,
                     S.lastz_a,
                     S.lastr_a,
                     S.rd,
                     S.tt,
                     P.profiles && P.cross};
}

// Walk the block's parked packets, a warp each; then, in a run so small that its blocks started with that
// few, what is left of the ids. Not inlined: the step loop's code came out 4 % slower beside it.
template <int FAST, bool CORE, bool PROF> __device__ __noinline__ void walk_parked(const WalkParams &P, int total) {
    extern __shared__ __align__(16) unsigned long long smem[];
    const SmemLayout S = smem_layout(P);
    PlainCtx<FAST, CORE, PROF> C = plain_ctx<FAST, CORE, PROF>(P, S, smem);
    AloneState &A = *reinterpret_cast<AloneState *>(smem + S.alone);
    const unsigned lane = threadIdx.x & 31u;
    AloneTables &T = alone_tables(smem + S.ring, threadIdx.x >> 5);
    for (;;) {
        Lane M;
        const int r = next_parked(A, lane);
        if (r < total) {
            M = unpark(alone_tables(smem + S.ring, static_cast<unsigned>(r) / kAlonePerWarp).parked[r % kAlonePerWarp]);
        } else {
            if (P.lanes > alone_per_warp<FAST>()) break;
            uint32_t my = 0u;
            if (lane == 0) my = atomicAdd(P.counter, 1u);
            my = __shfl_sync(0xffffffffu, my, 0);
            if (my >= static_cast<uint32_t>(P.photons)) break;
            const uint32_t id = P.id_base + my;
            launch(M, C, id, batch_of(id, P.plan_base, P.plan_extra, P.plan_bnd), P.launch_w);
        }
        walk_alone<FAST>(M, C, lane, T);
    }
}

// ALONE: the run's last packets are walked alone (walk_step.cuh); large runs, whose end is a small part
// of them, take the kernel without it.
template <int FAST, bool CORE, bool PROF, bool ALONE>
__device__ __forceinline__ void walk_body(const WalkParams &P) {
    extern __shared__ __align__(16) unsigned long long smem[];
    const SmemLayout S = smem_layout(P);
    for (int i = S.batch + threadIdx.x; i < S.layers; i += blockDim.x) smem[i] = 0ull;
    {
        const float *src = reinterpret_cast<const float *>(P.layers);
        float *dst = reinterpret_cast<float *>(smem + S.layers);
        for (int i = threadIdx.x; i < P.nl * static_cast<int>(sizeof(LayerC) / 4); i += blockDim.x) dst[i] = src[i];
    }
    volatile AloneState &A = *reinterpret_cast<volatile AloneState *>(smem + S.alone);
    if (threadIdx.x < 8) A.live[threadIdx.x] = threadIdx.x < P.threads / 32 ? static_cast<unsigned char>(P.lanes) : 0;
    if (threadIdx.x == 0) A.next = 0u;
    __syncthreads();
    PlainCtx<FAST, CORE, PROF> C = plain_ctx<FAST, CORE, PROF>(P, S, smem);

    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;
    const uint32_t n_photons = static_cast<uint32_t>(P.photons);  // at most 2^31 (validated)
    const uint32_t chunk = static_cast<uint32_t>(P.chunk);

    WarpPool pool;                           // warp-uniform photon-id pool
    // warp-uniform: lanes with no photon left to take (from the start, those a small run leaves idle)
    unsigned ex_mask = P.lanes < 32 ? ~0u << P.lanes : 0u;
    bool alive = false;
    bool held = false;  // L holds a photon whose totals are not yet published
    Lane L;
    const int alone_at = alone_per_warp<FAST>() * static_cast<int>(P.threads / 32u);
    static_assert(kAlonePerWarp * 8 < 32, "a block with a full warp does not turn to walking alone");

    for (;;) {
        // ---- relaunch: lanes without a photon take the next ids from the warp's pool
        const unsigned need = ~__ballot_sync(0xffffffffu, alive) & ~ex_mask;
        if (need) {
            if (((need >> lane) & 1u) && held) {  // the lane's last photon ended: publish it
                finish_photon(L, C);
                held = false;
            }
            const uint32_t n = static_cast<uint32_t>(__popc(need));
            const uint32_t rank = static_cast<uint32_t>(__popc(need & lt_mask));
            uint32_t base = 0u;
            // a run too small to fill its warps' lanes claims no more ids than it launches now: what a warp
            // held in its pool, the idle lanes of others could have walked
            const uint32_t claim = P.lanes < 32 ? n : chunk;
            if (pool.must_claim(n)) {  // one lane claims the next ids for the warp
                const int leader = __ffs(need) - 1;
                if (static_cast<int>(lane) == leader) base = atomicAdd(P.counter, claim);
                base = __shfl_sync(0xffffffffu, base, leader);
            }
            const uint32_t my = pool.take(n, rank, base, claim);
            const bool mine = (need >> lane) & 1u;
            ex_mask |= __ballot_sync(0xffffffffu, mine && my >= n_photons);
            if (mine && my < n_photons) {
                const uint32_t id = P.id_base + my;  // the run's photon id: its stream and its batch
                launch(L, C, id, batch_of(id, P.plan_base, P.plan_extra, P.plan_bnd), P.launch_w);
                alive = true;
                held = true;
            }
        }
        if constexpr (ALONE) {
            // Ids have run out (or the run is small): few enough packets to walk alone? A warp that leaves holds
            // no id that it has not launched: with all 32 lanes walking, a lane is exhausted only after the
            // pool's last id, and 32 live lanes are too many; with fewer, the pool never holds any.
            if (ex_mask) {
                if (lane == 0) A.live[threadIdx.x >> 5] = static_cast<unsigned char>(__popc(~ex_mask));
                // (one decision for the warp: the lanes read the counts while other warps write them. Counts
                // only fall, so whoever sees few enough first decides for all)
                if (__any_sync(0xffffffffu, live_lanes(A) <= alone_at)) break;
            }
        } else {
            if (ex_mask == 0xffffffffu) break;  // exhausted lanes hold no photon: the warp is done
        }
        top_up<FAST>(L, C, alive);
        if (!alive) continue;
        {
            bool ended = false;
#pragma unroll
            for (int k = 0; k < steps_per_pass<FAST>(); ++k)
                if (!ended) ended = walk_step<FAST>(L, C);
            if (ended) alive = false;
        }
    }

    // ---- every lane that is not exhausted holds a packet
    if constexpr (ALONE) walk_parked<FAST, CORE, PROF>(P, park(L, C, ~ex_mask, lane, smem + S.ring, A));

    // ---- publish the block's shared tallies into the global ones (integer adds: exact)
    __syncthreads();
    const int bstride = 4 + P.nl;
    if (P.batch_smem) {
        for (int i = threadIdx.x; i < P.nb * bstride; i += blockDim.x) {
            const unsigned long long v = smem[S.batch + i];
            if (v) atomicAdd(&P.g_batch[i], v);
        }
    }
    for (int i = threadIdx.x; i < (CORE ? P.tr_a * P.tz_a : 0); i += blockDim.x) {
        const unsigned long long v = smem[S.core_a + i];
        if (v) atomicAdd(&P.g_arz[static_cast<size_t>(i / P.tz_a) * P.nz + (i % P.tz_a)], v);
    }
    if (C.cross) {
        for (int i = threadIdx.x; i < P.nr; i += blockDim.x) {
            const unsigned long long v = smem[S.lastz_a + i];
            if (v) atomicAdd(&P.g_arz[static_cast<size_t>(i) * P.nz + (P.nz - 1)], v);
        }
        for (int i = threadIdx.x; i < P.nz; i += blockDim.x) {
            const unsigned long long v = smem[S.lastr_a + i];
            if (v) atomicAdd(&P.g_arz[static_cast<size_t>(P.nr - 1) * P.nz + i], v);
        }
    }
    for (int i = threadIdx.x; i < P.tr_rd * P.na; i += blockDim.x) {
        const unsigned long long v = smem[S.rd + i];
        if (v) atomicAdd(&P.g_rd[i], v);
    }
    for (int i = threadIdx.x; i < P.tr_tt * P.na; i += blockDim.x) {
        const unsigned long long v = smem[S.tt + i];
        if (v) atomicAdd(&P.g_tt[i], v);
    }
}

// The walk of a run with profile tallies (CORE: with a shared core tile of A(r,z)).
template <int FAST, bool CORE, bool ALONE>
__global__ void TMC_WALK_BOUNDS walk_kernel(const __grid_constant__ WalkParams P) {
    walk_body<FAST, CORE, true, ALONE>(P);
}

// The walk of a run of totals only (no profile tallies).
template <int FAST, bool ALONE>
__global__ void TMC_WALK_BOUNDS walk_kernel_totals(const __grid_constant__ WalkParams P) {
    walk_body<FAST, false, false, ALONE>(P);
}

}  // namespace tmc
