// The batched sweep: thousands of independent tissue configurations in one persistent launch.
//
// No reference code exists for this (it is an addition of this engine); each configuration's
// photons follow exactly the single-run walk (walk_step.cuh) with the Philox key of that
// configuration, so a configuration's tallies are bit for bit those of a single run with the
// same seed, photons, batches and grid.
//
// A sweep with profile tallies runs in sweep_block_kernel (below, with its own comment), unless the
// options ask for a tile of A(r,z) per warp; what follows here is the kernel for that and for totals only.
//
// Work is a queue of items (configuration, first photon, count): configuration c's photons in
// items of item_photons, numbered through a prefix sum and taken band by band, in a strided
// permutation inside each band (work_queue.cuh, SweepOrder), so that the warps at work at any
// moment are spread over many configurations (their tallies then rarely meet on one L2 line). The
// host lays the configurations out longest photons first, so the bands run from the configurations
// whose photons take the most steps to those whose photons take the fewest. A warp takes items one
// at a time and hands their photons to its idle lanes; every lane carries the configuration of its
// own photon (its Philox key schedule in shared memory, written when the lane changes
// configuration; the layer table pointer; the tally base), so a warp moves on to the next item
// while some of its lanes still finish photons of the previous one, and no lane waits for an item
// to drain. Tallies of configuration c live at tally + c * stride in the single-run layout (batch
// totals, A(r,z), R_d(r,a), T_t(r,a)), accumulated with 64-bit integer atomics in global memory
// (L2).
//
// Optionally (tile_r x tile_z > 0) each warp privatises the first tile_r x tile_z bins of A(r,z) of
// one configuration, the one of the item it took last, in shared memory: deposits of its lanes'
// photons of that configuration into those bins are shared-memory atomics. When the warp takes an
// item of another configuration, it adds the tile's non-zero words into the configuration's global
// tallies and clears it (integer sums: the totals are the same whichever way they are summed).
#pragma once

#include "walk_step.cuh"
#include "work_queue.cuh"

namespace tmc {

// One configuration, as the kernel reads it.
struct SweepConfigC {
    uint32_t photons, plan_base, plan_extra, plan_bnd;  // photons and their BatchPlan
    uint32_t k0, k1;                                     // Philox key: this configuration's seed
    float launch_w;                                      // 1 - specular reflectance (float)
    int nl;                                              // layers
    int layer_base;                                      // index of layer 0 in the layer table
    uint32_t chunk;                                      // photons per chunk of the block kernel
    int pad[2];
    uint4 sched[5];                                      // the key's schedule (key_schedule_store)
};
static_assert(sizeof(SweepConfigC) == 128, "SweepConfigC layout");

// Per-sweep header in device memory (written by the sweep's host-to-device copy, so that one
// captured graph serves sweeps of different sizes).
struct SweepHeader {
    uint32_t blocks, lanes; // block kernel: blocks at work, and lanes of each warp (fewer in a small sweep)
    uint32_t n_cfg;         // configurations
    uint32_t item_photons;  // item kernel: photons per item (the last item of a configuration may hold fewer)
    SweepOrder order;       // order.total items (configuration c has ceil(photons_c / item_photons); block
                            // kernel: its chunks) and the order in which they are taken
};

struct SweepParams {
    const SweepHeader *hdr;
    const SweepConfigC *cfgs;
    const uint32_t *prefix;         // [n_cfg + 1] first item of each configuration
    const LayerC *layers;
    unsigned int *item_counter;     // next unclaimed item (zeroed before launch)
    unsigned long long *tally;      // [configs * stride]
    int stride;                     // 64-bit words per configuration
    int nb, lmax, nz, nr, na;       // batches, layer slots per batch row, grid
    float dz, dr, da, inv_dz, inv_dr, inv_da;
    int profiles;
    uint32_t step_cap;
    uint32_t threads;
    int tile_r, tile_z;             // per-warp shared tile of A(r,z) (0: none)
    int tile_words;                 // block kernel: the block's shared tile, the first words of A(r,z)
};

// The item kernel (a tile per warp, or totals only). 1: an ended packet's totals are published when its lane
// relaunches (as in the other kernels) instead of in the step. Measured on 1,024 sampled configurations: totals only
// 239.3 ms with 0, 237.4 with 1, tiles of 8 x 8 511 and 510; left at 0, as it came out ahead or level in
// earlier forms of the loop
#ifndef TMC_SWEEP_PUBLISH_AT_RELAUNCH
#define TMC_SWEEP_PUBLISH_AT_RELAUNCH 0
#endif

template <int FAST, bool TILE, bool PROF> struct SweepCtx {
    const SweepParams &P;
    Ring ring;
    uint32_t step_cap;
    int a_off, rd_off, tt_off, bstride;  // word offsets inside one configuration's tallies
    // the configuration of this lane's current photon, and its Philox key schedule (shared memory)
    uint32_t cfg;
    uint4 *sched;
    int nl;
    const LayerC *layers;
    int t;  // word offset of the configuration's tallies in P.tally (they hold < 2^31 words)
    // the warp's tile (warp-uniform): its words, and the configuration it holds (none: 0xFFFFFFFF)
    unsigned long long *tile;
    uint32_t tile_cfg;
    int tile_t;  // tally offset of tile_cfg

    // where an ended packet is published (TMC_SWEEP_PUBLISH_AT_RELAUNCH): in the step by default
    static constexpr bool kPublishAtRelaunch = TMC_SWEEP_PUBLISH_AT_RELAUNCH != 0;

    __device__ __forceinline__ void refill(Lane &L) const { ring.refill(L, [&](int q) { return sched[q * static_cast<int>(P.threads)]; }); }
    __device__ __forceinline__ void refill2(Lane &L) const { ring.refill2(L, [&](int q) { return sched[q * static_cast<int>(P.threads)]; }); }
    __device__ __forceinline__ float path(const Lane &L, const Hot &h) const { return step_length<FAST>(h, unit_open(ring.peek(L))); }
    __device__ __forceinline__ float unit(Lane &L) const { return unit_open(ring.draw(L)); }
    __device__ __forceinline__ void skip(Lane &L) const { ring.skip(L); }
    __device__ __forceinline__ void pass(Lane &L, uint32_t n) const { L.rp += n; }
    __device__ __forceinline__ void scatter(Lane &L, const Hot &h, float dwa) const { scatter_now<FAST>(L, *this, h, dwa); }
    __device__ __forceinline__ void leave_layer(Lane &) const {}
    __device__ __forceinline__ void enter_layer(Lane &) const {}
    __device__ __forceinline__ const LayerC &layer(const Lane &, int l) const { return layers[l]; }
    __device__ __forceinline__ int num_layers(const Lane &) const { return nl; }
    __device__ __forceinline__ void batch_add(const Lane &L, int slot, unsigned long long v) const {
        atomicAdd(&P.tally[t + L.batch * bstride + slot], v);
    }
    __device__ __forceinline__ void absorb(float2 xy, float z, unsigned long long v) const {
        if constexpr (!PROF) return;
        const float rr = radius<FAST>(xy);
        int ir, iz;
        bins_rz<FAST>(rr, z, P.dr, P.dz, P.inv_dr, P.inv_dz, P.nr, P.nz, ir, iz);
        if (TILE && cfg == tile_cfg && ir < P.tile_r && iz < P.tile_z) atomicAdd(&tile[ir * P.tile_z + iz], v);
        else atomicAdd(&P.tally[t + a_off + ir * P.nz + iz], v);
    }
    // Whole warp: hand the tile's sums to the global tallies of its configuration and clear it.
    __device__ __forceinline__ void flush_tile(unsigned lane) {
        __syncwarp();
        if (tile_cfg != 0xFFFFFFFFu) {
            for (int i = static_cast<int>(lane); i < P.tile_r * P.tile_z; i += 32) {
                const unsigned long long w = tile[i];
                if (w) {
                    atomicAdd(&P.tally[tile_t + a_off + (i / P.tile_z) * P.nz + i % P.tile_z], w);
                    tile[i] = 0ull;
                }
            }
        }
        __syncwarp();
    }
    __device__ __forceinline__ void exit(const Lane &L, int kind, unsigned long long v) const {
        if constexpr (!PROF) return;
        const float rr = radius<FAST>(L.xy);
        const int ir = bin_of<FAST>(rr, P.dr, P.inv_dr, P.nr);
        const int ia = P.na > 1 ? bin_of<FAST>(acosf(fminf(fabsf(L.uz), 1.0f)), P.da, P.inv_da, P.na) : 0;
        atomicAdd(&P.tally[t + (kind == 1 ? rd_off : tt_off) + ir * P.na + ia], v);
    }
};

// Minimum resident 256-thread blocks per SM the compiler must allow for (0: no bound). Three allow 80
// registers; four (64) spilled in the step loop: the block kernel on 4096 configurations 1.44 s with four,
// 1.22 s with three, 1.24 s without a bound (92 registers, two blocks). The step's arithmetic has its
// rounding pinned (walk.cuh), so the register budget cannot change any photon's path: the tallies stay
// bit-identical to the single-run kernel's.
#ifndef TMC_SWEEP_MIN_BLOCKS
#define TMC_SWEEP_MIN_BLOCKS 3
#endif
#if TMC_SWEEP_MIN_BLOCKS > 0
#define TMC_SWEEP_BOUNDS __launch_bounds__(256, TMC_SWEEP_MIN_BLOCKS)
#else
#define TMC_SWEEP_BOUNDS __launch_bounds__(256)
#endif

// TILE: the per-warp shared tile of A(r,z) is on (P.tile_r, P.tile_z > 0); the kernel without it
// (sweeps of totals only) is a separate instantiation.
template <int FAST, bool TILE, bool PROF>
__device__ __forceinline__ void sweep_body(const SweepParams &P) {
    extern __shared__ __align__(16) unsigned long long smem[];
    SweepCtx<FAST, TILE, PROF> C{P,
                     Ring{reinterpret_cast<uint32_t *>(smem) + ring_lane_offset()},
                     P.step_cap,
                     P.nb * (4 + P.lmax),
                     P.nb * (4 + P.lmax) + P.nr * P.nz,
                     P.nb * (4 + P.lmax) + P.nr * P.nz + P.nr * P.na,
                     4 + P.lmax,
                     0xFFFFFFFFu,
                     // after the rings (kRingWords words per lane): 5 x 16 bytes of key schedule per lane
                     reinterpret_cast<uint4 *>(reinterpret_cast<uint32_t *>(smem) + kRingWords * P.threads) +
                         threadIdx.x,
                     1,
                     P.layers,
                     0,
                     // after the key schedules: one tile per warp
                     reinterpret_cast<unsigned long long *>(reinterpret_cast<uint32_t *>(smem) +
                                                            (kRingWords + 20) * P.threads) +
                         static_cast<size_t>(threadIdx.x >> 5) * P.tile_r * P.tile_z,
                     0xFFFFFFFFu,
                     0};
    const unsigned lane = threadIdx.x & 31u;
    if constexpr (TILE) {
        for (int i = static_cast<int>(lane); i < P.tile_r * P.tile_z; i += 32) C.tile[i] = 0ull;
        __syncwarp();
    }
    const unsigned lt_mask = (1u << lane) - 1u;
    const SweepHeader &H = *P.hdr;  // read where an item is taken (rare), not held in registers

    // warp-uniform: the item being handed out
    uint32_t it_cfg = 0u, it_next = 0u, it_end = 0u;
    bool items_done = false;
    unsigned ex_mask = 0u;  // warp-uniform: lanes with no photon left to take
    bool alive = false;
    bool held = false;  // L holds an ended photon whose totals are not yet published
    Lane L;

    for (;;) {
        unsigned need = ~__ballot_sync(0xffffffffu, alive) & ~ex_mask;
        if constexpr (decltype(C)::kPublishAtRelaunch) {
            if (((need >> lane) & 1u) && held) {  // the lane's last photon ended: publish it
                finish_photon(L, C);
                held = false;
            }
        }
        while (need) {  // warp-uniform: hand out photons, taking new items as they run out
            const uint32_t avail = it_end - it_next;
            if (avail == 0u) {
                if (!items_done) {
                    const int leader = __ffs(need) - 1;
                    uint32_t idx = 0u;
                    if (static_cast<int>(lane) == leader) idx = atomicAdd(P.item_counter, 1u);
                    idx = __shfl_sync(0xffffffffu, idx, leader);
                    if (idx < H.order.total) {
                        sweep_item(idx, H.order, H.item_photons, H.n_cfg, P.prefix,
                                   [&](uint32_t c) { return P.cfgs[c].photons; }, it_cfg, it_next, it_end);
                        if (TILE && it_cfg != C.tile_cfg) {  // the tile follows the warp's item
                            C.flush_tile(lane);
                            C.tile_cfg = it_cfg;
                            C.tile_t = static_cast<int>(it_cfg) * P.stride;
                        }
                        continue;
                    }
                    items_done = true;
                }
                ex_mask |= need;
                break;
            }
            const uint32_t n = static_cast<uint32_t>(__popc(need));
            const uint32_t take = n < avail ? n : avail;
            const uint32_t rank = static_cast<uint32_t>(__popc(need & lt_mask));
            const bool mine = ((need >> lane) & 1u) && rank < take;
            if (mine) {
                const SweepConfigC cf = P.cfgs[it_cfg];
                const uint32_t id = it_next + rank;
                if (it_cfg != C.cfg) {  // the lane's key schedule follows its configuration
                    C.cfg = it_cfg;
                    key_schedule_store(C.sched, static_cast<int>(P.threads), cf.k0, cf.k1);
                }
                C.nl = cf.nl;
                C.layers = P.layers + cf.layer_base;
                C.t = static_cast<int>(it_cfg) * P.stride;
                const int batch = batch_of(id, cf.plan_base, cf.plan_extra, cf.plan_bnd);
                launch(L, C, id, batch, cf.launch_w);
                alive = true;
                held = true;
            }
            need &= ~__ballot_sync(0xffffffffu, mine);
            it_next += take;
        }
        if (ex_mask == 0xffffffffu) break;  // exhausted lanes hold no photon: the warp is done
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
    if constexpr (TILE) C.flush_tile(lane);
}

// The sweep with profile tallies and the per-warp shared tile of A(r,z) that the options ask for.
template <int FAST>
__global__ void TMC_SWEEP_BOUNDS sweep_kernel(const __grid_constant__ SweepParams P) {
    sweep_body<FAST, true, true>(P);
}

// The sweep of totals only (no profile tallies).
template <int FAST>
__global__ void TMC_SWEEP_BOUNDS sweep_kernel_totals(const __grid_constant__ SweepParams P) {
    sweep_body<FAST, false, false>(P);
}

// ------------------------------------------------------------------------------ the block kernel
// The sweep whose blocks work on one configuration at a time, with the leading rows of its A(r,z) (all
// of a 64 x 64 grid) in shared memory, and walk their last packets alone (walk_step.cuh): a sweep lasts as
// long as its longest photon, and in a thick, weakly absorbing slab one takes a hundred thousand steps.
// Against items of 256 photons per warp, every deposit in L2: 97 configurations of 1e3 photons 13.6 ->
// 3.3 ms, of 1e5 48 -> 21 ms, 1024 of 1e5 166 -> 135 ms, 4096 of 1e4 to 1e6 1.30 -> 1.23 s.
//
// A block takes chunks (configuration, first photon, count) from the launch's counter, in the order of
// the item queue; its warps hand the chunk's photons to their idle lanes. When the chunk runs out the
// block switches: at the top of a pass all warps meet, the tile's sums go to the old configuration's
// tallies (unless the next chunk is the same configuration's) and the warps go on. Lanes still walking
// photons of an earlier configuration are not waited for; their deposits go to global memory. A chunk
// holds at most a block's share of the work, by the estimate the queue is ordered by (sweep.cu); a switch
// takes two or three microseconds. Warp 0 fetches the next chunk while the block works.
template <int FAST> struct BlockSweepCtx {
    const SweepParams &P;
    Ring ring;
    uint32_t step_cap;
    int a_off, rd_off, tt_off, bstride;
    uint32_t cfg;         // the configuration of this lane's photon
    const LayerC *layers; // its layers
    unsigned long long *words;  // the block's tile through a generic address (one native 64-bit atomic)
    uint32_t tile_cfg;    // the configuration the tile belongs to
    static constexpr bool kPublishAtRelaunch = true;

    __device__ __forceinline__ uint4 key(int q) const { return __ldg(&P.cfgs[cfg].sched[q]); }
    __device__ __forceinline__ void refill(Lane &L) const { ring.refill(L, [&](int q) { return key(q); }); }
    __device__ __forceinline__ void refill2(Lane &L) const { ring.refill2(L, [&](int q) { return key(q); }); }
    __device__ __forceinline__ void block(uint32_t id, uint32_t blk, uint32_t &w0, uint32_t &w1, uint32_t &w2, uint32_t &w3) const {
        philox4x32_10_sched(id, 0u, blk, [&](int q) { return key(q); }, w0, w1, w2, w3);
    }
    __device__ __forceinline__ uint32_t tag() const { return cfg; }
    __device__ __forceinline__ void adopt(uint32_t its_cfg) {
        cfg = its_cfg;
        layers = P.layers + P.cfgs[cfg].layer_base;
    }
    __device__ __forceinline__ float path(const Lane &L, const Hot &h) const { return step_length<FAST>(h, unit_open(ring.peek(L))); }
    __device__ __forceinline__ float unit(Lane &L) const { return unit_open(ring.draw(L)); }
    __device__ __forceinline__ void skip(Lane &L) const { ring.skip(L); }
    __device__ __forceinline__ void pass(Lane &L, uint32_t n) const { L.rp += n; }
    __device__ __forceinline__ void scatter(Lane &L, const Hot &h, float dwa) const { scatter_now<FAST>(L, *this, h, dwa); }
    __device__ __forceinline__ void leave_layer(Lane &) const {}
    __device__ __forceinline__ void enter_layer(Lane &) const {}
    __device__ __forceinline__ const LayerC &layer(const Lane &, int l) const { return layers[l]; }
    __device__ __forceinline__ int num_layers(const Lane &) const { return __ldg(&P.cfgs[cfg].nl); }
    // the sweep's tallies hold fewer than 2^31 words
    __device__ __forceinline__ int base() const { return static_cast<int>(cfg) * P.stride; }
    __device__ __forceinline__ void batch_add(const Lane &L, int slot, unsigned long long v) const {
        atomicAdd(&P.tally[base() + L.batch * bstride + slot], v);
    }
    __device__ __forceinline__ void absorb(float2 xy, float z, unsigned long long v) const {
        const float rr = radius<FAST>(xy);
        int ir, iz;
        bins_rz<FAST>(rr, z, P.dr, P.dz, P.inv_dr, P.inv_dz, P.nr, P.nz, ir, iz);
        const int w = ir * P.nz + iz;
        const bool shared = cfg == tile_cfg && w < P.tile_words;
        atomicAdd((shared ? words : P.tally) + (shared ? w : base() + a_off + w), v);
    }
    __device__ __forceinline__ void exit(const Lane &L, int kind, unsigned long long v) const {
        const float rr = radius<FAST>(L.xy);
        const int ir = bin_of<FAST>(rr, P.dr, P.inv_dr, P.nr);
        const int ia = P.na > 1 ? bin_of<FAST>(acosf(fminf(fabsf(L.uz), 1.0f)), P.da, P.inv_da, P.na) : 0;
        atomicAdd(&P.tally[base() + (kind == 1 ? rd_off : tt_off) + ir * P.na + ia], v);
    }
};

constexpr uint32_t kNoConfig = 0xFFFFFFFFu;

// The block's state after its rings and tile, in shared memory.
struct BlockSweepState {
    uint32_t cfg, next, end;           // the chunk being handed out
    uint32_t want_switch;              // a warp found it used up
    uint32_t up_cfg, up_next, up_end;  // the chunk after it (up_cfg = kNoConfig: there is none)
    uint32_t pad;
    AloneState alone;
};

// The block's shared memory after its rings: the tile, then the state.
__device__ __forceinline__ unsigned long long *block_tile(const SweepParams &P, unsigned long long *smem) {
    return smem + kRingWords / 2 * P.threads;
}
__device__ __forceinline__ BlockSweepState &block_state(const SweepParams &P, unsigned long long *smem) {
    return *reinterpret_cast<BlockSweepState *>(block_tile(P, smem) + ((P.tile_words + 1) & ~1));
}
template <int FAST> __device__ __forceinline__ BlockSweepCtx<FAST> block_ctx(const SweepParams &P, unsigned long long *smem, uint32_t tile_cfg) {
    const int a_off = P.nb * (4 + P.lmax);
    return BlockSweepCtx<FAST>{P,
                               Ring{reinterpret_cast<uint32_t *>(smem) + ring_lane_offset()},
                               P.step_cap,
                               a_off,
                               a_off + P.nr * P.nz,
                               a_off + P.nr * P.nz + P.nr * P.na,
                               4 + P.lmax,
                               0u,
                               P.layers,
                               block_tile(P, smem),
                               tile_cfg};
}

// Walk the block's parked packets, a warp each (not inlined: the step loop keeps its registers and code).
template <int FAST> __device__ __noinline__ void sweep_parked(const SweepParams &P, uint32_t tile_cfg, int total) {
    extern __shared__ __align__(16) unsigned long long smem[];
    BlockSweepCtx<FAST> C = block_ctx<FAST>(P, smem, tile_cfg);
    BlockSweepState &S = block_state(P, smem);
    const unsigned lane = threadIdx.x & 31u;
    AloneTables &T = alone_tables(smem, threadIdx.x >> 5);
    for (;;) {
        const int r = next_parked(S.alone, lane);
        if (r >= total) break;
        const Parked &k = alone_tables(smem, static_cast<unsigned>(r) / kAlonePerWarp).parked[r % kAlonePerWarp];
        Lane M = unpark(k);
        C.adopt(k.tag);
        walk_alone<FAST>(M, C, lane, T);
    }
}

template <int FAST> __global__ void TMC_SWEEP_BOUNDS sweep_block_kernel(const __grid_constant__ SweepParams P) {
    extern __shared__ __align__(16) unsigned long long smem[];
    const SweepHeader &H = *P.hdr;
    if (blockIdx.x >= H.blocks) return;
    unsigned long long *const tile = block_tile(P, smem);
    volatile BlockSweepState &S = block_state(P, smem);
    BlockSweepCtx<FAST> C = block_ctx<FAST>(P, smem, kNoConfig);
    const int a_off = C.a_off;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned lt_mask = (1u << lane) - 1u;

    // warp 0: the block's next chunk
    const auto fetch = [&]() {
        if (lane != 0) return;
        const uint32_t idx = atomicAdd(P.item_counter, 1u);
        if (idx >= H.order.total) {
            S.up_cfg = kNoConfig;
            return;
        }
        const uint32_t j = H.order.item(idx), c = sweep_owner(j, H.n_cfg, P.prefix);
        const uint32_t chunk = P.cfgs[c].chunk, first = (j - P.prefix[c]) * chunk, left = P.cfgs[c].photons - first;
        S.up_cfg = c;
        S.up_next = first;
        S.up_end = first + (left < chunk ? left : chunk);
    };
    // whole block: the tile's sums into its configuration's tallies, and clear it
    const auto flush = [&]() {
        if (C.tile_cfg == kNoConfig) return;
        unsigned long long *const a = P.tally + static_cast<size_t>(C.tile_cfg) * P.stride + a_off;
        for (int i = static_cast<int>(threadIdx.x); i < P.tile_words; i += static_cast<int>(blockDim.x)) {
            const unsigned long long w = tile[i];
            if (w) {
                atomicAdd(a + i, w);
                tile[i] = 0ull;
            }
        }
    };
    for (int i = static_cast<int>(threadIdx.x); i < P.tile_words; i += static_cast<int>(blockDim.x)) tile[i] = 0ull;
    if (threadIdx.x == 0) {
        S.next = S.end = 0u;
        S.want_switch = 1u;
        S.alone.next = 0u;
    }
    if (threadIdx.x < 8) S.alone.live[threadIdx.x] = threadIdx.x < P.threads / 32 ? 32 : 0;
    if (threadIdx.x < 32) fetch();
    __syncthreads();

    bool done = false;  // block-uniform: no chunk is left to take
    unsigned ex_mask = H.lanes < 32u ? ~0u << H.lanes : 0u;  // warp-uniform: lanes with no photon left to take
    bool alive = false;
    bool held = false;  // L holds an ended photon whose totals are not yet published
    Lane L;
    const int alone_at = alone_per_warp<FAST>() * static_cast<int>(P.threads / 32u);

    for (;;) {
        if (__any_sync(0xffffffffu, S.want_switch != 0u)) {  // set between two switches: every warp comes here once
            __syncthreads();  // no warp is depositing or handing out photons
            const uint32_t c = S.up_cfg;
            if (c == kNoConfig) {
                done = true;
            } else {
                if (c != C.tile_cfg) flush();
                C.tile_cfg = c;
            }
            if (threadIdx.x == 0) {
                S.cfg = c;
                S.next = S.up_next;
                S.end = S.up_end;
                S.want_switch = 0u;
            }
            __syncthreads();
            if (threadIdx.x < 32 && !done) fetch();
            __syncwarp();
        }
        const unsigned need = ~__ballot_sync(0xffffffffu, alive) & ~ex_mask;
        if (need) {
            const bool wants = (need >> lane) & 1u;
            if (wants && held) {  // the lane's last photon ended: publish it
                finish_photon(L, C);
                held = false;
            }
            if (done) {
                ex_mask |= need;
            } else {
                const uint32_t n = static_cast<uint32_t>(__popc(need));
                const uint32_t rank = static_cast<uint32_t>(__popc(need & lt_mask));
                uint32_t first = 0u;
                if (lane == 0) first = atomicAdd(const_cast<uint32_t *>(&S.next), n);
                first = __shfl_sync(0xffffffffu, first, 0);
                const uint32_t end = S.end, avail = first < end ? end - first : 0u;
                if (wants && rank < avail) {
                    C.cfg = C.tile_cfg;
                    const SweepConfigC &cf = P.cfgs[C.cfg];
                    C.layers = P.layers + cf.layer_base;
                    const uint32_t id = first + rank;
                    launch(L, C, id, batch_of(id, cf.plan_base, cf.plan_extra, cf.plan_bnd), cf.launch_w);
                    alive = true;
                    held = true;
                }
                if (avail < n && lane == 0) S.want_switch = 1u;
                __syncwarp();
            }
        }
        if (done) {  // no chunk is left: few enough packets to walk alone?
            if (lane == 0) S.alone.live[threadIdx.x >> 5] = static_cast<unsigned char>(__popc(~ex_mask));
            if (__any_sync(0xffffffffu, live_lanes(S.alone) <= alone_at)) break;  // one decision for the warp
        }
        top_up<FAST>(L, C, alive);
        if (!alive) continue;
        bool ended = false;
#pragma unroll
        for (int k = 0; k < steps_per_pass<FAST>(); ++k)
            if (!ended) ended = walk_step<FAST>(L, C);
        if (ended) alive = false;
    }
    // every lane that is not exhausted holds a packet
    sweep_parked<FAST>(P, C.tile_cfg, park(L, C, ~ex_mask, lane, smem, S.alone));
    __syncthreads();
    flush();
}

// Per-configuration summaries from the integer tallies, in double: R_d(r) per photon (nr values,
// summed over exit angles), then total R_d, T_t and absorbed weight per photon. One warp per
// configuration; deterministic (integer sums, converted once).
__global__ void sweep_finalize_kernel(const SweepConfigC *cfgs, const unsigned long long *tally, int n_cfg,
                                      int stride, int nb, int lmax, int nz, int nr, int na, double *summary) {
    const int warp = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (warp >= n_cfg) return;
    const unsigned long long *t = tally + static_cast<size_t>(warp) * stride;
    const int bstride = 4 + lmax;
    const int rd_off = nb * bstride + nr * nz;
    const double k = 1.0 / (4294967296.0 * static_cast<double>(cfgs[warp].photons));
    double *out = summary + static_cast<size_t>(warp) * (nr + 3);
    for (int ir = lane; ir < nr; ir += 32) {
        unsigned long long s = 0ull;
        for (int ia = 0; ia < na; ++ia) s += t[rd_off + ir * na + ia];
        out[ir] = static_cast<double>(s) * k;
    }
    unsigned long long rd = 0ull, tt = 0ull, ab = 0ull;
    for (int b = lane; b < nb; b += 32) {
        rd += t[b * bstride + 0];
        tt += t[b * bstride + 1];
        for (int l = 0; l < lmax; ++l) ab += t[b * bstride + 4 + l];
    }
    for (int o = 16; o > 0; o >>= 1) {
        rd += __shfl_down_sync(0xffffffffu, rd, o);
        tt += __shfl_down_sync(0xffffffffu, tt, o);
        ab += __shfl_down_sync(0xffffffffu, ab, o);
    }
    if (lane == 0) {
        out[nr] = static_cast<double>(rd) * k;
        out[nr + 1] = static_cast<double>(tt) * k;
        out[nr + 2] = static_cast<double>(ab) * k;
    }
}

}  // namespace tmc
