// One MCML step of one lane, shared by the single-run kernel (walk_kernel.cuh) and the
// multi-configuration sweep kernel (sweep_kernel.cuh).
//
// Step semantics: TissueMC's include/tissuemc/physics.hpp — step size :148-158, boundary distance
// :162-178, hop :180-184, drop :187-193, Henyey-Greenstein :101-113, spin :116-144, Fresnel
// :71-98, crossing :198-246, roulette :250-259, step_once :263-277. A kernel supplies a context
// `Ctx` that says where the layer table and the tallies live:
//   ctx.refill(lane)          append the lane's next Philox block to its random-word ring
//   ctx.path(lane, h)         the free path of the next random word, which stays unread
//   ctx.unit(lane)            the next random word as a float in (0, 1); ctx.skip(lane) passes over it,
//                             ctx.pass(lane, n) over the next n
//   ctx.layer(lane, l)        constants of layer l of the lane's tissue
//   ctx.num_layers(lane)
//   ctx.scatter(lane, dwa)    score an absorption of weight dwa at the lane's position and turn its
//                             direction by the next two random words
//   ctx.absorb(xy, z, v)      add v (fixed point) to A(r,z) at a position
//   ctx.exit(lane, kind, v)   score an exit (1: reflectance, 2: transmittance) of v
//   ctx.batch_add(lane, i, v) add v to slot i of the lane's batch totals
//   ctx.leave_layer(lane), ctx.enter_layer(lane)   before and after a packet changes layer
//   ctx.step_cap              steps after which a packet is ended as an anomaly
//   Ctx::kPublishAtRelaunch   true: the kernel publishes an ended packet's totals (finish_photon)
//                             when the lane relaunches; false: the step does
#pragma once

#include "walk.cuh"

namespace tmc {

// Steps a lane takes per pass of a kernel's persistent loop: the relaunch ballot, the lane's live test
// and the random words' top-up once per pass; a lane whose packet ends early in a pass waits out the
// rest of it. Fast math, skin5, 2e7 photons: 2 107.6 ms, 3 105.4 ms (4: a sixth slower, the loop body four
// steps long). Exact math, whose step is
// twice as long, three layers, 3e6 photons: 1 4.86 ms, 2 4.90 ms, 3 5.51 ms; slab, 3e5: 475, 444, 459 us.
template <int FAST> __device__ __forceinline__ constexpr int steps_per_pass() { return FAST ? 3 : 2; }
// Random words a lane keeps in its shared-memory ring. Before a pass every lane is topped up to the most
// that the pass may draw (4 a step), four at a time (one Philox block): while any lane of the
// warp is short, every lane with room for a block takes one, so the lanes of a warp refill together.
// The words each photon consumes, and their order, do not depend on it.
constexpr uint32_t kRingWords = 16;

constexpr float kCosZero = 1.0f - 1e-6f;  // physics.hpp:35 (float widening of MCML COSZERO)
constexpr float kCos90D = 1e-6f;          // physics.hpp:36
constexpr float kWeightMin = 1e-4f;       // physics.hpp:33 (MCML WEIGHT)
constexpr float kChance = 0.1f;           // physics.hpp:34 (MCML CHANCE)
constexpr float kTwoPi = 2.0f * 3.14159265358979323846f;  // evaluated as the reference does

// Register copy of the current layer's constants used on every step.
struct Hot {
    float mua, mut, inv_mut, absorb, z0, z1, g, hg_a, hg_b, hg_c, hg_d, inv_2g;
};

__device__ __forceinline__ void load_hot(Hot &h, const LayerC &L) {
    const float4 *q = reinterpret_cast<const float4 *>(&L);  // three 16-byte loads
    const float4 a = q[0], b = q[1], c = q[2];
    h.inv_mut = a.x;
    h.absorb = a.y;
    h.z0 = a.z;
    h.z1 = a.w;
    h.g = b.x;
    h.hg_a = b.y;
    h.hg_b = b.z;
    h.hg_c = b.w;
    h.hg_d = c.x;
    h.inv_2g = c.y;
    h.mut = c.z;
    h.mua = c.w;
}

// The boundary of layer L toward the top (up) or the bottom: the neighbour's index, the index
// ratio, the critical cosine and the normal-incidence reflectance, in one 16-byte load.
__device__ __forceinline__ float4 boundary_side(const LayerC &L, bool up) {
    return reinterpret_cast<const float4 *>(&L)[up ? 3 : 4];
}

// Fresnel reflectance for unpolarised light from index n1 into n2 at cos(incidence) ca1
// (physics.hpp:71-98); rn is the precomputed normal-incidence value and rat = n1 / n2.
template <int FAST>
__device__ __forceinline__ float fresnel(float n1, float n2, float ca1, float rn, float rat,
                                         float &ca2) {
    if (n1 == n2) {
        ca2 = ca1;
        return 0.0f;
    }
    if (ca1 > kCosZero) {
        ca2 = ca1;
        return rn;
    }
    if (ca1 < kCos90D) {
        ca2 = 0.0f;
        return 1.0f;
    }
    const float sa1 = m_sqrt<FAST>(ffma(-ca1, ca1, 1.0f));
    float sa2;
    if constexpr (Math<FAST>::div) sa2 = fmul(sa1, rat);
    else sa2 = fmul(n1, sa1) / n2;
    if (sa2 >= 1.0f) {
        ca2 = 0.0f;
        return 1.0f;
    }
    ca2 = m_sqrt<FAST>(ffma(-sa2, sa2, 1.0f));
    const float cc = fmul(ca1, ca2), ss = fmul(sa1, sa2), sc = fmul(sa1, ca2), cs = fmul(ca1, sa2);
    const float cap = fsub(cc, ss), cam = fadd(cc, ss), sap = fadd(sc, cs), sam = fsub(sc, cs);
    return m_div<FAST>(fmul(fmul(fmul(0.5f, sam), sam), norm2(cam, cap)), fmul(fmul(sap, sap), fmul(cam, cam)));
}

// Clamped bin index (src/cpu/engine.cpp:59-66 semantics, branch-free): x <= 0 or NaN -> 0,
// x / width >= n -> n - 1, else floor(x / width).
// The clamp is the conversion's own: a float-to-unsigned conversion that truncates turns negative
// values and NaN into 0 and saturates large ones, so min(u, n - 1) is the clamped bin.
__device__ __forceinline__ int clamp_bin(float i, int n) {
    return static_cast<int>(umin(__float2uint_rz(i), static_cast<unsigned>(n - 1)));
}
template <int FAST> __device__ __forceinline__ int bin_of(float x, float width, float inv_width, int n) {
    float i;
    if constexpr (Math<FAST>::div) i = fmul(x, inv_width);
    else i = x / width;
    return clamp_bin(i, n);
}
// The radius and depth bins of one deposit (r, z) together: in fast math the two products are one
// paired instruction.
template <int FAST>
__device__ __forceinline__ void bins_rz(float r, float z, float dr, float dz, float inv_dr, float inv_dz, int nr, int nz,
                                        int &ir, int &iz) {
    if constexpr (Math<FAST>::div) {
        const float2 i = fmul2(f2(r, z), f2(inv_dr, inv_dz));
        ir = clamp_bin(i.x, nr);
        iz = clamp_bin(i.y, nz);
    } else {
        ir = bin_of<FAST>(r, dr, inv_dr, nr);
        iz = bin_of<FAST>(z, dz, inv_dz, nz);
    }
}

// Free path -ln(u) / mu_t of an interaction step (physics.hpp:148-158), as -ln(u) and its scaling.
template <int FAST> __device__ __forceinline__ float minus_log(float u) {
    // the SFU logarithm's absolute error can flip the sign of log(u) for the two largest u of the
    // 23-bit grid; a step is never negative
    if constexpr (Math<FAST>::log) return fmaxf(-m_log<FAST>(u), 0.0f);
    else return -m_log<FAST>(u);
}
template <int FAST> __device__ __forceinline__ float scale_path(const Hot &h, float e) {
    if constexpr (Math<FAST>::div) return fmul(e, h.inv_mut);
    else return e / h.mut;
}
template <int FAST> __device__ __forceinline__ float step_length(const Hot &h, float u) {
    return scale_path<FAST>(h, minus_log<FAST>(u));
}

// Henyey-Greenstein cosine of the scattering angle from one uniform draw (physics.hpp:101-113).
template <int FAST> __device__ __forceinline__ float hg_cos(const Hot &h, float xi) {
    const float t = m_div<FAST>(h.hg_a, ffma(h.hg_c, xi, h.hg_b));
    float ct;
    if constexpr (Math<FAST>::div) ct = fmul(ffma(-t, t, h.hg_d), h.inv_2g);
    else ct = ffma(-t, t, h.hg_d) / h.hg_c;
    // an isotropic layer selects 2 xi - 1 (the formula above is 0 / 0 there, clamped, then
    // discarded): a select instead of a branch, measured 1.0 % faster on skin5
    return h.g == 0.0f ? ffma(2.0f, xi, -1.0f) : fminf(fmaxf(ct, -1.0f), 1.0f);
}

// Sine of the scattering angle from its cosine.
template <int FAST> __device__ __forceinline__ float sin_of(float ct) {
    return m_sqrt<FAST>(fmaxf(ffma(-ct, ct, 1.0f), 0.0f));
}
// Sine and cosine of the azimuth 2 pi u.
template <int FAST> __device__ __forceinline__ void azimuth(float u, float &sp, float &cp) {
    if constexpr (Math<FAST>::sincos) {
        // psi - pi lies in (-pi, pi), where the SFU sine and cosine are accurate
        __sincosf(fmul(kTwoPi, fsub(u, 0.5f)), &sp, &cp);
        sp = -sp;
        cp = -cp;
    } else {
        sincosf(fmul(kTwoPi, u), &sp, &cp);
    }
}

// Turn the direction (u.x, u.y, uz) by the polar angle (ct, st) and the azimuth (cp, sp), then renormalise
// it (physics.hpp:116-144). The x and y halves go through paired instructions, each half rounded as
// the scalar form would round it. A direction along z (|uz| > kCosZero) has a form of its own.
// nstcp = -st cp.
template <int FAST> __device__ __forceinline__ void renormalise(float2 &uxy, float &uz) {
    const float inv = m_rsqrt<FAST>(norm2(uxy, uz));
    uxy = fmul2(uxy, f2(inv));
    uz = fmul(uz, inv);
}
template <int FAST>
__device__ __forceinline__ void turn_oblique(float2 &uxy, float &uz, float ct, float st, float cp, float sp, float nstcp) {
    const float2 o = uxy;
    const float oz = uz;
    const float q = ffma(-oz, oz, 1.0f);  // 1 - uz^2
    // (ix, iy) = (ox oz cp - oy sp, oy oz cp + ox sp)
    const float2 ixy = ffma2(fmul2(o, f2(oz)), f2(cp), fmul2(f2(-o.y, o.x), f2(sp)));
    const float2 oct = fmul2(o, f2(ct));
    if constexpr (Math<FAST>::sqrt) {
        const float it = m_rsqrt<FAST>(q);
        uxy = ffma2(fmul2(f2(st), ixy), f2(it), oct);
        uz = ffma(fmul(nstcp, q), it, fmul(oz, ct));
    } else {
        const float tmp = sqrtf(q);
        uxy = f2(fadd(fmul(st, ixy.x) / tmp, oct.x), fadd(fmul(st, ixy.y) / tmp, oct.y));
        uz = ffma(nstcp, tmp, fmul(oz, ct));
    }
    renormalise<FAST>(uxy, uz);
}
template <int FAST>
__device__ __forceinline__ void turn(float2 &uxy, float &uz, float ct, float st, float cp, float sp) {
    if (fabsf(uz) > kCosZero) {
        uxy = fmul2(f2(st), f2(cp, sp));
        uz = uz >= 0.0f ? ct : -ct;
        renormalise<FAST>(uxy, uz);
    } else {
        turn_oblique<FAST>(uxy, uz, ct, st, cp, sp, fmul(-st, cp));
    }
}

// The same from the polar cosine and the uniform draw of the azimuth.
template <int FAST> __device__ __forceinline__ void rotate(float2 &uxy, float &uz, float ct, float u) {
    float sp, cp;
    azimuth<FAST>(u, sp, cp);
    turn<FAST>(uxy, uz, ct, sin_of<FAST>(ct), cp, sp);
}

// Radial distance of the packet from the source axis (the r of A(r,z), R_d(r,a), T_t(r,a)).
template <int FAST> __device__ __forceinline__ float radius(float2 xy) { return m_sqrt<FAST>(norm2(xy)); }

// All state of one lane's current photon (registers).
struct Lane {
    float2 xy;   // position across the layers (x, y) [cm]
    float2 uxy;  // direction cosines (ux, uy)
    float z, uz, w, sleft;
    int layer, batch;
    uint32_t id, blk, rp, wp;  // photon id, Philox block, ring read/write positions
    uint32_t events, anomalies, steps;
    unsigned long long run_abs;  // fixed-point weight absorbed in the current layer
    Hot h;
};

// Launch a packet at the origin, straight down, in layer 0 (physics.hpp:58-66).
template <class Ctx>
__device__ __forceinline__ void launch(Lane &L, Ctx &C, uint32_t id, int batch, float launch_w) {
    L.id = id;
    L.blk = 0u;
    L.rp = L.wp = 0u;
    L.xy = f2(0.f);
    L.z = 0.f;
    L.uxy = f2(0.f);
    L.uz = 1.f;
    L.w = launch_w;
    L.sleft = 0.f;
    L.layer = 0;
    load_hot(L.h, C.layer(L, 0));
    L.batch = batch;
    L.events = L.anomalies = L.steps = 0u;
    L.run_abs = 0ull;
}

// Score and publish an ended packet: its exit (check, totals, R_d(r,a) or T_t(r,a)), its events,
// anomalies and the weight absorbed in its last layer. An ended packet's `steps` says how it ended (0:
// inside, 1: reflectance, 2: transmittance). Once per pass for every lane that ended in it, instead of
// in the step with a lane or two: slab (22 steps a photon), 1e7 photons 3.14 -> 2.92 ms.
template <class Ctx> __device__ __forceinline__ void finish_photon(Lane &L, Ctx &C) {
    if (L.steps != 0u) {
        const float n2 = norm2(L.uxy, L.uz);
        if (!(L.w == L.w) || !(fabsf(fsub(n2, 1.0f)) <= 1e-5f)) ++L.anomalies;
        const unsigned long long v = to_fixed(L.w);
        C.batch_add(L, static_cast<int>(L.steps) - 1, v);
        C.exit(L, static_cast<int>(L.steps), v);
    }
    C.batch_add(L, 2, static_cast<unsigned long long>(L.events));
    if (L.anomalies) C.batch_add(L, 3, static_cast<unsigned long long>(L.anomalies));
    if (L.run_abs) C.batch_add(L, 4 + L.layer, L.run_abs);
}

// The first part of a step: the free path (or what is left of it), the
// distance to the layer's boundary, and the hop. Returns true when the hop ends on the boundary.
// The distance to the boundary the packet heads for, by a select instead of a branch (measured 1.2 %
// faster on skin5): with uz = 0 the quotient is infinite or NaN and the test for a hit discards it.
template <int FAST> __device__ __forceinline__ float boundary_distance(const Hot &h, float z, float uz) {
    return m_div<FAST>(fsub(uz > 0.0f ? h.z1 : h.z0, z), uz);
}

template <int FAST, class Ctx> __device__ __forceinline__ bool step_move(Lane &L, Ctx &C, const Hot &h) {
    ++L.steps;
    float s;
    {
        // both candidates, then a select: a fresh free path (which consumes the next word) or the
        // rest of the one a boundary cut short (which consumes none). The word is read either way
        // (the ring always holds it) and passed over only when used. Half of a warp's steps hold a
        // lane that has just left a boundary, so a branch here diverged; the select measured 5.4 %
        // faster on skin5.
        const bool fresh = L.sleft == 0.0f;
        const float s_fresh = C.path(L, h), s_rest = scale_path<FAST>(h, L.sleft);
        s = fresh ? s_fresh : s_rest;
        C.pass(L, fresh ? 1u : 0u);
        L.sleft = 0.0f;
    }
    const float db = boundary_distance<FAST>(h, L.z, L.uz);
    const bool hit = L.uz != 0.0f && s > db;
    L.sleft = hit ? fmul(fsub(s, db), h.mut) : 0.0f;
    s = hit ? db : s;
    L.xy = ffma2(f2(s), L.uxy, L.xy);
    L.z = ffma(s, L.uz, L.z);
    return hit;
}

// At the boundary: reflect, or transmit into the next layer or out (physics.hpp:198-246). Sets
// exit_kind (1: reflectance, top; 2: transmittance, bottom) and died when the packet leaves.
template <int FAST, class Ctx>
__device__ __forceinline__ void step_boundary(Lane &L, Ctx &C, int &exit_kind, bool &died) {
    const LayerC &Lc = C.layer(L, L.layer);
    const bool up = L.uz < 0.0f;
    const float ca1 = up ? -L.uz : L.uz;
    const float4 side = boundary_side(Lc, up);  // n_t, n / n_t, critical cosine, normal-incidence R
    const float nt = side.x, rat = side.y;
    float uz1 = 0.0f;
    bool through;
    if (nt == Lc.n) {
        // matched indices: R = 0, so the Fresnel word (in (0, 1), always above R) is drawn and not
        // needed, and the direction goes through unchanged (rat = 1, cos_t = cos_i); measured 2.8 %
        // faster on skin5, whose inner boundaries are all matched
        C.skip(L);
        through = true;
        uz1 = ca1;
    } else {
        const float r = (ca1 <= side.z) ? 1.0f : fresnel<FAST>(Lc.n, nt, ca1, side.w, rat, uz1);
        through = C.unit(L) > r;
    }
    if (through) {
        L.uxy = fmul2(L.uxy, f2(rat));
        L.uz = up ? -uz1 : uz1;
        if (up ? L.layer == 0 : L.layer == C.num_layers(L) - 1) {
            exit_kind = up ? 1 : 2;
            died = true;
        } else {
            C.leave_layer(L);
            C.batch_add(L, 4 + L.layer, L.run_abs);  // adds 0 when nothing was absorbed: no branch
            L.run_abs = 0ull;
            L.layer += up ? -1 : 1;
            load_hot(L.h, C.layer(L, L.layer));
            C.enter_layer(L);
        }
    } else {
        L.uz = -L.uz;
    }
}

// The weight an interaction of a packet of weight w leaves (physics.hpp:187-193).
template <int FAST> __device__ __forceinline__ float drop_of(const Hot &h, float w) {
    if constexpr (Math<FAST>::div) return fmul(w, h.absorb);
    else return fmul(w, h.mua) / h.mut;
}

// An interaction: drop (physics.hpp:187-193), score the absorption, spin (physics.hpp:101-144).
template <int FAST, class Ctx> __device__ __forceinline__ void step_interaction(Lane &L, Ctx &C, const Hot &h) {
    const float dwa = drop_of<FAST>(h, L.w);
    L.w = fsub(L.w, dwa);
    ++L.events;
    C.scatter(L, h, dwa);
}

// Whether an interaction's packet breaks an invariant: a weight that is no number, a direction off unit
// length. A NaN weight turns the norm's deviation into NaN (0 * NaN), which fails the comparison.
__device__ __forceinline__ bool broken(float2 uxy, float uz, float dwa) {
    return !(fabsf(ffma(dwa, 0.0f, fsub(norm2(uxy, uz), 1.0f))) <= 1e-5f);
}

// Ctx::scatter of a lane that steps beside others: score and turn at once.
template <int FAST, class Ctx> __device__ __forceinline__ void scatter_now(Lane &L, const Ctx &C, const Hot &h, float dwa) {
    if (broken(L.uxy, L.uz, dwa)) ++L.anomalies;
    const unsigned long long v = to_fixed(dwa);
    L.run_abs += v;
    C.absorb(L.xy, L.z, v);
    const float ct = hg_cos<FAST>(h, C.unit(L));
    rotate<FAST>(L.uxy, L.uz, ct, C.unit(L));
}

// The end of a step: score an exit, or play roulette (physics.hpp:250-259); the step cap; publish
// an ended packet (unless the kernel does: Ctx::kPublishAtRelaunch). Returns true when the packet
// has ended.
template <int FAST, class Ctx> __device__ __forceinline__ bool step_tail(Lane &L, Ctx &C, int exit_kind, bool died) {
    // one test on the common path for the three rare ends of a step: an exit, a weight below the
    // roulette threshold, the step cap (measured 0.4 % faster on skin5 than three tests)
    if (exit_kind != 0 || L.w < kWeightMin || L.steps >= C.step_cap) {
        if (exit_kind) {
            // scored when the packet is published (finish_photon)
        } else if (L.w < kWeightMin) {
            // ---- roulette (physics.hpp:250-259)
            if (L.w == 0.0f) {
                died = true;
            } else if (C.unit(L) < kChance) {
                if constexpr (Math<FAST>::div) L.w = fmul(L.w, 10.0f);
                else L.w /= kChance;
            } else {
                died = true;
            }
        }
        if (!died && L.steps >= C.step_cap) {  // a packet that never ends is an anomaly, not a hang
            ++L.anomalies;
            died = true;
        }
        if (died) L.steps = static_cast<uint32_t>(exit_kind);  // how the packet ended (finish_photon)
    }
    if constexpr (!Ctx::kPublishAtRelaunch) {
        if (died) finish_photon(L, C);
    }
    return died;
}

// One hop-drop-spin (or boundary) step plus roulette (step_once, physics.hpp:263-277); returns true
// when the packet has ended. Its per-photon totals are then published here, or, when the context
// says Ctx::kPublishAtRelaunch, by the kernel when the lane takes its next photon or runs out (one
// warp-uniform place instead of a branch in every step).
template <int FAST, class Ctx> __device__ __forceinline__ bool walk_step(Lane &L, Ctx &C) {
    bool died = false;
    int exit_kind = 0;
    const Hot h = L.h;
    if (step_move<FAST>(L, C, h)) step_boundary<FAST>(L, C, exit_kind, died);
    else step_interaction<FAST>(L, C, h);
    return step_tail<FAST>(L, C, exit_kind, died);
}

// Whole warp, before a pass: top up the random words of the lanes that hold a live packet, by two
// blocks at once (independent chains of rounds) when all of them have the room. Against a vote and a
// block in every step: 1e3 photons of skin5 (latency) 1,796 -> 1,758 us, slab 1e7 2.89 -> 2.84 ms, three
// layers in exact math, 3e5 photons, 1,220 -> 1,166 us.
template <int FAST, class Ctx> __device__ __forceinline__ void top_up(Lane &L, Ctx &C, bool alive) {
    constexpr uint32_t kPassWords = 4u * steps_per_pass<FAST>();
    static_assert(kPassWords + 4u <= kRingWords, "a short lane must have room for a block");
    if (__all_sync(0xffffffffu, !alive || L.wp - L.rp <= kRingWords - 8u)) {
        if (alive) {
            C.refill2(L);
        }
    }
    while (__any_sync(0xffffffffu, alive && L.wp - L.rp < kPassWords)) {
        if (alive && L.wp - L.rp <= kRingWords - 4u) C.refill(L);
    }
}

// This lane's slot 0 in its block's ring area: each warp has its own region of kRingWords slots,
// slot k of its 32 lanes contiguous, so the lanes of a warp never conflict on a bank.
__device__ __forceinline__ int ring_lane_offset() {
    return static_cast<int>((threadIdx.x >> 5) * (kRingWords * 32u) + (threadIdx.x & 31u));
}

// The random-word ring: kRingWords words per lane in shared memory.
struct Ring {
    uint32_t *base;  // this lane's slot 0 (ring_lane_offset)

    __device__ __forceinline__ uint32_t draw(Lane &L) const {
        const uint32_t o = base[(L.rp & (kRingWords - 1u)) * slot_stride()];
        ++L.rp;
        return o;
    }
    // pass over the next word without reading it
    __device__ __forceinline__ void skip(Lane &L) const { ++L.rp; }
    // read the next word without passing over it
    __device__ __forceinline__ uint32_t peek(const Lane &L) const { return base[(L.rp & (kRingWords - 1u)) * slot_stride()]; }
    // each warp's ring is its own region: slot k of its 32 lanes at k * 32 words (a constant stride:
    // the slot addresses take shifts instead of multiplications)
    __device__ __forceinline__ static constexpr int slot_stride() { return 32; }
    __device__ __forceinline__ void store(Lane &L, uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3) const {
        ++L.blk;
        uint32_t *const slot = base + (L.wp & (kRingWords - 4u)) * slot_stride();  // wp is a multiple of 4
        slot[0] = b0;
        slot[slot_stride()] = b1;
        slot[2 * slot_stride()] = b2;
        slot[3 * slot_stride()] = b3;
        L.wp += 4u;
    }
    // two blocks at once: two independent chains of rounds
    __device__ __forceinline__ void refill2(Lane &L, const uint32_t (&rk)[20]) const {
        uint32_t a0, a1, a2, a3, b0, b1, b2, b3;
        philox4x32_10_rk(L.id, 0u, L.blk, rk, a0, a1, a2, a3);
        philox4x32_10_rk(L.id, 0u, L.blk + 1u, rk, b0, b1, b2, b3);
        store(L, a0, a1, a2, a3);
        store(L, b0, b1, b2, b3);
    }
    template <class Key> __device__ __forceinline__ void refill2(Lane &L, Key key) const {
        uint32_t a0, a1, a2, a3, b0, b1, b2, b3;
        philox4x32_10_sched(L.id, 0u, L.blk, key, a0, a1, a2, a3);
        philox4x32_10_sched(L.id, 0u, L.blk + 1u, key, b0, b1, b2, b3);
        store(L, a0, a1, a2, a3);
        store(L, b0, b1, b2, b3);
    }
    // with a precomputed key schedule (one key for every lane of the launch)
    __device__ __forceinline__ void refill(Lane &L, const uint32_t (&rk)[20]) const {
        uint32_t b0, b1, b2, b3;
        philox4x32_10_rk(L.id, 0u, L.blk, rk, b0, b1, b2, b3);
        store(L, b0, b1, b2, b3);
    }
    // with this lane's key schedule in memory (philox4x32_10_sched)
    template <class Key> __device__ __forceinline__ void refill(Lane &L, Key key) const {
        uint32_t b0, b1, b2, b3;
        philox4x32_10_sched(L.id, 0u, L.blk, key, b0, b1, b2, b3);
        store(L, b0, b1, b2, b3);
    }
};

// ------------------------------------------------------------------------------ one photon per warp
// At the end of a run a few long photons are left, one lane of a warp here and there, and the run lasts
// as long as the longest of them: about 1,000 cycles a step, since the 230 instructions of a step follow
// one another in one lane while 31 wait. A block down to two packets per warp therefore shares them out
// and every warp walks a packet at a time with all its lanes: every lane carries the packet's state (the
// same instructions, no divergence), and what does not depend on the path is done for many steps at once
// by different lanes. For the next kAloneWords random words the warp generates the blocks and evaluates
// every form a word can be used in: the plain uniform value and, for a step that would start at the word,
// the free path, the polar angle and the azimuth of its three words in the current layer (again when the
// layer changes). Scores are kept as records and scored twelve at a time, one per lane. The step that is left
// reads its numbers from shared memory: the boundary distance, the hop, the weight, the turn.
// Every number is computed by the same operations from the same operands as in a lane of its own.
// One photon of skin5 (1,012 steps): 557 us in a lane, 172 us so; the runs' ends: walk_ends_alone in
// engine.cu; 97 configurations of 1e3 photons 11.5 -> 3.3 ms, 4096 of 1e4 to 1e6 1.31 -> 1.22 s.
constexpr int kAloneWords = 56, kAloneRecords = 12, kAlonePerWarp = 2, kBurst = 3;
// Packets per warp at which a block turns to walking them alone. In exact math, whose accurate functions
// make up most of a step either way, one packet after another gains less.
template <int FAST> __device__ __forceinline__ constexpr int alone_per_warp() { return FAST ? kAlonePerWarp : 1; }
// A packet set aside (its buffered words stay behind: `at` is the number of words it has consumed; `tag`
// is the context's).
struct Parked {
    unsigned long long run_abs;
    float x, y, z, ux, uy, uz, w, sleft;
    int layer, batch;
    uint32_t id, at, events, anomalies, steps, tag;
};
// The warp's region of the ring.
struct AloneTables {
    float u[kAloneWords];       // the words as uniform values
    float4 turn[kAloneWords];   // of a step that starts at the word: ct, st, cp, sp
    float2 path[kAloneWords];   // and its free path, -st cp
    float2 xy[kAloneRecords], uxy[kAloneRecords];  // scores: position, direction before the turn,
    float z[kAloneRecords], uz[kAloneRecords], dwa[kAloneRecords];  // weight dropped
    Parked parked[kAlonePerWarp];
};
static_assert(kAloneWords % 4 == 0 && kAloneWords > 32 && kAloneWords <= 64 && kAloneRecords <= 32, "one or two words a lane");
static_assert(sizeof(AloneTables) <= kRingWords * 32 * 4, "the tables fit the warp's ring");

template <int FAST, class Base> struct AloneCtx {
    Base &B;
    AloneTables &T;
    uint32_t step_cap;
    unsigned lane;
    uint32_t blk = 0u;  // first block in the tables
    int p = 0;          // next word in the tables
    int records = 0;
    static constexpr bool kPublishAtRelaunch = true;

    __device__ __forceinline__ AloneCtx(Base &b, AloneTables &t, unsigned ln) : B(b), T(t), step_cap(b.step_cap), lane(ln) {}
    __device__ __forceinline__ float path(const Lane &, const Hot &) const { return T.path[p].x; }
    __device__ __forceinline__ float unit(Lane &) { return T.u[p++]; }
    __device__ __forceinline__ void skip(Lane &) { ++p; }
    __device__ __forceinline__ void pass(Lane &, uint32_t n) { p += static_cast<int>(n); }
    __device__ __forceinline__ const LayerC &layer(const Lane &L, int l) const { return B.layer(L, l); }
    __device__ __forceinline__ int num_layers(const Lane &L) const { return B.num_layers(L); }
    __device__ __forceinline__ void batch_add(const Lane &L, int slot, unsigned long long v) const {
        if (lane == 0) B.batch_add(L, slot, v);
    }
    __device__ __forceinline__ void exit(const Lane &L, int kind, unsigned long long v) const {
        if (lane == 0) B.exit(L, kind, v);
    }

    // what a step from each word on would use, in the packet's layer (a step's words end inside the table
    // for every start that is used)
    __device__ __forceinline__ void steps_of(const Lane &L) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int i = static_cast<int>(lane) + 32 * k;
            if (i >= kAloneWords) break;
            const float ct = hg_cos<FAST>(L.h, T.u[min(i + 1, kAloneWords - 1)]), st = sin_of<FAST>(ct);
            float sp, cp;
            azimuth<FAST>(T.u[min(i + 2, kAloneWords - 1)], sp, cp);
            T.turn[i] = make_float4(ct, st, cp, sp);
            T.path[i] = f2(step_length<FAST>(L.h, T.u[i]), fmul(-st, cp));
        }
        __syncwarp();
    }
    // fill the tables from block b on; the next word is word `first` of it
    __device__ __forceinline__ void fill(Lane &L, uint32_t b, int first) {
        blk = b;
        p = first;
        __syncwarp();  // the tables' last readers are done
        if (lane < kAloneWords / 4) {
            uint32_t w0, w1, w2, w3;
            B.block(L.id, b + lane, w0, w1, w2, w3);
            reinterpret_cast<float4 *>(T.u)[lane] = make_float4(unit_open(w0), unit_open(w1), unit_open(w2), unit_open(w3));
        }
        __syncwarp();
        steps_of(L);
    }
    // score the records, one per lane
    __device__ __forceinline__ void score(Lane &L) {
        if (records == 0) return;
        __syncwarp();
        bool bad = false;
        unsigned long long v = 0ull;
        if (static_cast<int>(lane) < records) {
            const float dwa = T.dwa[lane];
            bad = broken(T.uxy[lane], T.uz[lane], dwa);
            v = to_fixed(dwa);
            B.absorb(T.xy[lane], T.z[lane], v);
        }
        L.anomalies += static_cast<uint32_t>(__popc(__ballot_sync(0xffffffffu, bad)));
        // the sum of the values, 24 bits at a time and what is left of 64 (a weight that is no number is 2^63)
        const uint32_t lo = __reduce_add_sync(0xffffffffu, static_cast<uint32_t>(v) & 0xFFFFFFu);
        const uint32_t mid = __reduce_add_sync(0xffffffffu, static_cast<uint32_t>(v >> 24) & 0xFFFFFFu);
        const uint32_t hi = __reduce_add_sync(0xffffffffu, static_cast<uint32_t>(v >> 48));
        L.run_abs += (static_cast<unsigned long long>(hi) << 48) + (static_cast<unsigned long long>(mid) << 24) + lo;
        records = 0;
        __syncwarp();
    }
    __device__ __forceinline__ void record(int at, float2 xy, float z, float2 uxy, float uz, float dwa) {
        // every lane holds the same values: one store of a warp to one word, and no branch
        T.xy[at] = xy;
        T.z[at] = z;
        T.uxy[at] = uxy;
        T.uz[at] = uz;
        T.dwa[at] = dwa;
    }
    __device__ __forceinline__ void scatter(Lane &L, const Hot &h, float dwa) {
        record(records, L.xy, L.z, L.uxy, L.uz, dwa);
        if (++records == kAloneRecords) score(L);
        const float ct = hg_cos<FAST>(h, unit(L));
        rotate<FAST>(L.uxy, L.uz, ct, unit(L));
    }
    // N plain interactions in a row: whole free paths inside the layer, directions off the axis, weights
    // above roulette, so that all of it is straight-line arithmetic. Returns false, with the packet as it
    // was, when one of them is not plain; the records written are then not counted.
    template <int N> __device__ __forceinline__ bool plain(Lane &L) {
        const Hot &h = L.h;
        float2 xy = L.xy, uxy = L.uxy, path[N];
        float4 t[N];
        float z = L.z, uz = L.uz, w = L.w;
        bool ok = true;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            path[k] = T.path[p + 3 * k];
            t[k] = T.turn[p + 3 * k];
        }
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float s = path[k].x, db = boundary_distance<FAST>(h, z, uz);
            const float dwa = drop_of<FAST>(h, w);
            w = fsub(w, dwa);
            // (a level direction's quotient is -inf or NaN: left to walk_step)
            ok = ok && s <= db && fabsf(uz) <= kCosZero && w >= kWeightMin;
            xy = ffma2(f2(s), uxy, xy);
            z = ffma(s, uz, z);
            record(records + k, xy, z, uxy, uz, dwa);
            turn_oblique<FAST>(uxy, uz, t[k].x, t[k].y, t[k].z, t[k].w, path[k].y);
        }
        if (!ok) return false;
        L.xy = xy;
        L.z = z;
        L.uxy = uxy;
        L.uz = uz;
        L.w = w;
        p += 3 * N;
        records += N;
        return true;
    }
    // Plain interactions, as many as the tables and records hold, kBurst at a time: one branch for that
    // many steps, and a step's boundary test is off the chain of the next step's direction. Returns false
    // when the next step is not plain.
    __device__ __forceinline__ bool burst(Lane &L) {
        if (step_cap - L.steps <= kAloneRecords || L.sleft != 0.0f) return false;  // a packet at its cap ends in walk_step
        const int n0 = min(kAloneRecords - records, (kAloneWords - p) / 3);
        int n = n0;
        while (n >= kBurst && plain<kBurst>(L)) n -= kBurst;
        bool more = true;
        while (n > 0 && (more = plain<1>(L))) --n;
        L.events += static_cast<uint32_t>(n0 - n);
        L.steps += static_cast<uint32_t>(n0 - n);
        return more;
    }
    __device__ __forceinline__ void leave_layer(Lane &L) { score(L); }
    __device__ __forceinline__ void enter_layer(Lane &L) {
        __syncwarp();  // every lane has read its free path (score() has no barrier when it has no records)
        steps_of(L);
    }
};

// How many live lanes each warp of a block has, and the next parked packet to take (shared memory).
struct AloneState {
    unsigned char live[8];
    uint32_t next, pad;
};
static_assert(sizeof(AloneState) == 16, "AloneState layout");
__device__ __forceinline__ int live_lanes(const volatile AloneState &S) {
    const volatile uint32_t *w = reinterpret_cast<const volatile uint32_t *>(&S);
    return static_cast<int>(__dp4a(w[0], 0x01010101u, __dp4a(w[1], 0x01010101u, 0u)));
}
// The tables of warp w in the block's ring area.
__device__ __forceinline__ AloneTables &alone_tables(void *ring, unsigned w) {
    return *reinterpret_cast<AloneTables *>(static_cast<uint32_t *>(ring) + w * (kRingWords * 32u));
}
// Whole block: set the packets of every warp's lanes in `live` aside, at most kAlonePerWarp per warp of the
// block; returns their number. The lanes' random words are overwritten. C.tag() of a lane and C.adopt(tag)
// carry its context over.
template <class Ctx> __device__ __forceinline__ int park(const Lane &L, const Ctx &C, unsigned live, unsigned lane, void *ring, volatile AloneState &S) {
    __syncthreads();  // every warp has left its step loop, with its count in S
    const unsigned warp = threadIdx.x >> 5;
    unsigned slot = __popc(live & ((1u << lane) - 1u));
    for (unsigned w = 0; w < warp; ++w) slot += S.live[w];
    if ((live >> lane) & 1u) {
        Parked &k = alone_tables(ring, slot / kAlonePerWarp).parked[slot % kAlonePerWarp];
        k.run_abs = L.run_abs;
        k.x = L.xy.x;
        k.y = L.xy.y;
        k.z = L.z;
        k.ux = L.uxy.x;
        k.uy = L.uxy.y;
        k.uz = L.uz;
        k.w = L.w;
        k.sleft = L.sleft;
        k.layer = L.layer;
        k.batch = L.batch;
        k.id = L.id;
        k.at = 4u * L.blk - (L.wp - L.rp);
        k.events = L.events;
        k.anomalies = L.anomalies;
        k.steps = L.steps;
        k.tag = C.tag();
    }
    const int total = live_lanes(S);
    __syncthreads();
    return total;
}
// The next parked packet of the block for this warp (a number at or past the total: none is left).
__device__ __forceinline__ int next_parked(AloneState &S, unsigned lane) {
    uint32_t r = 0u;
    if (lane == 0) r = atomicAdd(&S.next, 1u);
    return static_cast<int>(__shfl_sync(0xffffffffu, r, 0));
}
// A parked packet as every lane's.
__device__ __forceinline__ Lane unpark(const Parked &k) {
    Lane M;
    M.run_abs = k.run_abs;
    M.xy = f2(k.x, k.y);
    M.z = k.z;
    M.uxy = f2(k.ux, k.uy);
    M.uz = k.uz;
    M.w = k.w;
    M.sleft = k.sleft;
    M.layer = k.layer;
    M.batch = k.batch;
    M.id = k.id;
    M.blk = k.at >> 2;
    M.rp = k.at & 3u;
    M.events = k.events;
    M.anomalies = k.anomalies;
    M.steps = k.steps;
    return M;
}
// Whole warp: walk the packet M (the same in every lane, its next random word M.rp of block M.blk) to its
// end and publish it.
template <int FAST, class Ctx> __device__ __forceinline__ void walk_alone(Lane &M, Ctx &B, unsigned lane, AloneTables &T) {
    AloneCtx<FAST, Ctx> A(B, T, lane);
    load_hot(M.h, B.layer(M, M.layer));
    A.fill(M, M.blk, static_cast<int>(M.rp));
#pragma unroll 1
    for (;;) {
        const bool plain = A.burst(M);
        if (A.records == kAloneRecords) A.score(M);
        if (A.p > kAloneWords - 4) A.fill(M, A.blk + static_cast<uint32_t>(A.p >> 2), A.p & 3);  // a step draws at most 4
        if (!plain && walk_step<FAST>(M, A)) break;
    }
    A.score(M);
    finish_photon(M, A);
    __syncwarp();
}

}  // namespace tmc
