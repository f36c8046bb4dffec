// Runs of few photons through the walk kernel's and the sweep's own source on the CPU (kernel_emulator.hpp):
// blocks that start late, lanes of a warp that drift apart between two collectives. Every run's tallies must
// be those of one full warp walking the same photons one pass after the other, word for word. Built and run
// by tests/test_kernel_emulation.py; exits non-zero with a message on the first difference.
//
// Compiled with TMC_FAST_MASK = 0: fast math's loop (steps per pass, packets walked alone) on the accurate
// functions.

#include "kernel_emulator.hpp"

#include <array>
#include <string>

#include "../../tissuemc_b200/csrc/sweep_kernel.cuh"
#include "../../tissuemc_b200/csrc/walk_kernel.cuh"

namespace tmc {
alignas(16) unsigned long long smem[1 << 15];
}

namespace {

using tmc::LayerC;

struct Tissue {
    const char *name;
    std::vector<std::array<float, 5>> layers;  // n, mua, mus, g, d
};
// short photons; thin layers with and without matched indices (boundary after boundary); long photons
const Tissue kTissues[] = {
    {"slab", {{1.4f, 20.0f, 30.0f, 0.5f, 0.02f}}},
    {"thin layers", {{1.4f, 5.0f, 60.0f, 0.8f, 0.004f}, {1.4f, 2.0f, 5.0f, 0.0f, 0.003f}, {1.5f, 9.0f, 40.0f, 0.7f, 0.002f},
                     {1.5f, 1.0f, 3.0f, -0.3f, 0.003f}, {1.3f, 4.0f, 90.0f, 0.9f, 0.01f}}},
    {"thick", {{1.37f, 12.0f, 90.0f, 0.7f, 1.0f}}},
    // mua = 1e-46 and d = 1e39 in float32 (both are accepted): every score is no number, until the step cap
    {"clear and endless", {{1.0f, 0.0f, 0.0f, 0.0f, INFINITY}}},
};
constexpr int kNz = 6, kNr = 5, kNa = 3;
constexpr uint32_t kNoCap = 2000000000u;

void fill(const Tissue &t, LayerC *out) {
    float z = 0.0f;
    const size_t n = t.layers.size();
    for (size_t i = 0; i < n; ++i) {
        const auto &y = t.layers[i];
        const float up = i ? t.layers[i - 1][0] : 1.0f, dn = i + 1 < n ? t.layers[i + 1][0] : 1.0f, g = y[3];
        LayerC L{};
        L.mua = y[1];
        L.mus = y[2];
        L.mut = L.mua + L.mus;
        L.inv_mut = 1.0f / L.mut;
        L.absorb = L.mua / L.mut;
        L.z0 = z;
        L.z1 = z += y[4];
        L.g = g;
        L.hg_a = 1.0f - g * g;
        L.hg_b = 1.0f - g;
        L.hg_c = 2.0f * g;
        L.hg_d = 1.0f + g * g;
        L.inv_2g = g != 0.0f ? 1.0f / (2.0f * g) : 0.0f;
        L.n = y[0];
        const auto side = [&](float nt, float &index, float &rat, float &cc, float &rn) {
            index = nt;
            rat = L.n / nt;
            cc = L.n > nt ? std::sqrt(1.0f - (nt * nt) / (L.n * L.n)) : 0.0f;
            rn = (nt - L.n) / (nt + L.n) * ((nt - L.n) / (nt + L.n));
        };
        side(up, L.n_up, L.rat_up, L.cc_up, L.rn_up);
        side(dn, L.n_dn, L.rat_dn, L.cc_dn, L.rn_dn);
        out[i] = L;
    }
}

int g_failures = 0;
void fail(const char *what, const Tissue &t, uint32_t photons, int blocks, int threads, int lanes, uint64_t seed) {
    if (++g_failures <= 5)
        std::fprintf(stderr, "FAILED: %s (%s, %u photons, %d blocks of %d threads, %d lanes a warp, seed %llu)\n", what, t.name,
                     photons, blocks, threads, lanes, static_cast<unsigned long long>(seed));
}
std::vector<uint64_t> late(int blocks, uint64_t seed) {
    std::mt19937_64 rng(seed);
    std::vector<uint64_t> s(static_cast<size_t>(blocks), 0);
    for (uint64_t &x : s)
        if (rng() % 10 < 7) x = rng() % 2000;
    return s;
}

// ------------------------------------------------------------------------------ the walk
template <int FAST, bool ALONE>
const char *walk(const Tissue &t, uint32_t photons, int blocks, int threads, uint32_t step_cap, emu::Order order, uint64_t seed,
                 const std::vector<uint64_t> &start, std::vector<unsigned long long> &tally, int *lanes_out) {
    const int nl = static_cast<int>(t.layers.size()), nb = photons < 7 ? 1 : 7;
    tmc::WalkParams P{};
    P.photons = photons;
    P.plan_base = photons / nb;
    P.plan_extra = photons % nb;
    P.plan_bnd = P.plan_extra * (P.plan_base + 1u);
    P.threads = static_cast<uint32_t>(threads);
    P.nb = nb;
    P.nl = nl;
    P.nz = kNz;
    P.nr = kNr;
    P.na = kNa;
    const size_t at_arz = static_cast<size_t>(nb) * (4 + nl), at_rd = at_arz + kNz * kNr, at_tt = at_rd + kNr * kNa;
    tally.assign(at_tt + kNr * kNa, 0ull);
    unsigned counter = 0u;
    P.counter = &counter;
    P.g_batch = tally.data();
    P.g_arz = tally.data() + at_arz;
    P.g_rd = tally.data() + at_rd;
    P.g_tt = tally.data() + at_tt;
    P.launch_w = 1.0f;
    P.dz = 0.004f;
    P.dr = 0.01f;
    P.da = 0.53f;
    P.tr_a = kNr - 2;
    P.tz_a = kNz - 2;
    P.cross = 1;
    P.batch_smem = 1;
    P.profiles = 1;
    P.step_cap = step_cap;
    // as a launch of few photons spreads them: evenly over all warps
    const int warps = blocks * threads / 32;
    P.lanes = static_cast<int>(std::min<uint32_t>(32u, (photons + warps - 1) / warps));
    P.chunk = 32;
    *lanes_out = P.lanes;
    for (uint32_t r = 0; r < 10; ++r) {
        P.round_keys[2 * r] = 11u + r * 0x9E3779B9u;
        P.round_keys[2 * r + 1] = r * 0xBB67AE85u;
    }
    fill(t, P.layers);
    blockDim.x = static_cast<unsigned>(threads);
    return emu::run(blocks, threads, static_cast<size_t>(tmc::smem_layout(P).total), reinterpret_cast<uint64_t *>(tmc::smem), order, seed,
                    start, [&] { tmc::walk_body<FAST, true, true, ALONE>(P); }, threadIdx, blockIdx);
}

template <int FAST> void walk_case(const Tissue &t, uint32_t photons, int blocks, int threads, uint32_t cap, emu::Order order, uint64_t seed) {
    std::vector<unsigned long long> want, got;
    int lanes = 0;
    const char *e = walk<FAST, false>(t, photons, 1, 32, cap, emu::Order::Lockstep, 1, {}, want, &lanes);
    if (e) return fail(e, t, photons, 1, 32, lanes, 1);
    e = walk<FAST, true>(t, photons, blocks, threads, cap, order, seed, late(blocks, seed), got, &lanes);
    if (e) return fail(e, t, photons, blocks, threads, lanes, seed);
    if (got != want) fail("the tallies differ", t, photons, blocks, threads, lanes, seed);
}

// ------------------------------------------------------------------------------ the sweep
template <int FAST>
const char *sweep(const std::vector<uint32_t> &photons, int blocks, int threads, uint32_t chunk, uint32_t lanes, emu::Order order,
                  uint64_t seed, const std::vector<uint64_t> &start, std::vector<unsigned long long> &tally) {
    const uint32_t n = static_cast<uint32_t>(photons.size());
    std::vector<tmc::SweepConfigC> cfgs(n);
    std::vector<uint32_t> prefix(n + 1, 0u);
    std::vector<LayerC> layers(16 * n);
    for (uint32_t c = 0; c < n; ++c) {
        const Tissue &t = kTissues[c % 3];
        tmc::SweepConfigC &k = cfgs[c];
        k = {};
        k.photons = photons[c];
        k.plan_base = photons[c];
        k.k0 = 100u + c;
        k.launch_w = 1.0f;
        k.nl = static_cast<int>(t.layers.size());
        k.layer_base = static_cast<int>(16 * c);
        k.chunk = chunk + c % 5;
        uint32_t k0 = k.k0, k1 = k.k1;
        for (uint4 &q : k.sched) {
            q = make_uint4(k0, k1, k0 + 0x9E3779B9u, k1 + 0xBB67AE85u);
            k0 += 2u * 0x9E3779B9u;
            k1 += 2u * 0xBB67AE85u;
        }
        fill(t, layers.data() + 16 * c);
        prefix[c + 1] = prefix[c] + (photons[c] + k.chunk - 1) / k.chunk;
    }
    tmc::SweepHeader h{};
    h.blocks = static_cast<uint32_t>(blocks);
    h.lanes = lanes;
    h.n_cfg = n;
    h.order = tmc::sweep_order(prefix[n], 3);
    tmc::SweepParams P{};
    P.hdr = &h;
    P.cfgs = cfgs.data();
    P.prefix = prefix.data();
    P.layers = layers.data();
    unsigned counter = 0u;
    P.item_counter = &counter;
    P.nb = 1;
    P.lmax = 5;
    P.nz = kNz;
    P.nr = kNr;
    P.na = kNa;
    P.stride = 9 + kNz * kNr + 2 * kNr * kNa;
    tally.assign(static_cast<size_t>(P.stride) * n, 0ull);
    P.tally = tally.data();
    P.dz = 0.004f;
    P.dr = 0.01f;
    P.da = 0.53f;
    P.profiles = 1;
    P.step_cap = kNoCap;
    P.threads = static_cast<uint32_t>(threads);
    P.tile_words = 17;
    blockDim.x = static_cast<unsigned>(threads);
    const size_t words = tmc::kRingWords / 2 * static_cast<size_t>(threads) + 18 + (sizeof(tmc::BlockSweepState) + 7) / 8;
    return emu::run(blocks, threads, words, reinterpret_cast<uint64_t *>(tmc::smem), order, seed, start,
                    [&] { tmc::sweep_block_kernel<FAST>(P); }, threadIdx, blockIdx);
}

template <int FAST> void sweep_case(const std::vector<uint32_t> &photons, int blocks, int threads, uint32_t chunk, uint32_t lanes,
                                    emu::Order order, uint64_t seed) {
    std::vector<unsigned long long> want, got;
    const char *e = sweep<FAST>(photons, 1, 32, 1000u, 32u, emu::Order::Lockstep, 1, {}, want);
    if (e) return fail(e, kTissues[0], photons[0], 1, 32, 32, 1);
    e = sweep<FAST>(photons, blocks, threads, chunk, lanes, order, seed, late(blocks, seed), got);
    if (e) return fail(e, kTissues[0], photons[0], blocks, threads, static_cast<int>(lanes), seed);
    if (got != want) fail("the sweep's tallies differ", kTissues[0], photons[0], blocks, threads, static_cast<int>(lanes), seed);
}

template <int FAST> void walks(std::initializer_list<int> tissues, emu::Order order, int repeats, uint32_t cap) {
    uint64_t seed = 1;
    for (int tissue : tissues)
        for (int threads : {32, 64, 128})
            for (int lanes : {1, 2, 3, 4, 8, 9, 32})
                for (int r = 0; r < repeats; ++r, ++seed) {
                    const int blocks = 5, warps = blocks * threads / 32;
                    const uint32_t photons = static_cast<uint32_t>(warps * lanes) - static_cast<uint32_t>(seed % static_cast<uint64_t>(warps));
                    walk_case<FAST>(kTissues[tissue], photons, blocks, threads, cap, order, seed);
                }
}

}  // namespace

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "late_blocks") {
        walks<1>({0, 2}, emu::Order::Lockstep, 4, kNoCap);
        walks<0>({0, 2}, emu::Order::Lockstep, 4, kNoCap);
        walks<1>({0, 2}, emu::Order::Lockstep, 1, 7u);
    } else if (what == "layer_changes") {
        walks<1>({1}, emu::Order::Lockstep, 2, kNoCap);
        walks<0>({1}, emu::Order::Lockstep, 2, kNoCap);
    } else if (what == "no_numbers") {
        walks<1>({3}, emu::Order::Lockstep, 2, 23u);
        walks<0>({3}, emu::Order::Lockstep, 2, 20u);
    } else if (what == "lanes_apart") {
        walks<1>({0, 1, 2}, emu::Order::Skewed, 1, kNoCap);
        walks<0>({0, 1, 2}, emu::Order::Skewed, 1, kNoCap);
    } else if (what == "sweep_lanes_apart") {
        uint64_t seed = 1;
        for (emu::Order order : {emu::Order::Lockstep, emu::Order::Skewed})
            for (int threads : {32, 64, 128})
                for (uint32_t lanes : {1u, 7u, 32u})
                    for (uint32_t chunk : {1u, 13u, 40u}) {
                        sweep_case<1>({40, 1, 23, 9}, 3, threads, chunk, lanes, order, ++seed);
                        sweep_case<0>({5, 60, 2}, 2, threads, chunk, lanes, order, ++seed);
                    }
    } else {
        std::fprintf(stderr, "no such case\n");
        return 2;
    }
    if (g_failures) {
        std::fprintf(stderr, "%d failures\n", g_failures);
        return 1;
    }
    std::printf("%s: all runs agree\n", what.c_str());
    return 0;
}
