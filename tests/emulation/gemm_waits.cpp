// The tensor-core GEMM's roles (gemm_tc.cuh) on the CPU with waits that run out (kernel_emulator.hpp,
// umma_stub.hpp): the lanes of a warp poll a barrier at their own times, so some may see it complete on their
// last poll and others give up. The block must end either way, and either every warp writes its part of the
// tile and the status stays 0, or none does and the status says so. Built and run by
// tests/test_kernel_emulation.py.

#include "kernel_emulator.hpp"

struct CUtensorMap {};

#include "gemm_tc.cuh"  // a copy beside umma_stub.hpp under umma.cuh's name

namespace tmc {
alignas(16) unsigned char gsm_raw[GemmSmem<64>::bytes + 16];
}

namespace {

int g_pieces = 0;
struct Epi {
    const float *bias = nullptr;
    struct Regs {};
    void prefetch(int, int, Regs &) const {}
    void piece(int, int, int, const float (&)[32], const float *, unsigned char *, Regs &) const { ++g_pieces; }
};

}  // namespace

int main() {
    int failures = 0, given_up = 0, finished = 0;
    for (uint32_t limit : {2u, 5u, 10u, 20u, 40u, 100u, 100000u})
        for (uint64_t seed = 1; seed <= 40; ++seed)
            for (int withhold : {0, 1}) {
                if (withhold && limit > 100u) continue;
                int status = 0;
                g_pieces = 0;
                gridDim = {1, 1, 1};
                blockDim.x = tmc::kGemmThreads;
                const CUtensorMap a, b;
                const char *e = emu::run(1, tmc::kGemmThreads, sizeof(tmc::gsm_raw) / 8, reinterpret_cast<uint64_t *>(tmc::gsm_raw),
                                         emu::Order::Skewed, seed, {}, [&] {
                                             tmc::gemm_tc_kernel<64, Epi>(a, b, 128, 64, 7 * 64, Epi{}, &status, limit, withhold);
                                         }, threadIdx, blockIdx);
                // 128 x 64 outputs: eight warps with one piece of 32 x 32 each
                const bool wrote = g_pieces == tmc::kGemmThreads;
                if (!e && !(wrote && status == 0) && !(g_pieces == 0 && status != 0)) e = "part of the tile written, or a give-up not reported";
                if (!e && limit > 100u && !wrote) e = "gave up without need";
                if (e && ++failures <= 5)
                    std::fprintf(stderr, "FAILED: %s (limit %u, seed %llu, withhold %d: %d pieces, status %d)\n", e, limit,
                                 static_cast<unsigned long long>(seed), withhold, g_pieces, status);
                ++(wrote ? finished : given_up);
            }
    if (failures || !given_up || !finished) {
        std::fprintf(stderr, "%d failures (%d launches gave up, %d finished)\n", failures, given_up, finished);
        return 1;
    }
    std::printf("%d launches gave up, %d finished\n", given_up, finished);
    return 0;
}
