// What gemm_tc.cuh takes from umma.cuh, for the CPU: barriers whose phases end some polls after the copy or
// product that ends them was issued, and no arithmetic. A test's build puts this file in umma.cuh's place.
#pragma once

namespace tmc {

// an mbarrier: phases ended, and phases whose end is on its way (upper half)
inline void mbar_init(uint64_t *bar, uint32_t) { *bar = 0; }
inline void under_way(uint64_t *bar) { *bar += 1ull << 32; }
inline bool mbar_wait(uint64_t *bar, uint32_t parity, uint32_t limit) {
    for (uint32_t i = 0; i < limit; ++i) {
        emu::pause();
        if (*bar >> 32 && emu::g->rng() % 64 == 0) *bar += 1ull - (1ull << 32);
        if ((*bar & 1u) != parity) return true;
    }
    return false;
}
inline void mbar_arrive_expect_tx(uint64_t *bar, uint32_t) { under_way(bar); }
inline void umma_commit(uint64_t *bar) { under_way(bar); }
inline void tma_load_2d(void *, const void *, int, int, uint64_t *) {}
#define elect_one() (emu::collective(__LINE__, 0) != nullptr && threadIdx.x % 32 == 0)

// collectives of a warp that do nothing else here
inline void tmem_alloc(uint32_t *slot, uint32_t) { emu::collective(-1, 0), *slot = 0; }
inline void tmem_dealloc(uint32_t, uint32_t) { emu::collective(-2, 0); }
inline void tmem_ld32(uint32_t, float (&v)[32]) { emu::collective(-3, 0), std::fill(v, v + 32, 0.0f); }

inline void wait_for_inputs() {}
inline void dependents_may_start() {}
inline void tc_fence_before() {}
inline void tc_fence_after() {}
inline uint32_t smem_u32(const void *) { return 0; }
inline uint64_t umma_desc_sw128(uint32_t) { return 0; }
constexpr uint32_t umma_idesc_bf16(int, int) { return 0; }
inline void umma_bf16_k64(uint32_t, uint64_t, uint64_t, uint32_t, uint32_t) {}
inline uint32_t cluster_rank() { return 0; }
inline void cluster_barrier() {}
inline float4 ld_cluster_f32x4(const float4 *p, uint32_t) { return *p; }

}  // namespace tmc
