// Decoupled look-back over tiles with 64-bit descriptors, for kernels that place their output behind that of the tiles before.
#pragma once

#include "common.cuh"

namespace b200bpe {

constexpr uint32_t SC_MAX_SPINS = 1u << 22;

// Tile descriptor of the look-back: bits 63..62 = flag (1 aggregate, 2 prefix), low 62 bits = value.
__device__ __forceinline__ unsigned long long ld_d64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_d64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Sum of the counts of the tiles before `tile`; called by one whole warp.  The tile's own count goes out first.
// A wait that runs out sets ctl[1] and gives 0.
__device__ __forceinline__ unsigned long long sc_look_back(unsigned long long* __restrict__ desc, uint64_t tile, unsigned long long agg, int lane,
                                                           uint32_t max_spins, uint32_t* __restrict__ ctl) {
    unsigned long long excl = 0ull;
    if (tile == 0) {
        if (lane == 0) st_d64(desc, (2ull << 62) | agg);
    } else {
        if (lane == 0) st_d64(desc + tile, (1ull << 62) | agg);
        long long pos = (long long)tile - 1;
        uint32_t spins = 0;
        bool timed_out = false;
        for (;;) {
            const long long idx = pos - lane;
            unsigned long long d = 2ull << 62;  // before tile 0: a zero prefix
            for (;;) {
                if (idx >= 0) d = ld_d64(desc + idx);
                if (__all_sync(0xFFFFFFFFu, (d >> 62) != 0ull)) break;
                if (++spins > max_spins) { timed_out = true; break; }
                __nanosleep(40);
            }
            if (timed_out) break;
            const uint32_t pmask = __ballot_sync(0xFFFFFFFFu, (d >> 62) == 2ull);
            const int first = pmask ? (__ffs(pmask) - 1) : 32;
            unsigned long long contrib = (lane <= first) ? (d & 0x3FFFFFFFFFFFFFFFull) : 0ull;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) contrib += __shfl_xor_sync(0xFFFFFFFFu, contrib, o);
            excl += contrib;
            if (pmask) break;
            pos -= 32;
        }
        if (timed_out) {
            if (lane == 0) atomicExch(&ctl[1], 1u);
            excl = 0ull;
        }
        if (lane == 0) st_d64(desc + tile, (2ull << 62) | (excl + agg));
    }
    return excl;
}

}  // namespace b200bpe
