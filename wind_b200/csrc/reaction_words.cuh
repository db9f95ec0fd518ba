// reaction_words.cuh -- reactions of a mass-action system as 32-bit words, for the
// kernels that keep their lists in shared memory (N <= 32).
#pragma once

#include "common.cuh"

namespace wind {

// An incidence of a species, or a term of a Jacobian entry, in one word: the
// signed rate's byte offset (19 bits), two species (6 bits each: reactants a and
// b of an incidence, the other reactant and the column of a term), and whether
// the term is its entry's last.
constexpr uint32_t RX_MARK = 1u << 31;
__device__ __forceinline__ uint32_t rx_pack(int slot, int first, int second) {
    return (uint32_t)(slot * 8) | ((uint32_t)first << 19) | ((uint32_t)second << 25);
}
__device__ __forceinline__ double rx_at(const double* base, uint32_t bytes) {
    return *reinterpret_cast<const double*>(reinterpret_cast<const char*>(base) + bytes);
}
__device__ __forceinline__ double rx_rate(const double* rates, uint32_t q) { return rx_at(rates, q & 0x7ffffu); }
__device__ __forceinline__ uint32_t rx_first(uint32_t q) { return (q >> 16) & 0x1f8u; }   // byte offsets
__device__ __forceinline__ uint32_t rx_second(uint32_t q) { return (q >> 22) & 0x1f8u; }

// Inclusive sum of v over the L lanes of a team.
template <int L>
__device__ __forceinline__ int rx_scan(unsigned mask, int l, int v) {
#pragma unroll
    for (int s = 1; s < L; s <<= 1) {
        const int u = __shfl_up_sync(mask, v, s, L);
        if (l >= s) v += u;
    }
    return v;
}

// The ids of the reactions that touch species l (l < N), ascending, to out[0..],
// one list per lane of a team of L lanes; returns how many.  `touched`: N words of
// shared memory.
// The lanes take 32 reactions at a time and mark them in their species' words;
// every lane then lists its own marks.  (With every lane looking through all the
// reactions, a reaction cost some 200 cycles and pass.)
template <int L>
__device__ __forceinline__ int rx_list(unsigned mask, int l, int N, int R, const uint2* sp, uint32_t* touched,
                                       uint32_t* out) {
    int cnt = 0;
    constexpr int PER = 32 / L;
    uint2 next[PER];
#pragma unroll
    for (int u = 0; u < PER; u++)
        if (l + u * L < R) next[u] = __ldg(sp + l + u * L);
    if (l < N) touched[l] = 0u;
    __syncwarp(mask);
    for (int r0 = 0; r0 < R; r0 += 32) {
        uint2 q[PER];
#pragma unroll
        for (int u = 0; u < PER; u++) {
            q[u] = next[u];
            if (r0 + 32 + l + u * L < R) next[u] = __ldg(sp + r0 + 32 + l + u * L);
        }
#pragma unroll
        for (int u = 0; u < PER; u++) {
            if (r0 + l + u * L < R) {
                const uint32_t bit = 1u << (l + u * L);
                atomicOr(touched + (q[u].x & 0xffffu), bit);
                atomicOr(touched + (q[u].x >> 16), bit);
                atomicOr(touched + (q[u].y & 0xffffu), bit);
                atomicOr(touched + (q[u].y >> 16), bit);
            }
        }
        __syncwarp(mask);
        if (l < N) {
            for (uint32_t m = touched[l]; m; m &= m - 1u) out[cnt++] = (uint32_t)(r0 + __ffs(m) - 1);
            touched[l] = 0u;
        }
        __syncwarp(mask);
    }
    return cnt;
}

}  // namespace wind
