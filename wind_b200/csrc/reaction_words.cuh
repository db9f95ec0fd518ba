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

}  // namespace wind
