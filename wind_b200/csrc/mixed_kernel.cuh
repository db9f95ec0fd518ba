// mixed_kernel.cuh -- one persistent launch for a batch of mass-action
// groups of different sizes.
//
// The groups are visited in the order given (largest N first, so the longest
// systems start earliest and the short ones fill the tail).  For each group
// every block works on that group's device work queue -- one system per block
// for N > 32 (cta_run), one system per team of 8/16/32 lanes for N <= 32
// (warp_run for SIE with the LU or mixed solve, team_run otherwise) -- until
// the queue is empty, then moves on to the next group.
// A block that finishes a group early starts the next one while others are
// still on their last systems, so the groups overlap on the device.
#pragma once

#include "cta_kernel.cuh"
#include "lu_kernel.cuh"
#include "team_kernel.cuh"
#include "warp_kernel.cuh"

namespace wind {

constexpr int MIXED_THREADS = CTA_THREADS;

// Teams of a block that run a group of the team or LU kernel: all that the
// lanes hold, or as many as the shared-memory budget does.
__host__ __device__ inline int mixed_teams(int nmax, int team_bytes, int smem_cap) {
    const int full = MIXED_THREADS / nmax, fit = smem_cap / team_bytes;
    return fit < full ? fit : full;
}

// Whether a group's systems are staged by counting, a reaction per lane, or with
// every lane looking through all reactions.  Counting wins by the reaction: one
// attempt of 4,000 systems takes 2.75 ms by looking and 0.68 by counting with 32
// species and 640 reactions, 0.83 and 0.28 with 16 and 320.  But the LU of up to 16
// species and RK2 run slower in the kernel that has the counting beside them (40
// attempts of 8 species and 200 reactions: 1.71 and 2.68 ms, of 16 and 160: 1.81 and
// 2.88; the RK2 batch of 1,000 mixed sizes 1.79 and 2.46), so where looking costs
// little a launch takes the kernel without it.
__host__ __device__ constexpr bool mixed_counted(int n, int react) {
    return n <= 32 && react > 12 * n && react > 300;
}

template <int NMAX, int METHOD, int CTRL, bool COUNTED>
__device__ __forceinline__ void mixed_team_run(const KParams& p, unsigned char* smem_raw, int smem_cap) {
    const TeamLayout lay(NMAX, p.n_react, p.linear != nullptr, METHOD == WIND_METHOD_SIE);
    team_run<NMAX, METHOD, CTRL, COUNTED>(p, smem_raw, mixed_teams(NMAX, lay.bytes, smem_cap), 32 / NMAX);
}

template <int NMAX, int CTRL, int SOLVER, bool COUNTED>
__device__ __forceinline__ void mixed_warp_run(const KParams& p, unsigned char* smem_raw, int smem_cap) {
    if constexpr (SOLVER == WIND_SOLVER_LU_F64) {
        const LuLayout lay(NMAX, p.n_eq, p.n_react, p.linear != nullptr, true);
        lu_run<NMAX, NMAX, true, CTRL, COUNTED>(p, smem_raw, mixed_teams(NMAX, lay.bytes, smem_cap), 32 / NMAX, true);
    } else {
        warp_run<NMAX, CTRL>(p, smem_raw);
    }
}

// Two blocks per SM (128 registers) for the LU and mixed solvers, whose team
// and CTA paths fit that budget; the reference Gauss-Jordan keeps a row of M
// and of the inverse per lane in registers and gets the whole file.
// SMALL is the solver of the groups with N <= 32 (SOLVER for the others);
// the AUTO solver runs MIXED above 32 species and LU_F64 below in one launch.
// COUNTED is how the team and LU kernels' systems are staged (mixed_counted).
template <int METHOD, int CTRL, int SOLVER, int SMALL, bool COUNTED>
__global__ void __launch_bounds__(MIXED_THREADS, SOLVER == WIND_SOLVER_GJE_F64 ? 1 : 2)
    k_mixed(const KParams* __restrict__ groups, const int* __restrict__ order, int ngroups,
            double* gscratch, size_t gstride, int smem_cap) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    for (int gi = 0; gi < ngroups; gi++) {
        const KParams p = groups[order[gi]];
        if (p.nsys > 0) {
            constexpr bool REG = METHOD == WIND_METHOD_SIE && SMALL != WIND_SOLVER_GJE_F64;
            if (p.n_eq > 32) cta_run<METHOD, CTRL, SOLVER, false>(p, smem_raw, gscratch, gstride, smem_cap);
            else if constexpr (REG) {
                if (p.n_eq > 16) mixed_warp_run<32, CTRL, SMALL, COUNTED>(p, smem_raw, smem_cap);
                else if (p.n_eq > 8) mixed_warp_run<16, CTRL, SMALL, COUNTED>(p, smem_raw, smem_cap);
                else mixed_warp_run<8, CTRL, SMALL, COUNTED>(p, smem_raw, smem_cap);
            } else {
                if (p.n_eq > 16) mixed_team_run<32, METHOD, CTRL, COUNTED>(p, smem_raw, smem_cap);
                else if (p.n_eq > 8) mixed_team_run<16, METHOD, CTRL, COUNTED>(p, smem_raw, smem_cap);
                else mixed_team_run<8, METHOD, CTRL, COUNTED>(p, smem_raw, smem_cap);
            }
        }
        __syncthreads();
    }
}

// The kernel of a launch; one source file per COUNTED.
using MixedFn = void (*)(const KParams*, const int*, int, double*, size_t, int);
template <int METHOD, int CTRL, bool COUNTED>
MixedFn mixed_by_solver(int solver) {
    if constexpr (METHOD == WIND_METHOD_RK2) {
        return k_mixed<METHOD, CTRL, WIND_SOLVER_LU_F64, WIND_SOLVER_LU_F64, COUNTED>;
    } else {
        switch (solver) {
        case WIND_SOLVER_GJE_F64:
            return k_mixed<METHOD, CTRL, WIND_SOLVER_GJE_F64, WIND_SOLVER_GJE_F64, COUNTED>;
        case WIND_SOLVER_LU_F64: return k_mixed<METHOD, CTRL, WIND_SOLVER_LU_F64, WIND_SOLVER_LU_F64, COUNTED>;
        case WIND_SOLVER_AUTO: return k_mixed<METHOD, CTRL, WIND_SOLVER_MIXED, WIND_SOLVER_LU_F64, COUNTED>;
        default:
            // (the MIXED team kernel has lists of its own)
            if constexpr (COUNTED) return nullptr;
            else return k_mixed<METHOD, CTRL, WIND_SOLVER_MIXED, WIND_SOLVER_MIXED, false>;
        }
    }
}
template <bool COUNTED>
MixedFn mixed_fn(int method, int ctrl, int solver) {
    if (method == WIND_METHOD_SIE)
        return ctrl == WIND_CTRL_GOLD ? mixed_by_solver<WIND_METHOD_SIE, WIND_CTRL_GOLD, COUNTED>(solver)
                                      : mixed_by_solver<WIND_METHOD_SIE, WIND_CTRL_DEVICE, COUNTED>(solver);
    return ctrl == WIND_CTRL_GOLD ? mixed_by_solver<WIND_METHOD_RK2, WIND_CTRL_GOLD, COUNTED>(solver)
                                  : mixed_by_solver<WIND_METHOD_RK2, WIND_CTRL_DEVICE, COUNTED>(solver);
}

}  // namespace wind
