// lane_kernel.cuh -- persistent thread-per-system integrator for the builtin
// networks (compile-time N <= 5): NR_test, StiffTrig, Katz96.
//
// Design (replaces cuda/common/kernel.cu:140-311, which ran one CTA of N
// threads per system with the matrices in global memory):
//  * the whole system -- state, Jacobian, inverse/factors -- lives in the
//    registers of one thread; no shared or global scratch besides the work
//    counter;
//  * persistent grid: a team of W lanes pulls the next system index from a
//    device work queue (atomic ticket) the moment it finishes one, so systems
//    with very different step counts do not idle a warp;
//  * speculative refinement: the W lanes of a team evaluate the next W
//    refinement levels h, h/2, ..., h/2^(W-1) of the same attempt at once and
//    keep the first that passes (or the one at the refinement cap).  Each
//    attempt is computed exactly as the serial controller would compute it,
//    so results and step counts are identical to the serial loop
//    (kernel.cu:191-296, common_gold.c:77-149); only latency changes.
#pragma once

#include "common.cuh"
#include "networks.cuh"
#include "solvers_reg.cuh"

namespace wind {

constexpr int LANE_THREADS = 128;
// Minimum resident blocks per SM the compiler must plan registers for: 4 (128
// registers) for the FP64 solvers by blocks.  65,536 Katz96 cells with the LU
// at atol 1e-8 / rtol 1e-6 took 42.0, 42.1, 43.2 and 47.1 ms at 3, 4, 5 and 6
// (64.6 ms with the full-width 5 x 5 LU), 8,000 cells through the drop-in with
// the Gauss-Jordan inverse 1.19, 1.17, 1.20 and 1.22 ms (2.87 ms full width).
// The mixed path keeps the uncapped allocation.
template <int SOLVER>
struct LaneMinBlocks {
    static constexpr int value = SOLVER == WIND_SOLVER_MIXED ? 1 : 4;
};

// One SIE or explicit-Euler substep of length h, in place on y, with the
// full-width solvers.
template <class Net, int METHOD, int CTRL, int SOLVER>
__device__ __forceinline__ void lane_substep_full(const double (&c)[Net::NC], xd h, xd (&y)[Net::N]) {
    constexpr int N = Net::N;
    xd f[N];
    Net::rhs(c, y, f);
    if (METHOD == WIND_METHOD_RK2) {
        // rk2_gold.c:31-34, kernel.cu:128-130: y += h*f
#pragma unroll
        for (int e = 0; e < N; e++) y[e] += h * f[e];
        return;
    }
    xd M[N * N];
#pragma unroll
    for (int e = 0; e < N * N; e++) M[e] = 0.0;
    Net::jac(c, y, M);
    if (SOLVER == WIND_SOLVER_GJE_F64) {
        if (CTRL == WIND_CTRL_GOLD) {
            // sie_gold.c:17-36: J = -h*J; diag += 1
#pragma unroll
            for (int e = 0; e < N * N; e++) M[e] = -h * M[e];
#pragma unroll
            for (int i = 0; i < N; i++) M[i * (N + 1)] += 1.0;
        } else {
            // kernel.cu:49-52: J[i][j] = (i==j) - J[i][j]*h
#pragma unroll
            for (int i = 0; i < N; i++)
#pragma unroll
                for (int j = 0; j < N; j++) M[i * N + j] = xd(i == j ? 1.0 : 0.0) - M[i * N + j] * h;
        }
        xd Inv[N * N];
        gje_invert_reg<N>(M, Inv);
        if (CTRL == WIND_CTRL_GOLD) {
            // matrix_ops.c:6-27 (transposed matvec), then sie_gold.c:72-74
            xd out[N];
#pragma unroll
            for (int r = 0; r < N; r++) out[r] = 0.0;
#pragma unroll
            for (int cc = 0; cc < N; cc++)
#pragma unroll
                for (int r = 0; r < N; r++) out[r] += Inv[cc * N + r] * f[cc];
#pragma unroll
            for (int e = 0; e < N; e++) y[e] += h * out[e];
        } else {
            // kernel.cu:116-125: y_j += (Inv[k][j]*f_k)*h, k ascending
#pragma unroll
            for (int k = 0; k < N; k++)
#pragma unroll
                for (int j = 0; j < N; j++) y[j] += Inv[k * N + j] * f[k] * h;
        }
        return;
    }
    // Standard orientation A[r][c] = delta_rc - h * J_rc, J_rc = Jt[c][r].
    if (SOLVER == WIND_SOLVER_LU_F64) {
        double A[N * N], rinv[N];
        int perm[N];
#pragma unroll
        for (int r = 0; r < N; r++)
#pragma unroll
            for (int cc = 0; cc < N; cc++)
                A[r * N + cc] = (r == cc ? 1.0 : 0.0) - h.v * M[cc * N + r].v;
        lu_factor_reg<N, double>(A, rinv, perm);
        double x[N];
#pragma unroll
        for (int e = 0; e < N; e++) x[e] = f[e].v;
        lu_solve_reg<N, double, double>(A, rinv, perm, x);
#pragma unroll
        for (int e = 0; e < N; e++) y[e] = y[e].v + h.v * x[e];
        return;
    }
    // MIXED: FP32 factor, FP64 residual, one refinement step.
    float Af[N * N], rinvf[N];
    int perm[N];
#pragma unroll
    for (int r = 0; r < N; r++)
#pragma unroll
        for (int cc = 0; cc < N; cc++)
            Af[r * N + cc] = (float)((r == cc ? 1.0 : 0.0) - h.v * M[cc * N + r].v);
    lu_factor_reg<N, float>(Af, rinvf, perm);
    double x[N];
#pragma unroll
    for (int e = 0; e < N; e++) x[e] = f[e].v;
    lu_solve_reg<N, float, double>(Af, rinvf, perm, x);
    // r = f - A x with A = I - h J (FP64, from Jt)
    double res[N];
#pragma unroll
    for (int r = 0; r < N; r++) {
        double acc = 0.0;
#pragma unroll
        for (int cc = 0; cc < N; cc++) acc = fma(M[cc * N + r].v, x[cc], acc);
        res[r] = f[r].v - (x[r] - h.v * acc);
    }
    lu_solve_reg<N, float, double>(Af, rinvf, perm, res);
#pragma unroll
    for (int e = 0; e < N; e++) y[e] = y[e].v + h.v * (x[e] + res[e]);
}

// The same, out of line, for the substeps whose block solve met an infinite
// or NaN value (a full-width elimination spreads those across blocks).
template <class Net, int CTRL, int SOLVER>
__device__ __noinline__ void lane_substep_redo(const double* c_in, double h, double* y_io) {
    double c[Net::NC];
    xd y[Net::N];
#pragma unroll
    for (int k = 0; k < Net::NC; k++) c[k] = c_in[k];
#pragma unroll
    for (int e = 0; e < Net::N; e++) y[e] = y_io[e];
    lane_substep_full<Net, WIND_METHOD_SIE, CTRL, SOLVER>(c, xd(h), y);
#pragma unroll
    for (int e = 0; e < Net::N; e++) y_io[e] = y[e].v;
}

// The SIE substep of the diagonal block of size n at equation O, from the
// system's f and Jt (both at the state in y): the stepped components go to
// out, the high words of its pivots (GJE_F64) and results into hi.
template <class Net, int CTRL, int SOLVER, int O, int n, bool TRI>
__device__ __forceinline__ void lane_block_step(const xd (&Jt)[Net::N * Net::N], const xd (&f)[Net::N], xd h,
                                                const xd (&y)[Net::N], xd (&out)[Net::N], int& hi) {
    constexpr int N = Net::N;
    if (SOLVER == WIND_SOLVER_GJE_F64) {
        xd M[n * n], Inv[n * n];
#pragma unroll
        for (int i = 0; i < n; i++)
#pragma unroll
            for (int j = 0; j < n; j++) {
                const xd e = Jt[(O + i) * N + O + j];
                if (CTRL == WIND_CTRL_GOLD) {
                    // sie_gold.c:17-36: J = -h*J; diag += 1
                    M[i * n + j] = -h * e;
                    if (i == j) M[i * n + j] += 1.0;
                } else {
                    // kernel.cu:49-52: J[i][j] = (i==j) - J[i][j]*h
                    M[i * n + j] = xd(i == j ? 1.0 : 0.0) - e * h;
                }
            }
        gje_invert_block<n, TRI>(M, Inv, hi);
        if (CTRL == WIND_CTRL_GOLD) {
            // matrix_ops.c:6-27 (transposed matvec), then sie_gold.c:72-74
#pragma unroll
            for (int r = 0; r < n; r++) {
                xd acc = Inv[r] * f[O];
#pragma unroll
                for (int cc = 1; cc < n; cc++) acc += Inv[cc * n + r] * f[O + cc];
                out[O + r] = y[O + r] + h * acc;
            }
        } else {
            // kernel.cu:116-125: y_j += (Inv[k][j]*f_k)*h, k ascending
#pragma unroll
            for (int j = 0; j < n; j++) {
                xd acc = y[O + j];
#pragma unroll
                for (int k = 0; k < n; k++) acc += Inv[k * n + j] * f[O + k] * h;
                out[O + j] = acc;
            }
        }
    } else {
        // Standard orientation A[r][c] = delta_rc - h * J_rc, J_rc = Jt[c][r].
        double A[n * n], x[n];
#pragma unroll
        for (int r = 0; r < n; r++)
#pragma unroll
            for (int cc = 0; cc < n; cc++)
                A[r * n + cc] = (r == cc ? 1.0 : 0.0) - h.v * Jt[(O + cc) * N + O + r].v;
#pragma unroll
        for (int e = 0; e < n; e++) x[e] = f[O + e].v;
        lu_solve_block<n, TRI>(A, x);
#pragma unroll
        for (int e = 0; e < n; e++) {
            hi = max(hi, mag_hi(x[e]));
            out[O + e] = y[O + e].v + h.v * x[e];
        }
    }
    if (SOLVER == WIND_SOLVER_GJE_F64) {
#pragma unroll
        for (int e = 0; e < n; e++) hi = max(hi, mag_hi(out[O + e].v));
    }
}

// One SIE or explicit-Euler substep of length h, in place on y: the FP64
// solvers by the network's diagonal blocks.
template <class Net, int METHOD, int CTRL, int SOLVER>
__device__ __forceinline__ void lane_substep(const double (&c)[Net::NC], xd h, xd (&y)[Net::N]) {
    if constexpr (METHOD == WIND_METHOD_RK2 || SOLVER == WIND_SOLVER_MIXED) {
        lane_substep_full<Net, METHOD, CTRL, SOLVER>(c, h, y);
    } else {
        constexpr int N = Net::N;
        static_assert(Net::B0 + Net::B1 == N, "blocks cover the network");
        xd f[N], Jt[N * N], out[N];
        Net::rhs(c, y, f);
#pragma unroll
        for (int e = 0; e < N * N; e++) Jt[e] = 0.0;
        Net::jac(c, y, Jt);
        int hi = 0;
        lane_block_step<Net, CTRL, SOLVER, 0, Net::B0, false>(Jt, f, h, y, out, hi);
        if constexpr (Net::B1 > 0)
            lane_block_step<Net, CTRL, SOLVER, Net::B0, Net::B1, Net::TRI1>(Jt, f, h, y, out, hi);
        if (hi >= HI_INF) {
            double cs[Net::NC], ys[N];
#pragma unroll
            for (int k = 0; k < Net::NC; k++) cs[k] = c[k];
#pragma unroll
            for (int e = 0; e < N; e++) ys[e] = y[e].v;
            lane_substep_redo<Net, CTRL, SOLVER>(cs, h.v, ys);
#pragma unroll
            for (int e = 0; e < N; e++) out[e] = ys[e];
        }
#pragma unroll
        for (int e = 0; e < N; e++) y[e] = out[e];
    }
}

// take_step (sie_gold.c:38-51) / innerstep (kernel.cu:69-91): nsub substeps
// over [t0, t0+H]; DEVICE clamps each substep with fmin.
template <class Net, int METHOD, int CTRL, int SOLVER>
__device__ __forceinline__ void lane_take_step(const double (&c)[Net::NC], double t0, double H,
                                               int nsub, xd (&y)[Net::N]) {
    const double t1 = t0 + H;
    // (t1-t0)/nsub for nsub in {1,2}: multiplying by 1 or 0.5 rounds the
    // same real number, so it equals the division bit for bit
    double h = (t1 - t0) * (nsub == 1 ? 1.0 : 0.5);
    double t = t0;
    for (int i = 0; i < nsub; i++) {
        if (CTRL == WIND_CTRL_DEVICE) h = fmin(t1 - t, h);
        lane_substep<Net, METHOD, CTRL, SOLVER>(c, xd(h), y);
        t += h;
    }
}

// One attempt: the full step into y1 and the two half steps into y2, written
// as straight-line code so the full step and the first half step -- which
// are independent -- can be interleaved by the scheduler; the attempt's
// critical path is then two substeps instead of three.  Each substep is the
// same arithmetic as lane_take_step's (take_step, sie_gold.c:38-51;
// innerstep, kernel.cu:69-91).
template <class Net, int METHOD, int CTRL, int SOLVER>
__device__ __forceinline__ void lane_attempt(const double (&c)[Net::NC], double t0, double H,
                                             xd (&y1)[Net::N], xd (&y2)[Net::N]) {
    const double t1 = t0 + H;
    double hf = (t1 - t0) * 1.0;
    double hh = (t1 - t0) * 0.5;
    if (CTRL == WIND_CTRL_DEVICE) {
        hf = fmin(t1 - t0, hf);
        hh = fmin(t1 - t0, hh);
    }
    lane_substep<Net, METHOD, CTRL, SOLVER>(c, xd(hf), y1);
    lane_substep<Net, METHOD, CTRL, SOLVER>(c, xd(hh), y2);
    const double tm = t0 + hh;
    double hh2 = hh;
    if (CTRL == WIND_CTRL_DEVICE) hh2 = fmin(t1 - tm, hh);
    lane_substep<Net, METHOD, CTRL, SOLVER>(c, xd(hh2), y2);
}

// Lanes of the warp that point at the same owner form a team.  With a
// systems in the warp (owners), lane i works on owner (i mod a) at
// refinement level (i div a): lanes are spread round-robin, so team sizes
// differ by at most one and the lowest lane of a team carries level 0.

// Bits 0, n, 2n, ... below 32.
__device__ __forceinline__ unsigned every_nth(int n) {
    unsigned m = 1u;
    for (int s = n; s < 32; s <<= 1) m |= m << s;
    return m;
}
// Position of the n-th (from 0) set bit of m.
__device__ __forceinline__ int nth_bit(unsigned m, int n) {
    int pos = 0;
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
        const int c = __popc(m & ((1u << w) - 1u));
        if (n >= c) {
            n -= c;
            m >>= w;
            pos += w;
        }
    }
    return pos;
}
// x halved n times (0 <= n <= 32): one exact multiplication while the result
// stays normal.
__device__ __forceinline__ double halved(double x, int n) {
    const int e = (__double2hiint(x) >> 20) & 0x7ff;
    if (e > 32) return x * __hiloint2double((1023 - n) << 20, 0);
    for (int q = 0; q < n; q++) x /= 2.0;
    return x;
}

// Persistent kernel.  Every lane owns at most one system (its state lives in
// the owner's registers).  Each round:
//  1. lanes without a system take the next ticket from the work queue;
//  2. the a owned systems of the warp are assigned all 32 lanes round-robin;
//     a lane fetches its assigned system's state from the owner by shuffle;
//  3. each lane evaluates one attempt (full step + two half steps + error
//     test) at its refinement level;
//  4. per team, the lowest level that passes (or the one at the cap) is the
//     accepted attempt; every level below it is exactly the serial
//     controller's rejected attempt, so the owner applies "levels refined,
//     then accept" with results identical to the serial loop.
// While the queue is full every lane owns a system and a round is one attempt
// per system (no speculation, no waste).  As the queue drains, idle lanes join
// the remaining systems, which cuts the tail of slow systems by up to the
// refinement cap.  Only lanes below `opw` (owners per warp) take tickets; the
// others start as helpers, which spreads a small batch over many warps
// (opw = 32 / initial lanes per system).
template <class Net, int METHOD, int CTRL, int SOLVER>
__global__ void __launch_bounds__(LANE_THREADS, LaneMinBlocks<SOLVER>::value) k_lane(const KParams p, const int opw) {
    constexpr int N = Net::N;
    constexpr int NC = Net::NC;
    constexpr int CAP = Cap<METHOD, CTRL>::value;
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint64_t t_start = p.timeout_ns ? global_ns() : 0;
    const double tend = p.tend;

    // owner state
    bool has = false, drained = (lane >= opw);
    int64_t s_own = -1;
    double y_own[N];
    double t_own = 0.0, h_own = 0.0;
    int u_own = 0;
    int64_t a_own = 0;
    int32_t st_own = WIND_SYS_OK;
    // worker cache
    int64_t s_work = -1;
    double c[NC];
    // the warp's assignment, kept while the owners stay the same lanes
    unsigned owners_at = 0u, team = 0u;
    int src = lane, r = 0;

    while (true) {
        // 1. refill: take new tickets while without a system
        while (!has && !drained) {
            const unsigned long long ticket = atomicAdd(&p.counters[CNT_QUEUE], 1ull);
            if ((int64_t)ticket >= p.nsys) { drained = true; break; }
            s_own = (int64_t)ticket;
#pragma unroll
            for (int i = 0; i < N; i++) y_own[i] = p.y[s_own * N + i];
            t_own = p.tnow;
            h_own = p.h0;
            u_own = 0;
            a_own = 0;
            st_own = WIND_SYS_OK;
            has = true;
        }
        // finish systems that are done
        if (has) {
            bool fin = !(t_own < tend);
            if (!fin && a_own >= p.max_attempts) { st_own |= WIND_SYS_MAX_ATTEMPTS; fin = true; }
            if (!fin && p.timeout_ns && global_ns() - t_start > p.timeout_ns) {
                st_own |= WIND_SYS_TIMEOUT;
                fin = true;
            }
            if (fin) {
#pragma unroll
                for (int i = 0; i < N; i++) {
                    if (!finite64(y_own[i])) st_own |= WIND_SYS_NONFINITE;
                    p.y[s_own * N + i] = y_own[i];
                }
                if (p.sys_status) p.sys_status[s_own] = st_own;
                if (p.sys_nsteps) p.sys_nsteps[s_own] = 3 * a_own;
                atomicAdd(&p.counters[CNT_STEPS], (unsigned long long)(3 * a_own));
                has = false;
                continue;  // refill before the warp-wide round
            }
        }
        const unsigned owners = __ballot_sync(FULL, has);
        if (owners == 0u) {
            if (__all_sync(FULL, drained)) break;
            continue;
        }
        // 2. assignment and state fetch.  While every lane owns a system each
        // works on its own at level 0: nothing to fetch.
        const bool full = owners == FULL;
        if (owners != owners_at) {
            owners_at = owners;
            const int nact = __popc(owners);
            r = lane / nact;
            src = nth_bit(owners, lane - r * nact);
            team = every_nth(nact) << __popc(owners & ((1u << lane) - 1u));  // (owners')
        }
        int64_t s_j = s_own, a_j = a_own;
        double t_j = t_own, h_j = h_own;
        int u_j = u_own;
        xd y[N];
#pragma unroll
        for (int i = 0; i < N; i++) y[i] = y_own[i];
        if (!full) {
            s_j = __shfl_sync(FULL, s_own, src);
            t_j = __shfl_sync(FULL, t_own, src);
            h_j = __shfl_sync(FULL, h_own, src);
            u_j = __shfl_sync(FULL, u_own, src);
            a_j = __shfl_sync(FULL, a_own, src);
#pragma unroll
            for (int i = 0; i < N; i++) y[i] = __shfl_sync(FULL, y_own[i], src);
        }
        if (s_j != s_work) {
            s_work = s_j;
#pragma unroll
            for (int k = 0; k < NC; k++) c[k] = __ldg(p.constants + s_j * p.n_const + k);
        }
        // 3. one attempt at level r: kernel.cu:195 / common_gold.c:79 clamp,
        //    then r halvings (kernel.cu:262 / common_gold.c:123)
        const double hw = fmin(tend - t_j, h_j);
        const double hl = halved(hw, r);
        const int lvl = u_j + r;
        const bool valid = (lvl <= CAP) && (a_j + r < p.max_attempts);
        xd y1[N], y2[N];
#pragma unroll
        for (int i = 0; i < N; i++) { y1[i] = y[i]; y2[i] = y[i]; }
        bool err = true;
        if (valid) {
            lane_attempt<Net, METHOD, CTRL, SOLVER>(c, t_j, hl, y1, y2);
            err = false;
#pragma unroll
            for (int i = 0; i < N; i++) err |= elem_error<METHOD, CTRL>(y1[i], y2[i], p.atol, p.rtol);
        }
        const bool acc = valid && (!err || lvl == CAP);
        // 4. owners apply their team's outcome
        int take = lane;   // lane whose attempt this owner adopts (self = none)
        int done = 1;      // attempts consumed this round
        bool accepted = acc;
        const unsigned bal = full ? 0u : __ballot_sync(FULL, acc);
        if (!full && has) {
            accepted = false;
            const unsigned mine = bal & team;
            if (mine) {
                take = __ffs(mine) - 1;
                done = __popc(team & ((1u << take) - 1u)) + 1;
                accepted = true;
            } else {
                // every level of the team refined (the cap level would accept)
                int lim = __popc(team);
                if (a_own + lim > p.max_attempts) lim = (int)(p.max_attempts - a_own);
                done = lim;
            }
        }
        double ytake[N];
#pragma unroll
        for (int i = 0; i < N; i++)
            ytake[i] = (METHOD == WIND_METHOD_RK2) ? (xd(2.0) * y2[i] - y1[i]).v : y2[i].v;
        double htake = hl;
        if (!full) {
            htake = __shfl_sync(FULL, hl, take);
#pragma unroll
            for (int i = 0; i < N; i++) ytake[i] = __shfl_sync(FULL, ytake[i], take);
        }
        if (has) {
            a_own += done;
            if (accepted) {
#pragma unroll
                for (int i = 0; i < N; i++) y_own[i] = ytake[i];
                u_own = 0;
                if (t_own + htake == t_own) {
                    st_own |= WIND_SYS_STALLED;
                    t_own = tend;  // finishes at the top of the next round
                } else {
                    t_own += htake;
                    // kernel.cu:285-294: RK2 doubles h, SIE goes for gold
                    h_own = (METHOD == WIND_METHOD_RK2) ? htake * 2 : tend - t_own;
                }
            } else {
                u_own += done;
                h_own = halved(fmin(tend - t_own, h_own), done);
            }
        }
    }
}

}  // namespace wind
