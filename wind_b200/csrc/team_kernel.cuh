// team_kernel.cuh -- persistent team-per-system integrator for runtime
// mass-action networks with N <= 32 (optionally with a dense linear term):
// SIE with the reference's Gauss-Jordan inverse, and RK2.
//
// A team is NMAX lanes of one warp (NMAX = 8, 16 or 32).  Lane l owns equation
// l: its components of the state and the candidates live in registers, and it
// evaluates f_l and Jacobian column l (d f_l / d y_*) from the list of the
// reactions that touch species l (ids ascending, the sequential order of the
// mass-action contract restricted to the lane's elements).
//
// Gauss-Jordan by columns.  The reference inverts M by full-width row
// operations on [M | Inv] (gje_gold.c:56-134).  At pivot i of its downward
// pass only N of the 2N columns still hold anything but exact zeros and ones:
// M's columns right of i and Inv's columns up to i.  Lane t therefore holds
// M's column t until step t, hands it to the team (its entries are the
// multipliers of step t below the pivot, and of the upward pass above it) and
// carries Inv's column t from there on.  A step is one division and N - 1 - i
// multiply-subtracts per lane, on values the lane owns; the upward pass reads
// the handed-over columns and needs no exchange at all, and the product with f
// is local.  Every operation on a nonzero element is the reference's, in its
// order, so the result is the same bit for bit; the operations left out are
// x - f*0 and 0/s, which return their operand whenever s and f are finite and
// s is not zero.  A pivot that is zero or not finite, or a result that is not
// finite, sends the substep to the full-width elimination (team_gje_general).
//
// What bounds it: the chain of N pivot steps (hand-over through shared memory,
// one division, the first update) and the lane's incidence list.  The full-width
// row form this replaced spent about 130 us per substep at N = 16, in 2N
// divisions by one lane per step and in instruction fetch: 1,000 systems of 16
// species (160 reactions, dt = 1e-3, atol = rtol = 5e-3) took 219.4 ms, now
// 16.4 ms.
//
// One loop turn is one substep of every team of the warp, whatever part of its
// attempt the team is in, so teams never wait for each other's attempts or
// systems.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "networks.cuh"

namespace wind {

constexpr int TEAM_MAXN = 32;

// An incidence of species l: reaction id, reactants a and b, and how often l
// is consumed (nn) and produced (np) by it.
__device__ __forceinline__ uint32_t team_pack(int rr, int a, int b, int nn, int np) {
    return (uint32_t)rr | ((uint32_t)a << 16) | ((uint32_t)b << 21) | ((uint32_t)nn << 26) |
           ((uint32_t)np << 28);
}

struct TeamLayout {
    // byte offsets inside one team's shared slice: the Jacobian at the
    // accepted state, the Jacobian of the second half step / the columns handed
    // over by the elimination (SIE only), vectors, the dense term, rates and
    // incidence lists
    int jy, w, vec, lt, rates, inc_off, inc, bytes;
    __host__ __device__ static int align16(int x) { return (x + 15) & ~15; }
    __host__ __device__ TeamLayout(int nmax, int R, bool lin, bool matrices) {
        const int mat = matrices ? nmax * nmax * 8 : 0;
        int off = 0;
        jy = off; off = align16(off + mat);
        w = off; off = align16(off + mat);
        vec = off; off = align16(off + 2 * nmax * 8);
        lt = off; off = align16(off + (lin ? nmax * nmax * 4 : 0));
        rates = off; off = align16(off + R * 8);
        inc_off = off; off = align16(off + (nmax + 1) * 4);
        inc = off; off = align16(off + 4 * R * 4);
        bytes = off;
    }
};

// Team-local synchronisation: teams never span warps here.
__device__ __forceinline__ void team_sync(unsigned mask) { __syncwarp(mask); }

template <int NMAX>
struct TeamCtx {
    unsigned mask;
    int l;          // lane within team
    int leader;     // warp lane of the team's lane 0
    int N;
    double* jy;     // [NMAX*NMAX] Jt at the accepted state, Jt[i*NMAX + j] = d f_j / d y_i
    double* w;      // [NMAX*NMAX] Jt of the second half step; handed-over columns
    double* v;      // [NMAX] state being stepped
    double* f;      // [NMAX] RHS at v
    const float* LT;   // [NMAX*NMAX] LT[i*NMAX+j] = L[j][i], or null
    const double* rates;      // [R]
    const int* inc_off;       // [NMAX+1] CSR offsets
    const uint32_t* inc;      // packed incidences (team_pack)
};

// x - d (nn times), then x + d (np times), nn + np >= 1, each rounded.
__device__ __forceinline__ xd team_apply(xd x, xd d, int nn, int np) {
    x = x + (nn ? -d : d);
    if (nn + np > 1) {
        x = x + (nn == 2 ? -d : d);
        if (nn + np > 2) {
            x = x + d;
            if (nn + np > 3) x = x + d;
        }
    }
    return x;
}

// f_l and, with JAC, column l of Jt into J, for the current v.  The loads of
// four incidences are in flight before the first is used.
template <int NMAX, bool JAC>
__device__ __forceinline__ void team_rhs_jac(const TeamCtx<NMAX>& c, double* J) {
    const int l = c.l;
    if (l < c.N) {
        xd acc = 0.0;
        if (c.LT) {
            for (int k = 0; k < c.N; k++) acc += xd((double)c.LT[k * NMAX + l]) * xd(c.v[k]);
            if (JAC)
                for (int i = 0; i < c.N; i++) J[i * NMAX + l] = (double)c.LT[i * NMAX + l];
        } else if (JAC) {
            for (int i = 0; i < c.N; i++) J[i * NMAX + l] = 0.0;
        }
        const int e1 = c.inc_off[l + 1];
        for (int e = c.inc_off[l]; e < e1; e += 4) {
            uint32_t q[4];
            double k[4], ya[4], yb[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                q[u] = c.inc[e + u < e1 ? e + u : e];
                k[u] = c.rates[q[u] & 0xffffu];
                ya[u] = c.v[(q[u] >> 16) & 31u];
                yb[u] = c.v[(q[u] >> 21) & 31u];
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (e + u < e1) {
                    const int nn = (q[u] >> 26) & 3, np = q[u] >> 28;
                    const xd db = xd(k[u]) * xd(ya[u]);
                    acc = team_apply(acc, db * xd(yb[u]), nn, np);
                    if (JAC) {
                        double* ra = J + ((q[u] >> 16) & 31u) * NMAX + l;
                        double* rb = J + ((q[u] >> 21) & 31u) * NMAX + l;
                        *ra = team_apply(*ra, xd(k[u]) * xd(yb[u]), nn, np).v;
                        *rb = team_apply(*rb, db, nn, np).v;
                    }
                }
            }
        }
        c.f[l] = acc.v;
    }
    team_sync(c.mask);
}

// Element i of row or column l of M = I - h Jt, in the controller's order:
// sie_gold.c:17-36 (GOLD), kernel.cu:49-52 (DEVICE).
template <int CTRL>
__device__ __forceinline__ xd team_matrix_elem(double j, double h, bool diag) {
    if (CTRL == WIND_CTRL_GOLD) {
        xd m = -xd(h) * xd(j);
        if (diag) m += 1.0;
        return m;
    }
    return xd(diag ? 1.0 : 0.0) - xd(j) * xd(h);
}

// The state component stepped with the inverse's column l (or row storage
// read down column l): matrix_ops.c:6-27 then sie_gold.c:72-74 (GOLD);
// kernel.cu:121-125 (DEVICE).
template <int CTRL>
struct TeamProduct {
    xd acc;
    double h;
    __device__ __forceinline__ TeamProduct(double y, double hh) : acc(CTRL == WIND_CTRL_GOLD ? 0.0 : y), h(hh) {}
    __device__ __forceinline__ void add(xd inv, xd f) {
        if (CTRL == WIND_CTRL_GOLD) acc += inv * f;
        else acc += inv * f * xd(h);
    }
    __device__ __forceinline__ double result(double y) const {
        return CTRL == WIND_CTRL_GOLD ? (xd(y) + xd(h) * acc).v : acc.v;
    }
};

// The full-width elimination on rows held one per lane, for the substeps whose
// pivots or results are not finite: evaluates f and Jt at v itself (into w),
// uses jy as the exchange buffer and returns the stepped component.
template <int NMAX, int CTRL>
__device__ __noinline__ double team_gje_general(unsigned mask, int l, int leader, int N, double* jy, double* w,
                                                double* v, double* f, const float* LT, const double* rates,
                                                const int* inc_off, const uint32_t* inc, double h) {
    TeamCtx<NMAX> c;
    c.mask = mask; c.l = l; c.leader = leader; c.N = N;
    c.jy = jy; c.w = w; c.v = v; c.f = f;
    c.LT = LT; c.rates = rates; c.inc_off = inc_off; c.inc = inc;
    team_rhs_jac<NMAX, true>(c, w);
    xd Mr[NMAX], Ir[NMAX];
#pragma unroll
    for (int t = 0; t < NMAX; t++) {
        Mr[t] = team_matrix_elem<CTRL>((l < N && t < N) ? w[l * NMAX + t] : 0.0, h, t == l);
        Ir[t] = (t == l) ? 1.0 : 0.0;
    }
    constexpr int ROW = 2 * NMAX;
    // gjeUFactor (gje_gold.c:56-100)
#pragma unroll
    for (int i = 0; i < NMAX; i++) {
        if (i < N) {
            if (l == i) {
                const xd s = Mr[i];
#pragma unroll
                for (int t = 0; t < NMAX; t++) { Mr[t] /= s; Ir[t] /= s; }
#pragma unroll
                for (int t = 0; t < NMAX; t++) { jy[t] = Mr[t].v; jy[NMAX + t] = Ir[t].v; }
            }
            team_sync(mask);
            if (l > i && l < N) {
                const xd fct = Mr[i];
#pragma unroll
                for (int t = 0; t < NMAX; t++) {
                    Mr[t] -= fct * xd(jy[t]);
                    Ir[t] -= fct * xd(jy[NMAX + t]);
                }
            }
            team_sync(mask);
        }
    }
    // gjeLFactor (gje_gold.c:102-134): pivot rows bottom-up
#pragma unroll
    for (int b = NMAX - 1; b >= 0; b--) {
        if (b < N) {
            if (l == b) {
#pragma unroll
                for (int t = 0; t < NMAX; t++) { jy[t] = Mr[t].v; jy[NMAX + t] = Ir[t].v; }
            }
            team_sync(mask);
            if (l < b) {
                const xd fct = Mr[b];
#pragma unroll
                for (int t = 0; t < NMAX; t++) {
                    Mr[t] -= fct * xd(jy[t]);
                    Ir[t] -= fct * xd(jy[NMAX + t]);
                }
            }
            team_sync(mask);
        }
    }
    // inverse rows to shared memory, then the product by columns
    if (l < N) {
#pragma unroll
        for (int t = 0; t < NMAX; t++) w[l * NMAX + t] = Ir[t].v;
    }
    team_sync(mask);
    double out = 0.0;
    if (l < N) {
        TeamProduct<CTRL> prod(v[l], h);
        for (int k = 0; k < N; k++) prod.add(w[k * NMAX + l], f[k]);
        out = prod.result(v[l]);
    }
    team_sync(mask);
    static_assert(ROW <= NMAX * NMAX, "exchange buffer");
    return out;
}

// One SIE substep of size h from the state in v with f in f and Jt in J (jy
// or w); returns the stepped component l.  Column form of the file comment.
// `clean` is cleared when the full-width elimination had to be used, which
// overwrites jy.
template <int NMAX, int CTRL>
__device__ __forceinline__ double team_gje_step(const TeamCtx<NMAX>& c, const double* J, double h, bool& clean) {
    const int l = c.l, N = c.N;
    double* F = c.w;  // columns handed over, [step][row]
    xd x[NMAX];
#pragma unroll
    for (int t = 0; t < NMAX; t++)
        x[t] = team_matrix_elem<CTRL>((l < N && t < N) ? J[t * NMAX + l] : 0.0, h, t == l);
    bool ok = true;
    team_sync(c.mask);  // J may be w: every column is in registers before the first is handed over
#pragma unroll
    for (int i = 0; i < NMAX; i++) {
        if (i < N) {
            double* Fi = F + i * NMAX;
            if (l == i) {
#pragma unroll
                for (int t = 0; t < NMAX; t += 2)
                    *reinterpret_cast<double2*>(Fi + t) = make_double2(x[t].v, x[t + 1].v);
#pragma unroll
                for (int t = 0; t < NMAX; t++) x[t] = (t == i) ? 1.0 : 0.0;  // column i of Inv starts
            }
            team_sync(c.mask);
            const xd s = Fi[i];
            ok = ok && s.v != 0.0 && finite64(s.v);
            x[i] = x[i] / s;
#pragma unroll
            for (int k = i + 1; k < NMAX; k++) x[k] -= xd(Fi[k]) * x[i];
        }
    }
#pragma unroll
    for (int b = NMAX - 1; b > 0; b--) {
        if (b < N) {
            const double* Fb = F + b * NMAX;
#pragma unroll
            for (int k = 0; k < b; k++) x[k] -= xd(Fb[k]) * x[b];
        }
    }
    double out = 0.0;
    if (l < N) {
        TeamProduct<CTRL> prod(c.v[l], h);
#pragma unroll
        for (int k = 0; k < NMAX; k++)
            if (k < N) prod.add(x[k], c.f[k]);
        out = prod.result(c.v[l]);
        ok = ok && finite64(out);
    }
    if (!__all_sync(c.mask, ok)) {
        out = team_gje_general<NMAX, CTRL>(c.mask, l, c.leader, N, c.jy, c.w, c.v, c.f, c.LT, c.rates,
                                           c.inc_off, c.inc, h);
        clean = false;
    }
    return out;
}

// Stage system s: rates, the dense term transposed, and the per-species
// incidence lists (reaction ids ascending).  A species index >= N marks the
// system BAD_INPUT (returned) and nothing of it is read again.
template <int NMAX>
__device__ __forceinline__ bool team_stage(const TeamCtx<NMAX>& c, const KParams& p, int64_t s, double* rates,
                                           int* inc_off, uint32_t* inc, float* LT) {
    const int N = c.N, R = p.n_react, l = c.l;
    const uint2* sp = reinterpret_cast<const uint2*>(p.species) + s * R;
    bool bad = false;
    for (int r = l; r < R; r += NMAX) {
        rates[r] = p.rates[s * R + r];
        const uint2 q = __ldg(sp + r);
        const unsigned nn = (unsigned)N;
        bad = bad || (q.x & 0xffffu) >= nn || (q.x >> 16) >= nn || (q.y & 0xffffu) >= nn || (q.y >> 16) >= nn;
    }
    if (__any_sync(c.mask, bad)) return true;
    const unsigned ul = (unsigned)l;
    if (l < N) {
        int cnt = 0;
        for (int r = 0; r < R; r++) {
            const uint2 q = __ldg(sp + r);
            cnt += ((q.x & 0xffffu) == ul) | ((q.x >> 16) == ul) | ((q.y & 0xffffu) == ul) | ((q.y >> 16) == ul);
        }
        inc_off[l + 1] = cnt;
    }
    team_sync(c.mask);
    if (l == 0) {
        inc_off[0] = 0;
        for (int j = 0; j < N; j++) inc_off[j + 1] += inc_off[j];
    }
    team_sync(c.mask);
    if (l < N) {
        int o = inc_off[l];
        for (int r = 0; r < R; r++) {
            const uint2 q = __ldg(sp + r);
            const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
            const int nn = (a == l) + (b == l), np = (cc == l) + (d == l);
            if (nn + np) inc[o++] = team_pack(r, a, b, nn, np);
        }
        if (LT) {
            const float* Lg = p.linear + s * (int64_t)N * N;
            for (int k = 0; k < N; k++) LT[k * NMAX + l] = Lg[l * N + k];
        }
    }
    team_sync(c.mask);
    return false;
}

// The persistent team loop over one group's systems: the first `tpw` teams of
// every warp (of the block's first `teams` teams) take tickets from the group's
// queue until it is empty.  `smem_raw` holds `teams` team slices.
template <int NMAX, int METHOD, int CTRL>
__device__ __forceinline__ void team_run(const KParams& p, unsigned char* smem_raw, int teams, int tpw) {
    constexpr int CAP = Cap<METHOD, CTRL>::value;
    constexpr bool SIE = METHOD == WIND_METHOD_SIE;
    const bool lin = p.linear != nullptr;
    const TeamLayout lay(NMAX, p.n_react, lin, SIE);
    const int lane = threadIdx.x & 31;
    const int team = (threadIdx.x >> 5) * tpw + lane / NMAX;
    if (lane / NMAX >= tpw || team >= teams) return;
    TeamCtx<NMAX> c;
    c.l = lane % NMAX;
    c.leader = lane - c.l;
    c.mask = (NMAX >= 32) ? 0xffffffffu : (((1u << NMAX) - 1u) << c.leader);
    c.N = p.n_eq;
    unsigned char* base = smem_raw + team * lay.bytes;
    c.jy = reinterpret_cast<double*>(base + lay.jy);
    c.w = reinterpret_cast<double*>(base + lay.w);
    c.v = reinterpret_cast<double*>(base + lay.vec);
    c.f = c.v + NMAX;
    float* LT = lin ? reinterpret_cast<float*>(base + lay.lt) : nullptr;
    double* rates = reinterpret_cast<double*>(base + lay.rates);
    int* inc_off = reinterpret_cast<int*>(base + lay.inc_off);
    uint32_t* inc = reinterpret_cast<uint32_t*>(base + lay.inc);
    c.LT = LT;
    c.rates = rates;
    c.inc_off = inc_off;
    c.inc = inc;
    const int N = c.N, l = c.l;
    const uint64_t t_start = p.timeout_ns ? global_ns() : 0;
    const double tend = p.tend;

    enum { ATTEMPT, FULL, HALF1, HALF2 };
    int phase = ATTEMPT;
    int64_t s = -1, attempts = 0;
    double y = 0.0, y1 = 0.0, vh = 0.0, fy = 0.0;
    double tnow = 0.0, h = 0.0, hf = 0.0, h1 = 0.0, h2 = 0.0, h_vh = 0.0;
    int unsolved = 0;
    int32_t st = WIND_SYS_OK;
    bool stop = false;
    bool fj_ok = false;  // fy and jy belong to y
    bool vh_ok = false;  // vh is the substep of size h_vh from y
    while (true) {
        // ---- between attempts: finish, take the next system, set the sizes
        while (phase == ATTEMPT) {
            if (s < 0) {
                unsigned long long ticket = 0;
                if (l == 0) ticket = atomicAdd(&p.counters[CNT_QUEUE], 1ull);
                s = (int64_t)__shfl_sync(c.mask, ticket, c.leader);
                if (s >= p.nsys) return;
                stop = team_stage<NMAX>(c, p, s, rates, inc_off, inc, LT);
                st = stop ? WIND_SYS_BAD_INPUT : WIND_SYS_OK;
                y = (l < N) ? p.y[s * N + l] : 0.0;
                tnow = p.tnow;
                h = p.h0;
                unsolved = 0;
                attempts = 0;
                fj_ok = vh_ok = false;
            }
            if (!stop && tnow < tend) {
                if (attempts >= p.max_attempts) {
                    st |= WIND_SYS_MAX_ATTEMPTS;
                    stop = true;
                } else if (p.timeout_ns) {
                    // the leader's clock decides for the whole team
                    const int late = global_ns() - t_start > p.timeout_ns;
                    if (__shfl_sync(c.mask, late, c.leader)) {
                        st |= WIND_SYS_TIMEOUT;
                        stop = true;
                    }
                }
            }
            if (stop || !(tnow < tend)) {
                const bool bad = (l < N) && !finite64(y);
                if (__any_sync(c.mask, bad)) st |= WIND_SYS_NONFINITE;
                if (l < N) p.y[s * N + l] = y;
                if (l == 0) {
                    if (p.sys_status) p.sys_status[s] = st;
                    if (p.sys_nsteps) p.sys_nsteps[s] = 3 * attempts;
                    atomicAdd(&p.counters[CNT_STEPS], (unsigned long long)(3 * attempts));
                }
                team_sync(c.mask);
                s = -1;
                continue;
            }
            attempts++;
            h = fmin(tend - tnow, h);
            const double t1 = tnow + h;
            // (t1-tnow)/nsub for nsub in {1,2}: multiplying by 1 or 0.5 rounds
            // the same real number, so it equals the division bit for bit
            hf = t1 - tnow;
            h1 = (t1 - tnow) * 0.5;
            if (CTRL == WIND_CTRL_DEVICE) h1 = fmin(t1 - tnow, h1);
            h2 = (CTRL == WIND_CTRL_DEVICE) ? fmin(t1 - (tnow + h1), h1) : h1;
            // after a refinement the full step is the refined attempt's first
            // half step: the same state, Jacobian and (unless t1 rounded
            // differently) size, so the same bits
            phase = FULL;
            if (vh_ok && hf == h_vh) {
                y1 = vh;
                phase = HALF1;
            }
        }
        // ---- one substep
        const bool second = phase == HALF2;
        const double hs = phase == FULL ? hf : (second ? h2 : h1);
        const double v = second ? vh : y;
        team_sync(c.mask);
        if (l < N) c.v[l] = v;
        team_sync(c.mask);
        if (second || !fj_ok) {
            team_rhs_jac<NMAX, SIE>(c, second ? c.w : c.jy);
            if (!second) {
                if (l < N) fy = c.f[l];
                fj_ok = true;
            }
        } else {
            if (l < N) c.f[l] = fy;
            team_sync(c.mask);
        }
        double out;
        if (SIE) {
            bool clean = true;
            out = team_gje_step<NMAX, CTRL>(c, second ? c.w : c.jy, hs, clean);
            if (!clean) fj_ok = false;
        } else {
            // rk2_gold.c:31-34, kernel.cu:128-130: y += h*f
            out = (l < N) ? (xd(v) + xd(hs) * xd(c.f[l])).v : 0.0;
        }
        if (phase == FULL) {
            y1 = out;
            phase = HALF1;
        } else if (phase == HALF1) {
            vh = out;
            h_vh = h1;
            phase = HALF2;
        } else {
            bool err = false;
            if (l < N) err = elem_error<METHOD, CTRL>(xd(y1), xd(out), p.atol, p.rtol);
            err = __any_sync(c.mask, err);
            if (err && unsolved < CAP) {
                unsolved++;
                h /= 2.0;
                vh_ok = true;
            } else {
                unsolved = 0;
                y = (METHOD == WIND_METHOD_RK2) ? (xd(2.0) * xd(out) - xd(y1)).v : out;
                fj_ok = vh_ok = false;
                if (tnow + h == tnow) {
                    st |= WIND_SYS_STALLED;
                    stop = true;
                } else {
                    tnow += h;
                    h = (METHOD == WIND_METHOD_RK2) ? h * 2 : tend - tnow;
                }
            }
            phase = ATTEMPT;
        }
    }
}

template <int NMAX, int METHOD, int CTRL>
__global__ void __launch_bounds__(32) k_team(const KParams p, int tpw) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    team_run<NMAX, METHOD, CTRL>(p, smem_raw, tpw, tpw);
}

}  // namespace wind
