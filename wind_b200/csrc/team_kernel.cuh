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
// Both passes are loops of one step's code (two widths), the rows moving up one
// register per step: unrolled they were 2,000 instructions at N = 16 and 6,000 at
// N = 32, and waited for instruction fetch (68,800 cycles a solve with 1,500
// systems of 32 species on the GPU, now 30,300; 14,000 and 11,800 with 1,000 of 16).
//
// What bounds it: the chain of N pivot steps (hand-over through shared memory,
// one division, the first update).  1,000 systems of 16 species (160 reactions,
// dt = 1e-3, atol = rtol = 5e-3): 219.4 ms with the full-width row form (2N
// divisions by one lane per step), 16.4 ms by columns, 12.8 ms now.
//
// One loop turn is one substep of every team of the warp, whatever part of its
// attempt the team is in, so teams never wait for each other's attempts or
// systems.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "networks.cuh"
#include "reaction_words.cuh"

namespace wind {

constexpr int TEAM_MAXN = 32;

struct TeamLayout {
    // byte offsets inside one team's shared slice: the Jacobian at the
    // accepted state, the Jacobian of the second half step / the columns handed
    // over by the elimination (SIE only), vectors (the state followed by a zero),
    // the dense term, signed rates, unit lists and (SIE) Jacobian terms
    int jy, w, vec, lt, rates, inc_off, inc, term_off, term, bytes;
    __host__ __device__ static int align16(int x) { return (x + 15) & ~15; }
    __host__ __device__ TeamLayout(int nmax, int R, bool lin, bool matrices) {
        const int mat = matrices ? nmax * nmax * 8 : 0;
        int off = 0;
        jy = off; off = align16(off + mat);
        w = off; off = align16(off + mat + (matrices ? 2 * nmax * 8 : 0));  // and two exchange rows
        vec = off; off = align16(off + (2 * nmax + 2) * 8);
        lt = off; off = align16(off + (lin ? nmax * nmax * 4 : 0));
        rates = off; off = align16(off + (2 * R + 1) * 8);
        inc_off = off; off = align16(off + (nmax + 1) * 4);
        inc = off; off = align16(off + (4 * R + 3 * nmax + 4) * 4);     // and the word read ahead
        term_off = off; off = align16(off + (matrices ? (nmax + 1) * 4 : 0));
        term = off; off = align16(off + (matrices ? (8 * R + 3 * nmax + 4) * 4 : 0));
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
    const double* rates;      // [2R + 1]: -k, k of each reaction, 0
    const int* inc_off;       // [NMAX+1] CSR offsets
    const uint32_t* inc;      // unit list: one word per -w or +w of f_l
    const int* term_off;
    const uint32_t* term;     // one word per unit of a Jacobian entry, by column
};

// f_l and, with JAC, column l of Jt into J, for the current v.  The contract's
// updates are the units x - d and x + d, that is x + (-d) and x + d: the lists
// hold one word per unit with the signed rate, f's in reaction order, the
// Jacobian's by entry (each entry's units in the order of the contract, from the
// dense term on), so an entry is summed in a register and stored without being
// read back.  Padded to four words that add zero; the next four are in flight.
// (Scanning a list of reactions and updating entries in place took 400 cycles a
// reaction.)
template <int NMAX, bool JAC>
__device__ __forceinline__ void team_rhs_jac(const TeamCtx<NMAX>& c, double* J) {
    const int l = c.l;
    if (l < c.N) {
        xd acc = 0.0;
        if (c.LT)
            for (int k = 0; k < c.N; k++) acc += xd((double)c.LT[k * NMAX + l]) * xd(c.v[k]);
        {
            const int e1 = c.inc_off[l + 1];
            int e = c.inc_off[l];
            uint4 next = *reinterpret_cast<const uint4*>(c.inc + e);
            for (; e < e1; e += 4) {
                const uint32_t q[4] = {next.x, next.y, next.z, next.w};
                next = *reinterpret_cast<const uint4*>(c.inc + e + 4);
                xd w[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    w[u] = xd(rx_rate(c.rates, q[u])) * xd(rx_at(c.v, rx_first(q[u]))) *
                           xd(rx_at(c.v, rx_second(q[u])));
#pragma unroll
                for (int u = 0; u < 4; u++) acc += w[u];
            }
        }
        c.f[l] = acc.v;
        if (JAC) {
            for (int i = 0; i < c.N; i++) J[i * NMAX + l] = c.LT ? (double)c.LT[i * NMAX + l] : 0.0;
            const int e1 = c.term_off[l + 1];
            int e = c.term_off[l];
            uint4 next = *reinterpret_cast<const uint4*>(c.term + e);
            xd sum = 0.0;
            for (; e < e1; e += 4) {
                const uint32_t q[4] = {next.x, next.y, next.z, next.w};
                next = *reinterpret_cast<const uint4*>(c.term + e + 4);
                xd d[4];
                double start[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    d[u] = xd(rx_rate(c.rates, q[u])) * xd(rx_at(c.v, rx_first(q[u])));
                    // (padding's column is NMAX: no dense entry)
                    start[u] = 0.0;
                    if (c.LT && rx_second(q[u]) < 8u * NMAX)
                        start[u] = (double)c.LT[(rx_second(q[u]) >> 3) * NMAX + l];
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    // an entry's partial sums are stored over until its last unit
                    sum = ((q[u] & RX_MARK) ? xd(start[u]) : sum) + d[u];
                    J[(rx_second(q[u]) >> 3) * NMAX + l] = sum.v;
                }
            }
        }
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
                                                const int* inc_off, const uint32_t* inc, const int* term_off,
                                                const uint32_t* term, double h) {
    TeamCtx<NMAX> c;
    c.mask = mask; c.l = l; c.leader = leader; c.N = N;
    c.jy = jy; c.w = w; c.v = v; c.f = f;
    c.LT = LT; c.rates = rates; c.inc_off = inc_off; c.inc = inc;
    c.term_off = term_off; c.term = term;
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

// Steps [i0, i1) of the downward pass: x[k] holds row i + k of the lane's column,
// W rows from the pivot row on.  The pivot lane hands over its column (row i in
// F[0]), every lane divides its row-i entry, keeps it in X[i] and updates the rows
// below, which move up one register: the loop is one step's code, however many
// steps there are.
template <int W, int NMAX>
__device__ __forceinline__ bool team_gje_down(const TeamCtx<NMAX>& c, xd (&x)[NMAX], int i0, int i1) {
    const int l = c.l;
    double* X = c.w;
    bool ok = true;
#pragma unroll 1
    for (int i = i0; i < i1; i++) {
        double* F = c.w + NMAX * NMAX + (i & 1) * NMAX;
        if (l == i) {
#pragma unroll
            for (int t = 0; t < W; t += 2) *reinterpret_cast<double2*>(F + t) = make_double2(x[t].v, x[t + 1].v);
#pragma unroll
            for (int t = 0; t < W; t++) x[t] = (t == 0) ? 1.0 : 0.0;  // column i of Inv starts
        }
        team_sync(c.mask);
        const double2 f01 = *reinterpret_cast<const double2*>(F);
        const xd s = f01.x;
        ok = ok && s.v != 0.0 && finite64(s.v);
        const xd xi = x[0] / s;
        X[i * NMAX + l] = xi.v;
        x[0] = x[1] - xd(f01.y) * xi;
#pragma unroll
        for (int k = 2; k < W; k += 2) {
            const double2 f = *reinterpret_cast<const double2*>(F + k);
            x[k - 1] = x[k] - xd(f.x) * xi;
            x[k] = x[k + 1] - xd(f.y) * xi;
        }
        x[W - 1] = 0.0;
    }
    return ok;
}

// Steps b1 >= b > b0 of the upward pass: x[k] holds row b - k of the lane's
// column of Inv.  Row b is final and goes to X[b]; M's entries above the pivot
// stand in column b of X.  (Rows below zero read what precedes X and are not used.)
template <int W, int NMAX>
__device__ __forceinline__ void team_gje_up(const TeamCtx<NMAX>& c, xd (&x)[NMAX], int b1, int b0) {
    const int l = c.l;
    double* X = c.w;
#pragma unroll 1
    for (int b = b1; b > b0; b--) {
        const double* col = X + b * NMAX + b;
        const xd xb = x[0];
#pragma unroll
        for (int k = 1; k < W; k++) x[k - 1] = x[k] - xd(col[-k * NMAX]) * xb;
        x[W - 1] = 0.0;
        team_sync(c.mask);  // column entries of row b are read before the row is replaced
        X[b * NMAX + l] = xb.v;
    }
}

// One SIE substep of size h from the state in v with f in f and Jt in J (jy
// or w); returns the stepped component l.  Column form of the file comment.
// `clean` is cleared when the full-width elimination had to be used, which
// overwrites jy.
template <int NMAX, int CTRL>
__device__ __forceinline__ double team_gje_step(const TeamCtx<NMAX>& c, const double* J, double h, bool& clean) {
    constexpr int H = NMAX > 8 ? NMAX / 2 : NMAX;  // rows of the second half's steps
    const int l = c.l, N = c.N;
    double* X = c.w;  // rows as they leave the downward pass, then Inv
    xd x[NMAX];
#pragma unroll
    for (int t = 0; t < NMAX; t++)
        x[t] = team_matrix_elem<CTRL>((l < N && t < N) ? J[t * NMAX + l] : 0.0, h, t == l);
    team_sync(c.mask);  // J may be w: every column is in registers before the first is handed over
    const int mid = min(N, NMAX - H);
    bool ok = team_gje_down<NMAX>(c, x, 0, mid);
    if (N > NMAX - H) ok = team_gje_down<H>(c, x, mid, N) && ok;
    team_sync(c.mask);
#pragma unroll
    for (int t = 0; t < NMAX; t++) {
        const int row = N - 1 - t;
        x[t] = (row >= 0 && l <= row) ? X[row * NMAX + l] : 0.0;
    }
    team_sync(c.mask);
    if (N > H) team_gje_up<NMAX>(c, x, N - 1, H - 1);
    team_gje_up<H>(c, x, min(N, H) - 1, 0);
    X[l] = x[0].v;
    double out = 0.0;
    if (l < N) {
        TeamProduct<CTRL> prod(c.v[l], h);
        for (int k = 0; k < N; k++) prod.add(X[k * NMAX + l], c.f[k]);
        out = prod.result(c.v[l]);
        ok = ok && finite64(out);
    }
    if (!__all_sync(c.mask, ok)) {
        out = team_gje_general<NMAX, CTRL>(c.mask, l, c.leader, N, c.jy, c.w, c.v, c.f, c.LT, c.rates,
                                           c.inc_off, c.inc, c.term_off, c.term, h);
        clean = false;
    }
    return out;
}

// Stage a system (rates `k`, reactions `sp`, dense term `Lg` or null) into its
// team's slice: signed rates, the dense term transposed, the unit lists and, with
// JAC, the Jacobian terms.  A species index >= N marks it BAD_INPUT (returned) and
// nothing of it is read again.
template <int NMAX, bool JAC>
__device__ __forceinline__ bool team_stage(unsigned mask, int l, int N, int R, const double* k_in, const uint2* sp,
                                           const float* Lg, unsigned char* base) {
    const TeamLayout lay(NMAX, R, Lg != nullptr, JAC);
    double* rates = reinterpret_cast<double*>(base + lay.rates);
    int* inc_off = reinterpret_cast<int*>(base + lay.inc_off);
    uint32_t* inc = reinterpret_cast<uint32_t*>(base + lay.inc);
    int* term_off = reinterpret_cast<int*>(base + lay.term_off);
    uint32_t* term = reinterpret_cast<uint32_t*>(base + lay.term);
    float* LT = reinterpret_cast<float*>(base + lay.lt);
    double* v = reinterpret_cast<double*>(base + lay.vec);
    // `at` (in w, which no system uses yet), one row per species: the terms of each
    // column, counted, then where the column's next one goes
    constexpr int LDA = 2 * NMAX + 1;
    int* counts = reinterpret_cast<int*>(base + lay.w);
    int* at = counts + (l < N ? l : 0) * LDA;
    if (l < N) {
        inc_off[l + 1] = 0;  // units of species l, counted here
        if (JAC) {
#pragma unroll 1
            for (int col = 0; col < N; col++) at[col] = 0;
        }
    }
    team_sync(mask);
    bool bad = false;
    for (int r = l; r < R; r += NMAX) {
        const double k = __ldg(k_in + r);
        rates[2 * r] = -k;
        rates[2 * r + 1] = k;
        const uint2 q = __ldg(sp + r);
        const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
        if (max(max(a, b), max(cc, d)) >= N) {
            bad = true;
        } else {
            auto count = [&](int j) {
                atomicAdd(inc_off + 1 + j, 1);
                if (JAC) {
                    atomicAdd(counts + j * LDA + a, 1);
                    atomicAdd(counts + j * LDA + b, 1);
                }
            };
            count(a);
            count(b);
            count(cc);
            count(d);
        }
    }
    team_sync(mask);
    if (__any_sync(mask, bad)) return true;
    // units of species l in reaction (a, b -> cc, d): nn times -, then np times +;
    // two terms each
    const int units = l < N ? inc_off[l + 1] : 0;
    const int room = (units + 3) & ~3, term_room = JAC ? (2 * units + 3) & ~3 : 0;
    const int inc_end = rx_scan<NMAX>(mask, l, room), term_end = rx_scan<NMAX>(mask, l, term_room);
    if (l < N) {
        inc_off[l + 1] = inc_end;
        if (JAC) term_off[l + 1] = term_end;
    }
    if (l == 0) {
        inc_off[0] = 0;
        if (JAC) term_off[0] = 0;
        rates[2 * R] = 0.0;
        v[NMAX] = 0.0;
    }
    team_sync(mask);
    uint32_t* mine = inc + inc_end - room;
    int e = rx_list<NMAX>(mask, l, N, R, sp, reinterpret_cast<uint32_t*>(v + NMAX + 2), mine);
    if (l < N) {
        int t = term_end - term_room;
        if (JAC) {
#pragma unroll 1
            for (int col = 0; col < N; col++) {
                t += at[col];
                at[col] = t;  // where the column ends
            }
        }
        // reactions to units and terms, from the end of the list (which only grows)
        uint2 next = e ? __ldg(sp + mine[e - 1]) : make_uint2(0u, 0u);
#pragma unroll 1
        for (int o = units; e > 0;) {
            const uint2 q = next;
            const int r = (int)mine[--e];
            if (e) next = __ldg(sp + mine[e - 1]);
            const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
            const int nn = (a == l) + (b == l), n = nn + (cc == l) + (d == l);
            o -= n;
            // d w / d y_a = k y_b, then d w / d y_b = k y_a: per reaction all
            // units of the first before the second
            int ta = 0, tb = 0;
            if (JAC) {
                ta = at[a] - n;
                tb = (a == b ? ta : at[b]) - n;
                at[a] = ta;
                at[b] = tb;
                if (a == b) {
                    const int first = tb;
                    tb = ta;
                    ta = first;
                }
            }
            for (int u = 0; u < n; u++) {
                const int slot = 2 * r + (u >= nn);
                mine[o + u] = rx_pack(slot, a, b);
                if (JAC) {
                    term[ta + u] = rx_pack(slot, b, a);
                    term[tb + u] = rx_pack(slot, a, b);
                }
            }
        }
        if (JAC) {
            // (`at` is where the columns begin now)
            for (int col = 0; col < N; col++) {
                const int end = col + 1 < N ? at[col + 1] : t;
                if (end > at[col]) term[at[col]] |= RX_MARK;
            }
            while (t < term_end) term[t++] = rx_pack(2 * R, NMAX, NMAX) | RX_MARK;
        }
        for (e = units; e < room; e++) mine[e] = rx_pack(2 * R, NMAX, NMAX);
        if (Lg) {
            for (int k = 0; k < N; k++) LT[k * NMAX + l] = Lg[l * N + k];
        }
    }
    team_sync(mask);
    return false;
}

// The same with every lane looking through all reactions and walking its list once
// per column, for k_mixed on networks of few reactions (mixed_counted): system s's
// signed rates, the dense term transposed, the unit lists and, with JAC, the
// Jacobian terms.  A species index >= N marks the system BAD_INPUT
// (returned) and nothing of it is read again.
template <int NMAX, bool JAC>
__device__ __forceinline__ bool team_stage_scan(const TeamCtx<NMAX>& c, const KParams& p, int64_t s, double* rates,
                                                int* inc_off, uint32_t* inc, int* term_off, uint32_t* term, float* LT) {
    const int N = c.N, R = p.n_react, l = c.l;
    const uint2* sp = reinterpret_cast<const uint2*>(p.species) + s * R;
    bool bad = false;
    for (int r = l; r < R; r += NMAX) {
        const double k = p.rates[s * R + r];
        rates[2 * r] = -k;
        rates[2 * r + 1] = k;
        const uint2 q = __ldg(sp + r);
        const unsigned nn = (unsigned)N;
        bad = bad || (q.x & 0xffffu) >= nn || (q.x >> 16) >= nn || (q.y & 0xffffu) >= nn || (q.y >> 16) >= nn;
    }
    if (__any_sync(c.mask, bad)) return true;
    // units of species l in reaction (a, b -> cc, d): nn times -, then np times +
    if (l < N) {
        int cnt = 0;
        for (int r = 0; r < R; r++) {
            const uint2 q = __ldg(sp + r);
            const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
            cnt += (a == l) + (b == l) + (cc == l) + (d == l);
        }
        inc_off[l + 1] = (cnt + 3) & ~3;
        if (JAC) term_off[l + 1] = (2 * cnt + 3) & ~3;
    }
    team_sync(c.mask);
    if (l == 0) {
        inc_off[0] = 0;
        for (int j = 0; j < N; j++) inc_off[j + 1] += inc_off[j];
        if (JAC) {
            term_off[0] = 0;
            for (int j = 0; j < N; j++) term_off[j + 1] += term_off[j];
        }
        rates[2 * R] = 0.0;
        c.v[NMAX] = 0.0;
    }
    team_sync(c.mask);
    if (l < N) {
        int o = inc_off[l];
        for (int r = 0; r < R; r++) {
            const uint2 q = __ldg(sp + r);
            const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
            const int nn = (a == l) + (b == l), np = (cc == l) + (d == l);
            for (int u = 0; u < nn + np; u++) inc[o++] = rx_pack(2 * r + (u >= nn), a, b);
        }
        if (JAC) {
            // d w / d y_a = k y_b, then d w / d y_b = k y_a: per reaction all
            // units of the first before the second
            int t = term_off[l];
            for (int col = 0; col < N; col++) {
                const int t0 = t;
                for (int e = inc_off[l]; e < o;) {
                    const uint32_t q = inc[e];
                    const int r = (int)(q & 0x7ffffu) >> 4, a = (int)(rx_first(q) >> 3), b = (int)(rx_second(q) >> 3);
                    int n = e + 1;  // the reaction's units are neighbours
                    while (n < o && ((int)(inc[n] & 0x7ffffu) >> 4) == r) n++;
                    if (a == col)
                        for (int u = e; u < n; u++) term[t++] = rx_pack((int)(inc[u] & 0x7ffffu) >> 3, b, col);
                    if (b == col)
                        for (int u = e; u < n; u++) term[t++] = rx_pack((int)(inc[u] & 0x7ffffu) >> 3, a, col);
                    e = n;
                }
                if (t > t0) term[t0] |= RX_MARK;
            }
            while (t < term_off[l + 1]) term[t++] = rx_pack(2 * R, NMAX, NMAX) | RX_MARK;
        }
        while (o < inc_off[l + 1]) inc[o++] = rx_pack(2 * R, NMAX, NMAX);
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
template <int NMAX, int METHOD, int CTRL, bool COUNTED>
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
    c.f = c.v + NMAX + 2;
    float* LT = lin ? reinterpret_cast<float*>(base + lay.lt) : nullptr;
    double* rates = reinterpret_cast<double*>(base + lay.rates);
    int* inc_off = reinterpret_cast<int*>(base + lay.inc_off);
    uint32_t* inc = reinterpret_cast<uint32_t*>(base + lay.inc);
    c.LT = LT;
    c.rates = rates;
    c.inc_off = inc_off;
    c.inc = inc;
    int* term_off = reinterpret_cast<int*>(base + lay.term_off);
    uint32_t* term = reinterpret_cast<uint32_t*>(base + lay.term);
    c.term_off = term_off;
    c.term = term;
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
                if constexpr (COUNTED)
                    stop = team_stage<NMAX, SIE>(c.mask, l, N, p.n_react, p.rates + s * p.n_react,
                                                 reinterpret_cast<const uint2*>(p.species) + s * p.n_react,
                                                 lin ? p.linear + s * (int64_t)N * N : nullptr, base);
                else
                    stop = team_stage_scan<NMAX, SIE>(c, p, s, rates, inc_off, inc, term_off, term, LT);
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
    team_run<NMAX, METHOD, CTRL, true>(p, smem_raw, tpw, tpw);
}

}  // namespace wind
