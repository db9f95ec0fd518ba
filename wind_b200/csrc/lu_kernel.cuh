// lu_kernel.cuh -- persistent team-per-system SIE with the FP64 LU for runtime
// mass-action networks with N <= 32 (optionally with a dense linear term).
//
// A team is L lanes of one warp; lane l owns equation l of a system: its matrix
// row in registers (COLS >= N elements, indexed only by compile-time
// constants), its components of the state, of the candidates and of the
// right-hand side.  What another lane must read -- the state, the pivot row of
// an elimination step -- goes through shared memory.
//
// The teams of a warp run in lockstep: one loop turn is one substep of every
// team, whatever part of its attempt the team is in, and every barrier,
// reduction and shuffle inside it is warp-wide (with differing partial masks a
// reduction takes 170 cycles instead of 22 per team, measured).  Teams never
// wait for each other's attempts or systems.  An attempt after a refinement
// takes the refined attempt's first half step as its full step when the two
// sizes are the same number: the state, Jacobian and size are, so the bits are
// (t + h rounds differently in about half of the cases, and then it is
// computed).
//
// Elimination step k: the pivot is the largest |a_ik| of the rows not chosen
// yet (warp maximum over packed |a|/row keys), rows never move, the pivot row
// and its reciprocal are published, every other row takes one multiplier and
// COLS - k - 1 fused multiply-adds.  The next column's key and reciprocal are
// formed before the rest of the row is updated, so the reduction and the
// reciprocal run under the updates.  A chosen row's multiplier is zero instead
// of its update being branched around: the solve is straight-line code, and a
// solution that is not finite (a zero times an infinite pivot row) is computed
// again with the updates selected.
//
// Right-hand side and Jacobian: the species' incidences (reaction ids
// ascending) and, for the Jacobian, their terms sorted by column, so a row
// entry is summed in a register, in the order of the unsorted list, and
// stored without being read back.  Lists are padded to whole 16-byte words of
// four with entries that add zero.  (With many reactions the terms cost resident
// teams, and a launch may leave them out: lu_jac_row_in_place.)
//
// The dense term is widened to FP64 when a system is staged: a substep reads
// each entry twice, and a conversion takes 12 to 24 cycles of a unit that the
// pivot keys and reciprocals need too.  3,000 dense systems of 32 species and
// 64 reactions: 704 to 637 ms (893 before this kernel).  The 4 KB a team that this
// costs take teams away where there are many reactions, and the gain is smaller
// there: at looser tolerances 68.3 to 62.0 ms with 64 reactions, 79.6 to 76.0 ms
// with 160, 92.7 to 91.3 ms with 240.
//
// The values are those of the one-row-per-lane kernel this replaced, bit for
// bit: the same pivots, multipliers and order of every sum.
#pragma once

#include "common.cuh"
#include "reaction_words.cuh"
#include "solvers_reg.cuh"
#include "warp_kernel.cuh"

namespace wind {

// Signed rates s * k of a system (s the net stoichiometry of one species, 0,
// +-1 or +-2; exact): a reaction takes its reactants by one s and makes its
// products by another, so two entries per reaction hold them all, and two more
// serve s = 0 and padding.
struct LuLayout {
    // byte offsets inside one team's slice
    int rates, inc_off, inc, term_off, term, lt, vb, rows, rows2, pb, bytes;
    __host__ __device__ static int align16(int x) { return (x + 15) & ~15; }
    __host__ __device__ LuLayout(int cols, int n, int R, bool lin, bool sorted) {
        int off = 0;
        rates = off; off = align16(off + (2 * R + 2) * 8);       // signed rates
        inc_off = off; off = align16(off + (n + 1) * 4);
        inc = off; off = align16(off + (4 * R + 3 * n + 4) * 4);  // and the word read ahead
        term_off = off; off = align16(off + (sorted ? (n + 1) * 4 : 0));
        term = off; off = align16(off + (sorted ? (8 * R + 3 * n + 4) * 4 : 0));
        lt = off; off = align16(off + (lin ? n * n * 8 : 0));     // dense term, widened once
        vb = off; off = align16(off + (cols + 1) * 8);           // state, and a zero
        // Jacobian rows: at the accepted state, and at the half step -- of up
        // to 16 species a second set is small beside the lists, and keeps the
        // first over an attempt's refinements
        rows = off; off = align16(off + n * (cols + 2) * 8);
        rows2 = cols <= 16 ? off : rows;
        off = rows2 + align16(n * (cols + 2) * 8);
        pb = off; off = align16(off + 2 * (cols + 2) * 8);       // pivot-row buffers
        bytes = off;
    }
};

template <int L, int COLS>
struct LuCtx {
    static constexpr int LDR = COLS + 2;  // row pitch: an odd number of 16-byte chunks
    unsigned mask;     // lanes of the team
    int l, leader, N;
    int tm;            // the lane's team in its warp
    bool live;         // the team has a system
    const double* rates;
    const int* inc_off;
    const uint32_t* inc;
    const int* term_off;
    const uint32_t* term;  // null: the Jacobian is summed in place
    const double* LT;  // LT[k*N + r] = L[r][k], or null
    double* vb;
    double* rows;      // Jacobian rows in use
    double* pb;
};

// sum_k L[r][k] w[k] for the dense term (w in shared memory, FP64), four
// independent accumulators over a compile-time column loop.
template <int COLS>
__device__ __forceinline__ double lu_dense_dot(const double* LT, const double* w, int r, int N) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
    for (int k = 0; k < COLS; k += 4) {
        if (k < N) {
            const double2 w01 = *reinterpret_cast<const double2*>(w + k);
            s0 = fma(LT[k * N + r], w01.x, s0);
            if (k + 1 < N) s1 = fma(LT[(k + 1) * N + r], w01.y, s1);
            if (k + 2 < N) s2 = fma(LT[(k + 2) * N + r], w[k + 2], s2);
            if (k + 3 < N) s3 = fma(LT[(k + 3) * N + r], w[k + 3], s3);
        }
    }
    return (s0 + s1) + (s2 + s3);
}

// f of row r at the state in vb: dense term L v plus the incident reactions,
// even and odd incidences summed apart.
template <class Ctx, int COLS>
__device__ __forceinline__ double lu_rhs(const Ctx& c, int r) {
    double acc = 0.0, acc2 = 0.0;
    if (c.LT) acc = lu_dense_dot<COLS>(c.LT, c.vb, r, c.N);
    const int e1 = c.inc_off[r + 1];
    int e = c.inc_off[r];
    uint4 next = *reinterpret_cast<const uint4*>(c.inc + e);
    for (; e < e1; e += 4) {
        const uint32_t q[4] = {next.x, next.y, next.z, next.w};
        next = *reinterpret_cast<const uint4*>(c.inc + e + 4);
        double g[4], vb[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            g[u] = __dmul_rn(rx_rate(c.rates, q[u]), rx_at(c.vb, rx_first(q[u])));
            vb[u] = rx_at(c.vb, rx_second(q[u]));
        }
        acc = fma(g[0], vb[0], acc);
        acc2 = fma(g[1], vb[1], acc2);
        acc = fma(g[2], vb[2], acc);
        acc2 = fma(g[3], vb[3], acc2);
    }
    return acc + acc2;
}

// Mass-action Jacobian row r at the state in vb into its row of c.rows.
template <class Ctx, int COLS>
__device__ __forceinline__ void lu_jac_row(const Ctx& c, int r) {
    double* row = c.rows + r * Ctx::LDR;
#pragma unroll
    for (int t = 0; t < COLS; t += 2) *reinterpret_cast<double2*>(row + t) = make_double2(0.0, 0.0);
    double acc = 0.0;
    const int e1 = c.term_off[r + 1];
    int e = c.term_off[r];
    uint4 next = *reinterpret_cast<const uint4*>(c.term + e);
    for (; e < e1; e += 4) {
        const uint32_t q[4] = {next.x, next.y, next.z, next.w};
        next = *reinterpret_cast<const uint4*>(c.term + e + 4);
        double ks[4], v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            ks[u] = rx_rate(c.rates, q[u]);
            v[u] = rx_at(c.vb, rx_first(q[u]));
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            // an entry's partial sums are stored over until its last term
            acc = fma(ks[u], v[u], acc);
            *reinterpret_cast<double*>(reinterpret_cast<char*>(row) + rx_second(q[u])) = acc;
            acc = (q[u] & RX_MARK) ? 0.0 : acc;
        }
    }
}

// The same without the term list, which is half of what a reaction takes: an
// entry's terms are added where they stand, in the same order (70 to 100 cycles a
// term against 20 to 25 from the list).
template <int COLS>
__device__ __noinline__ void lu_jac_row_in_place(const double* rates, const uint32_t* inc, int cnt, const double* vb,
                                                 double* row, uint32_t last) {
#pragma unroll
    for (int t = 0; t < COLS; t += 2) *reinterpret_cast<double2*>(row + t) = make_double2(0.0, 0.0);
#pragma unroll 2
    for (int e = 0; e < cnt; e++) {
        const uint32_t q = inc[e];
        // (padding and s = 0, from `last` on, go to the column beside the row)
        const bool in = (q & 0x7ffffu) < last;
        const uint32_t a = in ? rx_first(q) : 8u * COLS, b = in ? rx_second(q) : 8u * COLS;
        const double ks = rx_rate(rates, q), va = rx_at(vb, a), vc = rx_at(vb, b);
        double* pa = reinterpret_cast<double*>(reinterpret_cast<char*>(row) + a);
        *pa = fma(ks, vc, *pa);
        double* pb = reinterpret_cast<double*>(reinterpret_cast<char*>(row) + b);
        *pb = fma(ks, va, *pb);
    }
}

// a[] = row r of I - h J, from the dense term and the Jacobian row.
template <class Ctx, int COLS>
__device__ __forceinline__ void lu_load_row(const Ctx& c, int r, double h, double (&a)[COLS]) {
    if (r >= c.N) {
#pragma unroll
        for (int t = 0; t < COLS; t++) a[t] = 0.0;
        return;
    }
    const double* row = c.rows + r * Ctx::LDR;
#pragma unroll
    for (int t0 = 0; t0 < COLS; t0 += 2) {
        const double2 w = *reinterpret_cast<const double2*>(row + t0);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int t = t0 + q;
            double j = q ? w.y : w.x;
            if (c.LT && t < c.N) j += c.LT[t * c.N + r];
            a[t] = (t == r) ? fma(-h, j, 1.0) : -h * j;
        }
    }
}

// Maximum of `key` over each team: one warp-wide reduction per team.
template <int L>
__device__ __forceinline__ unsigned lu_team_max(int tm, unsigned key) {
    if constexpr (L == 32) return __reduce_max_sync(0xffffffffu, key);
    unsigned best = 0u;
#pragma unroll
    for (int t = 0; t < 32 / L; t++) {
        const unsigned r = __reduce_max_sync(0xffffffffu, tm == t ? key : 0u);
        if (tm == t) best = r;
    }
    return best;
}

// Predicated 16-byte shared-memory stores of one to four pairs (no branch
// around them, one predicate for the group).
__device__ __forceinline__ void lu_put2(bool on, double* p, double x, double y) {
    asm volatile("{ .reg .pred p; setp.ne.s32 p, %0, 0; @p st.shared.v2.f64 [%1], {%2, %3}; }" ::"r"((int)on),
                 "r"((unsigned)__cvta_generic_to_shared(p)), "d"(x), "d"(y)
                 : "memory");
}
__device__ __forceinline__ void lu_put4(bool on, double* p, const double* a) {
    asm volatile(
        "{ .reg .pred p; setp.ne.s32 p, %0, 0; @p st.shared.v2.f64 [%1], {%2, %3}; @p st.shared.v2.f64 [%1+16], "
        "{%4, %5}; }" ::"r"((int)on),
        "r"((unsigned)__cvta_generic_to_shared(p)), "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3])
        : "memory");
}
__device__ __forceinline__ void lu_put8(bool on, double* p, const double* a) {
    asm volatile(
        "{ .reg .pred p; setp.ne.s32 p, %0, 0; @p st.shared.v2.f64 [%1], {%2, %3}; @p st.shared.v2.f64 [%1+16], "
        "{%4, %5}; @p st.shared.v2.f64 [%1+32], {%6, %7}; @p st.shared.v2.f64 [%1+48], {%8, %9}; }" ::"r"((int)on),
        "r"((unsigned)__cvta_generic_to_shared(p)), "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]),
        "d"(a[6]), "d"(a[7])
        : "memory");
}
// Elements [t0, COLS) of a row, t0 even.
template <int COLS>
__device__ __forceinline__ void lu_put_row(bool on, double* buf, const double (&a)[COLS], int t0) {
    if (t0 & 2) lu_put2(on, buf + t0, a[t0], a[t0 + 1]);
    const int t1 = (t0 + 3) & ~3;
    if ((COLS - t1) & 4) lu_put4(on, buf + t1, a + t1);
#pragma unroll
    for (int t = t1 + ((COLS - t1) & 4); t < COLS; t += 8) lu_put8(on, buf + t, a + t);
}

// State of a factorisation beside the rows.
struct LuPivots {
    int step;            // pivot step of the row, 64: none yet, -1: no row
    double rcp;          // 1 / U_kk of the row's pivot step
    uint32_t rows[6];    // pivot row of each step, 5 bits each, 6 to a word
    unsigned best;       // the next step's packed maximum
    double myrcp;        // reciprocal of this lane's entry in the next column
};

// Elimination steps [K0, K1) (a loop of its own per range: the compiler unrolls
// only so much at once).  GUARD: N may be any number up to COLS; otherwise it
// is above COLS - 4.  EXACT: updates of chosen rows selected away instead of
// multiplied by zero.
template <int K0, int K1, bool GUARD, bool EXACT, int L, int COLS>
__device__ __forceinline__ void lu_steps(const LuCtx<L, COLS>& c, double (&a)[COLS], double& b, LuPivots& pv) {
    const int l = c.l, N = c.N;
#pragma unroll
    for (int k = K0; k < K1; k++) {
        if ((!GUARD && k <= COLS - 4) || k < N) {
            const int p = 31 - (int)(pv.best & 31u);
            double* buf = c.pb + (k & 1) * (COLS + 2);
            const bool mine = c.live && p == l;
            lu_put_row(mine, buf, a, (k + 1) & ~1);
            lu_put2(mine, buf + COLS, b, pv.myrcp);
            pv.rcp = mine ? pv.myrcp : pv.rcp;
            pv.step = mine ? k : pv.step;
            pv.rows[k / 6] = (k % 6 ? pv.rows[k / 6] : 0u) | ((uint32_t)p << (5 * (k % 6)));
            __syncwarp();
            if (k + 1 < COLS) {
                const double2 br = *reinterpret_cast<const double2*>(buf + COLS);
                const bool act = pv.step == 64;
                const double m = act ? a[k] * br.y : 0.0;
                // the next column first: its key and reciprocal
                const double n = fma(-m, buf[k + 1], a[k + 1]);
                a[k + 1] = (!EXACT || act) ? n : a[k + 1];
                pv.best = lu_team_max<L>(c.tm, pivot_key(a[k + 1], l, act));
                pv.myrcp = nr_rcp(a[k + 1]);
                asm volatile("" : "+d"(pv.myrcp));  // here, under the updates, not after them
#pragma unroll
                for (int t = (k + 2) & ~1; t < COLS; t += 2) {
                    const double2 w = *reinterpret_cast<const double2*>(buf + t);
                    if (t > k + 1) {
                        const double u = fma(-m, w.x, a[t]);
                        a[t] = (!EXACT || act) ? u : a[t];
                    }
                    const double u = fma(-m, w.y, a[t + 1]);
                    a[t + 1] = (!EXACT || act) ? u : a[t + 1];
                }
                const double u = fma(-m, br.x, b);
                b = (!EXACT || act) ? u : b;
            }
        }
    }
}

// Factor the rows in a[] with partial pivoting and solve for the right-hand
// side b (this lane's component); returns x_l.
template <bool GUARD, bool EXACT, int L, int COLS>
__device__ __forceinline__ double lu_solve(const LuCtx<L, COLS>& c, double (&a)[COLS], double b) {
    const int l = c.l, N = c.N;
    LuPivots pv;
    pv.step = (l < N) ? 64 : -1;
    pv.rcp = 0.0;
    pv.best = lu_team_max<L>(c.tm, pivot_key(a[0], l, pv.step == 64));
    pv.myrcp = nr_rcp(a[0]);
    lu_steps<0, (COLS < 8 ? COLS : 8), GUARD, EXACT>(c, a, b, pv);
    if constexpr (COLS > 8) lu_steps<8, (COLS < 16 ? COLS : 16), GUARD, EXACT>(c, a, b, pv);
    if constexpr (COLS > 16) lu_steps<16, (COLS < 24 ? COLS : 24), GUARD, EXACT>(c, a, b, pv);
    if constexpr (COLS > 24) lu_steps<24, COLS, GUARD, EXACT>(c, a, b, pv);
    __syncwarp();  // the last pivot row is read before the next solve publishes
    // back substitution by columns: x_i from the lane that pivoted at step i
#pragma unroll
    for (int i = COLS - 1; i > 0; i--) {
        if ((!GUARD && i <= COLS - 4) || i < N) {
            const int p = (pv.rows[i / 6] >> (5 * (i % 6))) & 31;
            const double xi = __shfl_sync(0xffffffffu, b * pv.rcp, c.leader + (p & (L - 1)));
            const double u = fma(-a[i], xi, b);
            b = (pv.step >= 0 && pv.step < i) ? u : b;
        }
    }
    // component l is the pivot row's of step l
    uint32_t w = pv.rows[0];
#pragma unroll
    for (int q = 1; q < (COLS + 5) / 6; q++) w = (l >= 6 * q) ? pv.rows[q] : w;
    const int p = (int)(w >> (5 * (l % 6)));
    const double x = __shfl_sync(0xffffffffu, b * pv.rcp, c.leader + (p & (L - 1)));
    return l < N ? x : 0.0;
}

// The solve with selected updates, for solutions that are not finite.
template <bool GUARD, int L, int COLS>
__device__ __noinline__ double lu_solve_exact(int l, int leader, int N, int tm, bool live, const double* LT,
                                              double* rows, double* pb, double h, double f) {
    LuCtx<L, COLS> c;
    c.l = l; c.leader = leader; c.N = N; c.tm = tm; c.live = live;
    c.LT = LT; c.rows = rows; c.pb = pb;
    double a[COLS];
    lu_load_row<LuCtx<L, COLS>, COLS>(c, l, h, a);
    return lu_solve<GUARD, true>(c, a, f);
}

// Stage a system (rates `k_in`, reactions `sp`, dense term `Lg` or null) into its
// team's slice: signed rates, the dense term transposed, the incidence lists and,
// if `sorted`, the Jacobian terms.  A species index >= N marks it BAD_INPUT
// (returned) and nothing of it is read again.  U: reactions in flight in a lane.
//
// What has no order (counts, rates) is done with a reaction per lane; a lane then
// walks the list of its species once.  With a walk per column, behind two looks of
// every lane at every reaction, one attempt of 4,000 systems of 32 species took
// 5.3 ms with 1,000 reactions and 0.96 ms with 320; now 1.0 and 0.32 ms.
template <int L, int COLS, int U>
__device__ __forceinline__ bool lu_stage(unsigned mask, int l, int N, int R, const double* k_in, const uint2* sp,
                                         const float* Lg, unsigned char* base, bool sorted) {
    static_assert(COLS <= L, "a lane per species");
    constexpr int LDR = LuCtx<L, COLS>::LDR;
    const LuLayout lay(COLS, N, R, Lg != nullptr, sorted);
    double* rates = reinterpret_cast<double*>(base + lay.rates);
    int* inc_off = reinterpret_cast<int*>(base + lay.inc_off);
    uint32_t* inc = reinterpret_cast<uint32_t*>(base + lay.inc);
    int* term_off = reinterpret_cast<int*>(base + lay.term_off);
    uint32_t* term = reinterpret_cast<uint32_t*>(base + lay.term);
    double* LT = reinterpret_cast<double*>(base + lay.lt);
    double* rows = reinterpret_cast<double*>(base + lay.rows);
    // `at`, in each species' Jacobian row: the terms of each column, counted, then
    // where the column's next one goes
    int* at = reinterpret_cast<int*>(rows + (l < N ? l : 0) * LDR);
    if (l < N) {
        inc_off[l + 1] = 0;
#pragma unroll 1
        for (int col = 0; col < N; col++) at[col] = 0;
    }
    __syncwarp(mask);
    bool bad = false;
#pragma unroll U
    for (int r = l; r < R; r += L) {
        const double k = __ldg(k_in + r);
        const uint2 q = __ldg(sp + r);
        // the reactants' s is -2 where they are one species that is not made
        // again, the products' +2 where they are one that is not consumed
        const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
        rates[2 * r] = (double)min(-1, stoich(a, a, b, cc, d)) * k;
        rates[2 * r + 1] = (double)max(1, stoich(cc, a, b, cc, d)) * k;
        if (max(max(a, b), max(cc, d)) >= N) {
            bad = true;
        } else {
            auto count = [&](bool on, int j) {
                if (!on) return;
                atomicAdd(inc_off + 1 + j, 1);
                if (sorted && stoich(j, a, b, cc, d)) {
                    int* row = reinterpret_cast<int*>(rows + j * LDR);
                    atomicAdd(row + a, 1);
                    atomicAdd(row + b, 1);
                }
            };
            count(true, a);
            count(b != a, b);
            count(cc != a && cc != b, cc);
            count(d != a && d != b && d != cc, d);
        }
    }
    __syncwarp(mask);
    if (__any_sync(mask, bad)) return true;
    int terms = 0;
    if (l < N) {
#pragma unroll 1
        for (int col = 0; col < N; col++) terms += at[col];
    }
    const int room = l < N ? (inc_off[l + 1] + 3) & ~3 : 0, term_room = (terms + 3) & ~3;
    const int inc_end = rx_scan<L>(mask, l, room), term_end = rx_scan<L>(mask, l, term_room);
    if (l < N) {
        inc_off[l + 1] = inc_end;
        if (sorted) term_off[l + 1] = term_end;
    }
    if (l == 0) {
        inc_off[0] = 0;
        if (sorted) term_off[0] = 0;
        rates[2 * R] = 0.0;
        rates[2 * R + 1] = __longlong_as_double(0x7ff8000000000000ll);
        reinterpret_cast<double*>(base + lay.vb)[COLS] = 0.0;
    }
    __syncwarp(mask);
    uint32_t* mine = inc + inc_end - room;
    const int cnt = rx_list<L>(mask, l, N, R, sp, reinterpret_cast<uint32_t*>(base + lay.pb), mine);
    if (l < N) {
        int t = term_end - term_room;
        const int t_first = t;
#pragma unroll 1
        for (int col = 0; col < N; col++) {
            const int n = at[col];
            at[col] = t;
            t += n;
        }
        uint2 next = cnt ? __ldg(sp + mine[0]) : make_uint2(0u, 0u);
#pragma unroll 1
        for (int e = 0; e < cnt; e++) {
            const uint2 q = next;
            const int r = (int)mine[e];
            if (e + 1 < cnt) next = __ldg(sp + mine[e + 1]);
            const int a = q.x & 0xffff, b = q.x >> 16;
            const int st = stoich(l, a, b, (int)(q.y & 0xffff), (int)(q.y >> 16));
            int slot = st < 0 ? 2 * r : 2 * r + 1;
            if (st == 0) slot = finite64(rates[2 * r]) || finite64(rates[2 * r + 1]) ? 2 * R : 2 * R + 1;  // 0 * k
            mine[e] = rx_pack(slot, a, b);
            if (sorted && st) {
                // d w / d y_a = k y_b, then d w / d y_b = k y_a, per column in list order
                const int ta = at[a], tb = a == b ? ta + 1 : at[b];
                at[a] = ta + 1;
                at[b] = tb + 1;
                term[ta] = rx_pack(slot, b, a);
                term[tb] = rx_pack(slot, a, b);
            }
        }
        // padding: rate zero, the zero beside the state, the column beside the row
#pragma unroll 1
        for (int e = cnt; e < room; e++) mine[e] = rx_pack(2 * R, COLS, COLS);
        if (sorted) {
            for (int col = 0, t0 = t_first; col < N; t0 = at[col], col++)
                if (at[col] > t0) term[at[col] - 1] |= RX_MARK;
            while (t < term_end) term[t++] = rx_pack(2 * R, COLS, COLS);
        }
        if (Lg) {
#pragma unroll 1
            for (int k = 0; k < N; k++) LT[k * N + l] = Lg[l * N + k];
        }
    }
    __syncwarp(mask);
    return false;
}

// The same, out of line: its registers are not the solve's.  (k_mixed, whose
// registers are those of the CTA kernels, has it inline.)
template <int L, int COLS>
__device__ __noinline__ bool lu_stage_apart(unsigned mask, int l, int N, int R, const double* k_in, const uint2* sp,
                                            const float* Lg, unsigned char* base, bool sorted) {
    return lu_stage<L, COLS, 4>(mask, l, N, R, k_in, sp, Lg, base, sorted);
}

// The same with every lane looking through all reactions and walking its list once
// per column, for k_mixed on networks of few reactions (mixed_counted): system s's
// rates, the dense term transposed, the incidence lists and the Jacobian terms.  A species index >= N marks the system BAD_INPUT
// (returned) and nothing of it is read again.
template <int L, int COLS>
__device__ __forceinline__ bool lu_stage_scan(const LuCtx<L, COLS>& c, const KParams& p, int64_t s, double* rates,
                                              int* inc_off, uint32_t* inc, int* term_off, uint32_t* term, double* LT) {
    const int N = c.N, R = p.n_react, l = c.l;
    const uint2* sp = reinterpret_cast<const uint2*>(p.species) + s * R;
    bool bad = false;
    for (int r = l; r < R; r += L) {
        const double k = p.rates[s * R + r];
        const uint2 q = __ldg(sp + r);
        // the reactants' s is -2 where they are one species that is not made
        // again, the products' +2 where they are one that is not consumed
        const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
        rates[2 * r] = (double)min(-1, stoich(a, a, b, cc, d)) * k;
        rates[2 * r + 1] = (double)max(1, stoich(cc, a, b, cc, d)) * k;
        const unsigned nn = (unsigned)N;
        bad = bad || (q.x & 0xffffu) >= nn || (q.x >> 16) >= nn || (q.y & 0xffffu) >= nn || (q.y >> 16) >= nn;
    }
    if (__any_sync(c.mask, bad)) return true;
    for (int j = l; j < N; j += L) {
        int cnt = 0, terms = 0;
        for (int r = 0; r < R; r++) {
            const uint2 q = __ldg(sp + r);
            const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
            cnt += (a == j) | (b == j) | (cc == j) | (d == j);
            terms += stoich(j, a, b, cc, d) ? 2 : 0;
        }
        inc_off[j + 1] = (cnt + 3) & ~3;
        term_off[j + 1] = (terms + 3) & ~3;
    }
    __syncwarp(c.mask);
    if (l == 0) {
        inc_off[0] = term_off[0] = 0;
        for (int j = 0; j < N; j++) {
            inc_off[j + 1] += inc_off[j];
            term_off[j + 1] += term_off[j];
        }
        rates[2 * R] = 0.0;
        rates[2 * R + 1] = __longlong_as_double(0x7ff8000000000000ll);
        c.vb[COLS] = 0.0;
    }
    __syncwarp(c.mask);
    for (int j = l; j < N; j += L) {
        int o = inc_off[j];
        for (int r = 0; r < R; r++) {
            const uint2 q = __ldg(sp + r);
            const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
            if (a != j && b != j && cc != j && d != j) continue;
            const int st = stoich(j, a, b, cc, d);
            int slot = st < 0 ? 2 * r : 2 * r + 1;
            if (st == 0) slot = finite64(rates[2 * r]) || finite64(rates[2 * r + 1]) ? 2 * R : 2 * R + 1;  // 0 * k
            inc[o++] = rx_pack(slot, a, b);
        }
        // d w / d y_a = k y_b, then d w / d y_b = k y_a, per column in list order
        const int e0 = inc_off[j];
        int t = term_off[j];
        for (int col = 0; col < N; col++) {
            const int t0 = t;
            for (int e = e0; e < o; e++) {
                const uint32_t q = inc[e];
                const int slot = (int)(q & 0x7ffffu) >> 3, a = (int)(rx_first(q) >> 3), b = (int)(rx_second(q) >> 3);
                if (slot >= 2 * R) continue;
                if (a == col) term[t++] = rx_pack(slot, b, col);
                if (b == col) term[t++] = rx_pack(slot, a, col);
            }
            if (t > t0) term[t - 1] |= RX_MARK;
        }
        // padding: rate zero, the zero beside the state, the column beside the row
        while (o < inc_off[j + 1]) inc[o++] = rx_pack(2 * R, COLS, COLS);
        while (t < term_off[j + 1]) term[t++] = rx_pack(2 * R, COLS, COLS);
        if (LT) {
            const float* Lg = p.linear + s * (int64_t)N * N;
            for (int k = 0; k < N; k++) LT[k * N + j] = Lg[j * N + k];
        }
    }
    __syncwarp(c.mask);
    return false;
}

// Warps per SM the registers are planned for.  8 (250 registers at 32 columns)
// and 10 or 12 (200, 168) measured alike on 3,000 dense systems of 32 species
// (696, 682, 701 ms); alone on an SM a substep takes 6.0 us with 8, 7.1 us with
// the others.
constexpr int LU_BLOCKS = 8;

// The persistent team loop over one group's systems: the first `tpw` teams of
// every warp (of the block's first `teams` teams) take tickets from the group's
// queue until it is empty.  `smem_raw` holds `teams` team slices, laid out with or
// without the sorted Jacobian terms (GUARD: with).
template <int L, int COLS, bool GUARD, int CTRL, bool COUNTED>
__device__ __forceinline__ void lu_run(const KParams& p, unsigned char* smem_raw, int teams, int tpw, bool sorted) {
    using Ctx = LuCtx<L, COLS>;
    constexpr int CAP = Cap<WIND_METHOD_SIE, CTRL>::value;
    const bool lin = p.linear != nullptr;
    const LuLayout lay(COLS, p.n_eq, p.n_react, lin, sorted);
    const int lane = threadIdx.x & 31;
    Ctx c;
    c.l = lane % L;
    c.leader = lane - c.l;
    c.mask = (L >= 32) ? 0xffffffffu : (((1u << (L & 31)) - 1u) << c.leader);
    c.tm = lane / L;
    // Every lane of the warp stays in the loop to the end, so its steps use
    // warp-wide barriers, reductions and shuffles; teams beyond the working
    // ones, and those left without a system, write nothing (they read the
    // slice of the warp's first team).
    const int team0 = (threadIdx.x >> 5) * tpw;
    if (team0 >= teams) return;
    const bool works = c.tm < min(tpw, teams - team0);
    const int team = works ? team0 + c.tm : team0;
    c.live = false;
    c.N = p.n_eq;
    unsigned char* base = smem_raw + team * lay.bytes;
    double* rates = reinterpret_cast<double*>(base + lay.rates);
    int* inc_off = reinterpret_cast<int*>(base + lay.inc_off);
    uint32_t* inc = reinterpret_cast<uint32_t*>(base + lay.inc);
    int* term_off = reinterpret_cast<int*>(base + lay.term_off);
    uint32_t* term = sorted ? reinterpret_cast<uint32_t*>(base + lay.term) : nullptr;
    double* LT = lin ? reinterpret_cast<double*>(base + lay.lt) : nullptr;
    c.rates = rates;
    c.inc_off = inc_off;
    c.inc = inc;
    c.term_off = term_off;
    c.term = term;
    c.LT = LT;
    c.vb = reinterpret_cast<double*>(base + lay.vb);
    double* rows = reinterpret_cast<double*>(base + lay.rows);
    double* rows2 = reinterpret_cast<double*>(base + lay.rows2);
    c.pb = reinterpret_cast<double*>(base + lay.pb);
    const int N = c.N, l = c.l;
    const uint64_t t_start = p.timeout_ns ? global_ns() : 0;
    const double tend = p.tend;

    enum { ATTEMPT, FULL, HALF1, HALF2 };
    int phase = works ? ATTEMPT : FULL;
    int64_t s = -1, attempts = 0;
    double y = 0.0, y1 = 0.0, vh = 0.0, fy = 0.0;
    double tnow = 0.0, h = 0.0, hf = 0.0, h1 = 0.0, h2 = 0.0, h_vh = 0.0;
    int unsolved = 0;
    int32_t st = WIND_SYS_OK;
    bool stop = false;
    bool fy_ok = false;  // fy is f(y)
    bool jy_ok = false;  // the rows hold the Jacobian at y
    bool vh_ok = false;  // vh is the substep of size h_vh from y
    while (true) {
        // ---- between attempts: finish, take the next system, set the sizes
        while (phase == ATTEMPT) {
            if (s < 0) {
                unsigned long long ticket = 0;
                if (l == 0) ticket = atomicAdd(&p.counters[CNT_QUEUE], 1ull);
                s = (int64_t)__shfl_sync(c.mask, ticket, c.leader);
                c.live = s < p.nsys;
                if (!c.live) {
                    phase = FULL;  // no system left: idle turns from here on
                    break;
                }
                if constexpr (COUNTED) {
                    const double* k = p.rates + s * p.n_react;
                    const uint2* sp = reinterpret_cast<const uint2*>(p.species) + s * p.n_react;
                    const float* Lg = lin ? p.linear + s * (int64_t)N * N : nullptr;
                    stop = GUARD ? lu_stage<L, COLS, 1>(c.mask, l, N, p.n_react, k, sp, Lg, base, true)
                                 : lu_stage_apart<L, COLS>(c.mask, l, N, p.n_react, k, sp, Lg, base, sorted);
                } else {
                    stop = lu_stage_scan(c, p, s, rates, inc_off, inc, term_off, term, LT);
                }
                st = stop ? WIND_SYS_BAD_INPUT : WIND_SYS_OK;
                y = (l < N) ? p.y[s * N + l] : 0.0;
                tnow = p.tnow;
                h = p.h0;
                unsolved = 0;
                attempts = 0;
                fy_ok = jy_ok = vh_ok = false;
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
                if (l < N) p.y[s * N + l] = y;
                if (__any_sync(c.mask, bad)) st |= WIND_SYS_NONFINITE;
                if (l == 0) {
                    if (p.sys_status) p.sys_status[s] = st;
                    if (p.sys_nsteps) p.sys_nsteps[s] = 3 * attempts;
                    atomicAdd(&p.counters[CNT_STEPS], (unsigned long long)(3 * attempts));
                }
                __syncwarp(c.mask);
                s = -1;
                continue;
            }
            attempts++;
            h = fmin(tend - tnow, h);
            const double t1 = tnow + h;
            hf = t1 - tnow;            // the full substep
            h1 = (t1 - tnow) * 0.5;    // the first half substep
            h2 = (CTRL == WIND_CTRL_DEVICE) ? fmin(t1 - (tnow + h1), h1) : h1;
            phase = FULL;
            if (vh_ok && hf == h_vh) {
                y1 = vh;
                phase = HALF1;
            }
        }
        // ---- one substep
        if (!__any_sync(0xffffffffu, c.live)) return;
        const bool second = phase == HALF2;
        const double hs = phase == FULL ? hf : (second ? h2 : h1);
        const double v = second ? vh : y;
        if (c.live && l < N) c.vb[l] = v;
        __syncwarp();
        double f = fy;
        if (c.live && (second || !fy_ok)) {
            f = (l < N) ? lu_rhs<Ctx, COLS>(c, l) : 0.0;
            if (!second) fy = f;
            fy_ok = true;  // f(vh) leaves f(y) in fy
        }
        c.rows = second ? rows2 : rows;
        if (c.live && (second || !jy_ok)) {
            if (l < N) {
                if (GUARD || c.term) lu_jac_row<Ctx, COLS>(c, l);
                else lu_jac_row_in_place<COLS>(c.rates, c.inc + c.inc_off[l], c.inc_off[l + 1] - c.inc_off[l], c.vb,
                                               c.rows + l * Ctx::LDR, 16u * p.n_react);
            }
            jy_ok = !second || lay.rows2 != lay.rows;
        }
        double x;
        {
            double a[COLS];
            lu_load_row<Ctx, COLS>(c, l, hs, a);
            x = lu_solve<GUARD, false>(c, a, f);
        }
        const bool finite = mag_hi(x) < HI_INF || !c.live;
        if (!__all_sync(0xffffffffu, finite))
            x = lu_solve_exact<GUARD, L, COLS>(l, c.leader, N, c.tm, c.live, c.LT, c.rows, c.pb, hs, f);
        const double out = fma(hs, x, v);
        const bool err = (__ballot_sync(0xffffffffu, c.live && second && l < N &&
                                        elem_error<WIND_METHOD_SIE, CTRL>(xd(y1), xd(out), p.atol, p.rtol)) &
                          c.mask) != 0u;
        if (!c.live) continue;
        if (phase == FULL) {
            y1 = out;
            phase = HALF1;
        } else if (phase == HALF1) {
            vh = out;
            h_vh = h1;
            phase = HALF2;
        } else {
            if (err && unsolved < CAP) {
                unsolved++;
                h /= 2.0;
                vh_ok = true;
            } else {
                unsolved = 0;
                y = out;
                fy_ok = jy_ok = vh_ok = false;
                if (tnow + h == tnow) {
                    st |= WIND_SYS_STALLED;
                    stop = true;
                } else {
                    tnow += h;
                    h = tend - tnow;
                }
            }
            phase = ATTEMPT;
        }
    }
}

template <int L, int COLS, int CTRL>
__global__ void __launch_bounds__(32, LU_BLOCKS) k_lu(const KParams p, int tpw, int sorted) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    lu_run<L, COLS, false, CTRL, true>(p, smem_raw, tpw, tpw, sorted != 0);
}

}  // namespace wind
