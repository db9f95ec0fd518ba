// solvers_reg.cuh -- register-resident linear solves for small compile-time N
// (one thread owns a whole system).  All loops unroll, so the matrices stay in
// registers.
#pragma once

#include "common.cuh"

namespace wind {

// The reference's unpivoted Gauss-Jordan inverse of M (row-major), same
// operation order as cuda/c_baseline/linear_algebra/gje_gold.c:5-144 and
// cuda/linear_algebra/gauss_jordan_elimination.cu:15-212: per pivot row, every
// element of the row of M and of Inv is divided by the saved pivot; rows below
// (U phase) then rows above (L phase, bottom-up) subtract factor*pivot row
// over the full width.
template <int N>
__device__ __forceinline__ void gje_invert_reg(xd (&M)[N * N], xd (&Inv)[N * N]) {
#pragma unroll
    for (int e = 0; e < N * N; e++) Inv[e] = 0.0;
#pragma unroll
    for (int i = 0; i < N; i++) Inv[i * (N + 1)] = 1.0;
#pragma unroll
    for (int i = 0; i < N; i++) {
        xd s = M[i * N + i];
#pragma unroll
        for (int t = 0; t < N; t++) M[i * N + t] /= s;
#pragma unroll
        for (int t = 0; t < N; t++) Inv[i * N + t] /= s;
#pragma unroll
        for (int k = i + 1; k < N; k++) {
            xd f = M[k * N + i];
#pragma unroll
            for (int t = 0; t < N; t++) M[k * N + t] -= f * M[i * N + t];
#pragma unroll
            for (int t = 0; t < N; t++) Inv[k * N + t] -= f * Inv[i * N + t];
        }
    }
#pragma unroll
    for (int ri = 0; ri < N; ri++) {
        const int bri = N - 1 - ri;
#pragma unroll
        for (int nri = ri + 1; nri < N; nri++) {
            const int bnri = N - 1 - nri;
            xd f = M[bnri * N + bri];
#pragma unroll
            for (int t = 0; t < N; t++) M[bnri * N + t] -= f * M[bri * N + t];
#pragma unroll
            for (int t = 0; t < N; t++) Inv[bnri * N + t] -= f * Inv[bri * N + t];
        }
    }
}

// Partial-pivot LU factorisation of A (row-major, standard orientation) in
// place, with the row swaps applied as predicated selects so indexing stays
// static.  Returns the reciprocal pivots in `rinv` and applies the same row
// permutation to the right-hand sides through `perm` (perm[i] = original row).
template <int N, typename T>
__device__ __forceinline__ void lu_factor_reg(T (&A)[N * N], T (&rinv)[N], int (&perm)[N]) {
#pragma unroll
    for (int i = 0; i < N; i++) perm[i] = i;
#pragma unroll
    for (int i = 0; i < N; i++) {
        int p = i;
        T best = fabs(A[i * N + i]);
#pragma unroll
        for (int k = i + 1; k < N; k++) {
            T v = fabs(A[k * N + i]);
            if (v > best) { best = v; p = k; }
        }
#pragma unroll
        for (int k = i + 1; k < N; k++) {
            const bool sw = (p == k);
#pragma unroll
            for (int t = 0; t < N; t++) {
                T a = A[i * N + t], b = A[k * N + t];
                A[i * N + t] = sw ? b : a;
                A[k * N + t] = sw ? a : b;
            }
            int pa = perm[i], pb = perm[k];
            perm[i] = sw ? pb : pa;
            perm[k] = sw ? pa : pb;
        }
        T r = nr_rcp(A[i * N + i]);
        rinv[i] = r;
#pragma unroll
        for (int k = i + 1; k < N; k++) {
            T l = A[k * N + i] * r;
            A[k * N + i] = l;
#pragma unroll
            for (int t = i + 1; t < N; t++) A[k * N + t] = fma(-l, A[i * N + t], A[k * N + t]);
        }
    }
}

// Solve with the factors from lu_factor_reg: x = A^-1 b (b in original row
// order, x in place of b).
template <int N, typename T, typename B>
__device__ __forceinline__ void lu_solve_reg(const T (&A)[N * N], const T (&rinv)[N],
                                             const int (&perm)[N], B (&b)[N]) {
    B z[N];
    // permute: z[i] = b[perm[i]] via selects
#pragma unroll
    for (int i = 0; i < N; i++) {
        B v = b[0];
#pragma unroll
        for (int q = 1; q < N; q++) v = (perm[i] == q) ? b[q] : v;
        z[i] = v;
    }
    // forward (unit lower)
#pragma unroll
    for (int i = 1; i < N; i++) {
        B acc = z[i];
#pragma unroll
        for (int t = 0; t < i; t++) acc = fma(-(B)A[i * N + t], z[t], acc);
        z[i] = acc;
    }
    // backward
#pragma unroll
    for (int i = N - 1; i >= 0; i--) {
        B acc = z[i];
#pragma unroll
        for (int t = i + 1; t < N; t++) acc = fma(-(B)A[i * N + t], z[t], acc);
        z[i] = acc * (B)rinv[i];
    }
#pragma unroll
    for (int i = 0; i < N; i++) b[i] = z[i];
}

// ---------------------------------------------------------------------------
// Block forms.  The compiled networks' Jacobians are block diagonal (Katz96:
// hydrogen 2x2, helium 3x3 tridiagonal), and an off-block entry of the
// full-width eliminations above is an exact zero: a row operation with a zero
// multiplier, a quotient 0/s or a product with a zero leaves every in-block
// value as it is while nothing is infinite or NaN.  The block forms do the
// in-block operations only, in the same order, so their results are the
// full-width ones bit for bit (a zero's sign aside) whenever the largest high
// word of the values named below stays under HI_INF; otherwise the caller repeats
// the substep full width.  The Gauss-Jordan inverse of a Katz96 substep (blocks of
// 2 and 3) then takes 12 divisions instead of the full width's 50, and its row
// operations are those inside the blocks instead of 20 of 10 elements; the LU takes
// one pivot comparison per column.
constexpr int HI_INF = 0x7ff00000;
__device__ __forceinline__ int mag_hi(double x) { return __double2hiint(x) & 0x7fffffff; }

// The reference's Gauss-Jordan inverse of one n x n block (reference
// orientation).  Columns of M left of the pivot and columns of Inv right of it
// are still zeros in the downward pass, and M's rows are unit rows by the time
// the upward pass uses them.  `hi`: largest high word over the pivots.
template <int n, bool TRI>
__device__ __forceinline__ void gje_invert_block(xd (&M)[n * n], xd (&Inv)[n * n], int& hi) {
#pragma unroll
    for (int i = 0; i < n; i++) {
        const xd s = M[i * n + i];
        hi = max(hi, mag_hi(s.v));
#pragma unroll
        for (int t = i + 1; t < n; t++)
            if (!TRI || t == i + 1) M[i * n + t] /= s;
#pragma unroll
        for (int t = 0; t < i; t++) Inv[i * n + t] /= s;
        Inv[i * n + i] = xd(1.0) / s;
#pragma unroll
        for (int k = i + 1; k < n; k++) {
            if (TRI && k > i + 1) continue;
            const xd f = M[k * n + i];
#pragma unroll
            for (int t = i + 1; t < n; t++)
                if (!TRI || t == i + 1) M[k * n + t] -= f * M[i * n + t];
#pragma unroll
            for (int t = 0; t <= i; t++) {
                // Inv[k][t] is zero until the first row that reaches it
                const bool first = TRI || t == i;
                Inv[k * n + t] = first ? -(f * Inv[i * n + t]) : Inv[k * n + t] - f * Inv[i * n + t];
            }
        }
    }
#pragma unroll
    for (int b = n - 1; b > 0; b--) {
#pragma unroll
        for (int k = b - 1; k >= 0; k--) {
            if (TRI && k < b - 1) continue;
            const xd f = M[k * n + b];
#pragma unroll
            for (int t = 0; t < n; t++) {
                // right of the diagonal Inv[k][t] is zero until the first
                // pivot row that reaches it
                const bool first = t > k && (TRI || b == n - 1);
                Inv[k * n + t] = first ? -(f * Inv[b * n + t]) : Inv[k * n + t] - f * Inv[b * n + t];
            }
        }
    }
}

// Partial-pivot LU solve of one block, A x = b (x in place of b): the pivots,
// multipliers and sums of lu_factor_reg / lu_solve_reg.  In a tridiagonal
// block only the next row holds a nonzero below the pivot.
template <int n, bool TRI>
__device__ __forceinline__ void lu_solve_block(double (&A)[n * n], double (&b)[n]) {
    double rinv[n];
#pragma unroll
    for (int i = 0; i < n; i++) {
        int p = i;
        double best = fabs(A[i * n + i]);
#pragma unroll
        for (int k = i + 1; k < n; k++) {
            if (TRI && k > i + 1) continue;
            const double v = fabs(A[k * n + i]);
            if (v > best) { best = v; p = k; }
        }
#pragma unroll
        for (int k = i + 1; k < n; k++) {
            if (TRI && k > i + 1) continue;
            const bool sw = (p == k);
#pragma unroll
            for (int t = i; t < n; t++) {
                const double u = A[i * n + t], w = A[k * n + t];
                A[i * n + t] = sw ? w : u;
                A[k * n + t] = sw ? u : w;
            }
            const double u = b[i], w = b[k];
            b[i] = sw ? w : u;
            b[k] = sw ? u : w;
        }
        const double r = nr_rcp(A[i * n + i]);
        rinv[i] = r;
#pragma unroll
        for (int k = i + 1; k < n; k++) {
            if (TRI && k > i + 1) continue;
            const double l = A[k * n + i] * r;
#pragma unroll
            for (int t = i + 1; t < n; t++) A[k * n + t] = fma(-l, A[i * n + t], A[k * n + t]);
            b[k] = fma(-l, b[i], b[k]);
        }
    }
#pragma unroll
    for (int i = n - 1; i >= 0; i--) {
        double acc = b[i];
#pragma unroll
        for (int t = i + 1; t < n; t++) acc = fma(-A[i * n + t], b[t], acc);
        b[i] = acc * rinv[i];
    }
}

}  // namespace wind
