// cta_kernel.cuh -- persistent CTA-per-system integrator for mass-action
// networks with 32 < N <= 256 (the 64- and 157-species classes).
//
// One CTA (128 or 256 threads, cta_block_threads) integrates one system at a time
// and pulls the next ticket from the device work queue when it finishes.  Thread l
// owns equation l (N <= 256): its y, y1, y2 live in registers.  Per system the CTA
// builds per-species incidence lists of the reactions (CSR, reaction ids
// ascending) and, for the implicit solves, records of them where a launch has the
// room (cta_incidences), so thread j evaluates f_j and row j of the Jacobian from
// the ~4R/N reactions that touch species j instead of all R.
//
// Solvers (selected at compile time):
//  GJE_F64  the reference's unpivoted Gauss-Jordan inverse, reference
//           operation order, on M and Inv in a per-CTA global scratch slot
//           (2 N^2 doubles; L2-resident) -- bit-exact parity path;
//  LU_F64   blocked right-looking LU with partial pivoting, FP64, on the
//           matrix [A | b] in shared memory (global scratch when it does not
//           fit), followed by blocked triangular solves;
//  MIXED    one FP32 Gauss-Jordan inverse per attempt, unpivoted and blocked
//           (cta_gj_invert) or, at step sizes where that one failed, pivoted
//           (cta_gj_invert_pivoted); every solve of the attempt refines around it
//           in FP64 with the residual r = f - (x - h J x) from the reactions, no
//           FP64 matrix, until the predicted error is below 2^-33 of |x|
//           (cta_refine).  What does not refine goes to an FP32 LU with partial
//           pivoting (cta_mixed_pivoted_solve).  Its footprint lets two CTAs
//           share an SM at N = 157.
//
// Blocked LU (cta_lu, panel width CTA_NB = 16).  Rows never move: logical row i is
// physical row piv[i].  For each panel:
//  1. panel factorisation: thread p holds the 16 panel entries of physical
//     row p in registers.  Per column one CTA barrier: each warp's best
//     candidate (max |a| by a __reduce_max_sync key) publishes its row's
//     panel entries and reciprocal pivot in a per-warp slot (double-
//     buffered) and its packed (key, row) in a 64-bit atomicMax vote (lowest
//     row on ties); after the barrier every thread reads the winner and
//     eliminates its own row in registers;
//  2. the still-active rows are compacted into act[] (warp ballots);
//  3. U12 = L11^-1 A12 for the 16 pivot rows, one thread per column;
//  4. trailing update A22 -= L21 U12 over act[] x columns, 4x4 register
//     tiles with 16-byte shared-memory vectors.
// The right-hand side is column N, so the forward elimination comes with the
// factorisation; the row stride is padded so that rows start 16 bytes apart
// in the bank space (no conflicts when 32 rows are read at one column).
#pragma once

#include <type_traits>

#include "common.cuh"
#include "tc_sm100.cuh"
#include "networks.cuh"

namespace wind {

constexpr int CTA_THREADS = 256;
constexpr int CTA_WARPS = CTA_THREADS / 32;
constexpr int CTA_MAXN = 256;
constexpr int CTA_NB = 16;  // LU panel width
constexpr int CTA_REC_MAXR = 8192;  // reactions up to which a slot holds records (0.8 MB)
constexpr int CTA_CONV = 14; // misc[] slot: refinement converged (0/1)
constexpr int CTA_TCPAR = 15; // misc[] slot: phase parity of the tensor-core mbarrier

// Threads of a k_cta block.  A small system leaves half of 256 threads without an
// equation, and half the threads let more blocks onto an SM (registers), which
// counts while there are more systems than SMs (`many`).  The Gauss-Jordan
// elimination and the implicit solves' rank updates share N^2 elements out over
// the block, whose size counts where they last.  128 against 256 threads, us:
//   Gauss-Jordan  N = 48: 1 system 963, 778; 600 systems 2064, 3583
//                 N = 64: 1 system 1691, 1226; 600 systems 5193, 5894
//                 N = 80: 600 systems 16137, 9468; N = 128: 1 system 25781, 10354
//   LU_F64        N = 48: 1 system 1251, 1266; 600 systems 3623, 5849
//                 N = 128: 1 system 3656, 3563; 600 systems 17344, 16916
//   MIXED         N = 33: 600 systems 2599, 2976; N = 80: 1188, 1138 and 3600, 4056
//                 N = 128: 1 system 2308, 2171; 600 systems 7924, 7623
//   RK2           N = 64: 1 system 823, 824; 600 systems 1858, 2483
// The tensor-core staging is laid out for 256.
__host__ __device__ constexpr int cta_block_threads(int n, int solver, bool rk2, bool tc, bool many) {
    const int half = CTA_THREADS / 2;
    if (tc || n > half) return CTA_THREADS;
    if (rk2) return half;
    if (solver == WIND_SOLVER_GJE_F64) return many && n <= 64 ? half : CTA_THREADS;
    return n <= 64 || (many && solver == WIND_SOLVER_MIXED && n <= 112) ? half : CTA_THREADS;
}

// A warp's pivot candidate for one panel column: its best row's panel
// entries and the reciprocal of the entry in the column.
template <typename T>
struct CtaCand {
    T rcp;                      // 1 / vals[column] (computed before the vote)
    alignas(16) T vals[CTA_NB];
};
static_assert(sizeof(CtaCand<float>) == 16 + CTA_NB * 4, "candidate slot size");
static_assert(sizeof(CtaCand<double>) == 16 + CTA_NB * 8, "candidate slot size");

// Shared-memory and global-scratch layout of one CTA, computed on the host
// and the device alike.  Shared memory holds, in order of priority, the
// vectors, the pivot bookkeeping, the dense linear term, the matrix and the
// incidence lists; whatever does not fit under `smem_cap` goes to the CTA's
// global scratch slot.
struct CtaLayout {
    int ld;            // matrix row stride (elements)
    int cols;          // columns that hold data (<= ld, a multiple of 4)
    int esz;           // matrix element size (bytes)
    int nvec;          // FP64 vectors of length N
    int vec, piv, act, misc, cand, tcs, lt, mat, inc_off, inc, rt, spc, bytes;
    bool mat_in_smem, inc_in_smem, data_in_smem;
    size_t g_mat, g_inc, g_doubles;  // global slot: offsets and size in doubles
    // Reaction records (SIE with LU_F64 or MIXED; RK2 reads none): rec_cap records
    // of 12 bytes, in shared memory at `rec` (rec_in_smem) or behind the global
    // slot's other parts (g_rec, rec_doubles); a launch without that room goes
    // without them.
    int rec_cap, rec;
    bool rec_in_smem;
    size_t g_rec, rec_doubles;
    __host__ __device__ static int a16(int x) { return (x + 15) & ~15; }
    // columns read or written: >= N+1, whole panels, whole 4-wide tiles
    __host__ __device__ static int data_cols(int N) {
        const int a = (N + 15) & ~15, b = (N + 1 + 3) & ~3;
        return a > b ? a : b;
    }
    // rows 16 bytes apart modulo the 128-byte bank space
    __host__ __device__ static int row_stride(int N, int esz) {
        const int base = data_cols(N);
        const int per = 128 / esz, want = 16 / esz;  // elements per bank sweep / per 16 B
        return base + ((want - base % per) + per) % per;
    }
    // Tensor-core staging of the MIXED inverse's rank-16 updates (tc): the
    // mbarrier and tensor-memory address (64 B), the update's left operand
    // (128 rows x 16, TF32 high and low parts, 16 KB) and right operand
    // (columns rounded up to 16 x 16, high and low parts).
    __host__ __device__ static int tc_stage_bytes(int N) {
        return 64 + 4 * 4096 + 4 * ((N + 15) & ~15) * 32;
    }
    __host__ __device__ CtaLayout(int N, int R, bool lin, int solver, int smem_cap, bool tc = false,
                                  bool records = true) {
        esz = (solver == WIND_SOLVER_MIXED) ? 4 : 8;
        ld = row_stride(N, esz);
        cols = data_cols(N);
        nvec = (solver == WIND_SOLVER_GJE_F64) ? 3 : (solver == WIND_SOLVER_LU_F64 ? 4 : 5);
        int off = 0;
        vec = off; off = a16(off + nvec * N * 8);
        piv = off; off = a16(off + N * 4);
        act = off; off = a16(off + N * 4);
        misc = off; off = a16(off + 2 * CTA_WARPS * 4);
        cand = off; off = a16(off + (solver == WIND_SOLVER_GJE_F64 ? 0 : 2 * CTA_WARPS * (16 + CTA_NB * esz)));
        tcs = off; off = a16(off + (tc ? tc_stage_bytes(N) : 0));
        lt = off; off = a16(off + (lin ? N * N * 4 : 0));
        const int mbytes = (solver == WIND_SOLVER_GJE_F64) ? 0 : a16(N * ld * esz);
        mat = off;
        mat_in_smem = (off + mbytes) <= smem_cap;
        if (mat_in_smem) off += mbytes;
        const int ibytes = a16((N + 1) * 4) + a16(4 * R * 2);
        inc_off = off;
        inc_in_smem = (off + ibytes) <= smem_cap;
        if (inc_in_smem) {
            inc = off + a16((N + 1) * 4);
            off += ibytes;
        } else {
            inc = 0;
        }
        // the system's rates and species, staged once per system
        rt = off;
        spc = a16(off + R * 8);
        data_in_smem = (spc + a16(R * 8)) <= smem_cap;
        if (data_in_smem) off = spc + a16(R * 8);
        // room for twice the average incidence count in every species' list
        rec_cap = !records || solver == WIND_SOLVER_GJE_F64 || R > CTA_REC_MAXR ? 0 : 8 * R + 8 * ((N + 31) & ~31);
        rec = off;
        rec_in_smem = rec_cap > 0 && off + 12 * rec_cap <= smem_cap;
        if (rec_in_smem) off = a16(off + 12 * rec_cap);
        bytes = off;
        // global slot: [GJE M, Inv][matrix][incidence lists]
        size_t g = (solver == WIND_SOLVER_GJE_F64) ? (size_t)2 * N * N : 0;
        g_mat = g;
        if (!mat_in_smem) g += ((size_t)N * ld * esz + 15) / 16 * 2;
        g_inc = g;
        if (!inc_in_smem) g += ((size_t)ibytes + 15) / 16 * 2;
        g_doubles = g;
        g_rec = (g + 1) & ~(size_t)1;
        rec_doubles = rec_cap && !rec_in_smem ? (size_t)rec_cap * 3 / 2 + 2 : 0;
    }
    // the global slot of a launch that may allocate
    __host__ __device__ size_t slot_doubles() const { return rec_doubles ? g_rec + rec_doubles : g_doubles; }
};

struct CtaCtx {
    int N, R, ld, cols;
    const double* rates;     // global [R]
    const uint16_t* sp;      // global [R*4]
    const float* LT;         // smem [N*N] or null
    const int* inc_off;      // [N+1] (shared or global)
    const uint16_t* inc;
    double *v, *f, *x, *r, *rinv, *scr;
    // reaction records of the species of each warp, transposed: entry e of
    // species 32 w + i at (rec_off[w] + e) * 32 + i; null: none (the lists above)
    const double* rec_k;     // s * k, s the species' net stoichiometry (not 0)
    const uint32_t* rec_ab;  // reactants a | b << 16
    int rec_off[CTA_WARPS + 1];
    int* piv;    // logical row -> physical row
    int* act;    // active rows of the trailing update
    int* misc;   // warp counts [CTA_WARPS]
    unsigned long long* best;  // pivot vote, three rotating slots (in misc, behind the counts)
    // CTA-wide maxima (float bits), three rotating slots.  A vote leaves its last
    // pivot in `best`, and a refinement right behind it may start in any slot: the
    // two share no word.
    unsigned maxima[3];
    void* cand;  // CtaCand<T>[2][CTA_WARPS]
    // tensor-core rank updates (MIXED_TC): accumulator base in tensor
    // memory, completion mbarrier, operand staging, columns rounded to 16
    uint32_t tmem;
    uint64_t* mbar;
    unsigned char* tcs;
    int tc_cols16;
};

// The block's context, in shared memory: the out-of-line routines read it there
// (passed by reference it would live in each thread's local memory, which the
// two blocks' shared memory leaves no cache for).
static __shared__ CtaCtx cta_ctx;

// 4 consecutive elements through 16-byte shared/global vectors.
__device__ __forceinline__ void ld4(const float* p, float (&a)[4]) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    a[0] = t.x; a[1] = t.y; a[2] = t.z; a[3] = t.w;
}
__device__ __forceinline__ void ld4(const double* p, double (&a)[4]) {
    const double2 t0 = reinterpret_cast<const double2*>(p)[0];
    const double2 t1 = reinterpret_cast<const double2*>(p)[1];
    a[0] = t0.x; a[1] = t0.y; a[2] = t1.x; a[3] = t1.y;
}
__device__ __forceinline__ void st4(float* p, const float (&a)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(a[0], a[1], a[2], a[3]);
}
__device__ __forceinline__ void st4(double* p, const double (&a)[4]) {
    reinterpret_cast<double2*>(p)[0] = make_double2(a[0], a[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(a[2], a[3]);
}

template <typename T>
__device__ __forceinline__ void ld4at(const T* p, T* a) {
    T t[4];
    ld4(p, t);
    a[0] = t[0]; a[1] = t[1]; a[2] = t[2]; a[3] = t[3];
}
template <typename T>
__device__ __forceinline__ void st4at(T* p, const T* a) {
    const T t[4] = {a[0], a[1], a[2], a[3]};
    st4(p, t);
}

// Threads of the block: CTA_THREADS, or fewer for small systems (at least N).
__device__ __forceinline__ int cta_threads() { return (int)blockDim.x; }
__device__ __forceinline__ int cta_warps() { return (int)blockDim.x >> 5; }

// Pivot ordering key: |a| as an unsigned integer (FP64: the high word, so
// magnitudes within 2^-20 of each other tie and the lower row wins).
__device__ __forceinline__ uint32_t mag_key(float a) { return __float_as_uint(fabsf(a)); }
__device__ __forceinline__ uint32_t mag_key(double a) {
    return (uint32_t)((unsigned long long)__double_as_longlong(fabs(a)) >> 32);
}

// f_j for j = tid (FP64, the sequential per-element order of the
// mass-action contract) into c.f.
__device__ __forceinline__ void cta_rhs() {
    const CtaCtx& c = cta_ctx;
    const int N = c.N, j = (int)threadIdx.x;
    if (j < N) {
        xd acc = 0.0;
        if (c.LT)
            for (int k = 0; k < N; k++) acc += xd((double)c.LT[k * N + j]) * xd(c.v[k]);
        const int e0 = c.inc_off[j], e1 = c.inc_off[j + 1];
        for (int e = e0; e < e1; e++) {
            const int rr = c.inc[e];
            const uint2 q = *reinterpret_cast<const uint2*>(c.sp + 4 * rr);
            const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
            const xd w = xd(c.rates[rr]) * xd(c.v[a]) * xd(c.v[b]);
            if (a == j) acc -= w;
            if (b == j) acc -= w;
            if (cc == j) acc += w;
            if (d == j) acc += w;
        }
        c.f[j] = acc.v;
    }
    __syncthreads();
}

// Visit the reactions that change species j = threadIdx.x (ascending ids):
// fn(load(ks, a, b)) with the reactants a, b and ks = s k, s = [C == j] + [D == j]
// - [A == j] - [B == j] (s = 0 skipped), `cnt` of them.  From the records, four
// at a time with the operands of the next four and the records after those in
// flight: coalesced, no dependent lookups and no branches around the loads (the
// species' lists through rates and species arrays, tested per entry, took 375
// cycles an entry in shared memory and 1,100 from L2).  fn is called on every
// entry of the warp's longest list and told whether it counts.
template <typename L, typename F>
__device__ __forceinline__ void cta_incidences(int cnt, L&& load, F&& fn) {
    const CtaCtx& c = cta_ctx;
    const int j = (int)threadIdx.x;
    if (c.rec_k) {
        const int w = j >> 5, width = c.rec_off[w + 1] - c.rec_off[w];  // a multiple of 4
        if (width == 0) return;
        const double* rk = c.rec_k + (size_t)c.rec_off[w] * 32 + (j & 31);
        const uint32_t* rab = c.rec_ab + (size_t)c.rec_off[w] * 32 + (j & 31);
        using Op = decltype(load(0.0, 0, 0));
        double k[4];
        uint32_t ab[4];
        Op op[4];
#pragma unroll
        for (int u = 0; u < 4; u++) op[u] = load(rk[32 * u], (int)(rab[32 * u] & 0xffffu), (int)(rab[32 * u] >> 16));
        int en = width > 4 ? 4 : 0;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            k[u] = rk[32 * (en + u)];
            ab[u] = rab[32 * (en + u)];
        }
        for (int e = 0; e < width; e += 4) {
            // the records after the next four, the operands of the next four
            Op next[4];
#pragma unroll
            for (int u = 0; u < 4; u++) next[u] = load(k[u], (int)(ab[u] & 0xffffu), (int)(ab[u] >> 16));
            en = e + 8 < width ? e + 8 : e;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                k[u] = rk[32 * (en + u)];
                ab[u] = rab[32 * (en + u)];
            }
#pragma unroll
            for (int u = 0; u < 4; u++) fn(op[u], e + u < cnt);
#pragma unroll
            for (int u = 0; u < 4; u++) op[u] = next[u];
        }
        return;
    }
    const int e1 = c.inc_off[j + 1];
    for (int e = c.inc_off[j]; e < e1; e++) {
        const int rr = c.inc[e];
        const uint2 q = *reinterpret_cast<const uint2*>(c.sp + 4 * rr);
        const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
        const int sg = (cc == j) + (d == j) - (a == j) - (b == j);
        if (sg) fn(load((double)sg * c.rates[rr], a, b), true);
    }
}

// [A | b] = [I - h J | f] in standard orientation (J[j][c] = Jt[c][j]), and
// f into c.f.  Thread j owns row j: it starts the row from L (or zero),
// accumulates f_j and the row's Jacobian entries from its reactions, then
// scales the row and writes f_j as column N.  (The LU and mixed solvers are
// not bit-exact by design; the reference-order evaluation is cta_rhs /
// cta_gje_exact.)
template <typename T, bool SMEM>
__device__ __noinline__ void cta_build(double h, T* A, int cnt) {
    const CtaCtx& c = cta_ctx;
    if (SMEM) __builtin_assume(__isShared(A));
    const int N = c.N, j = (int)threadIdx.x, ld = c.ld;
    const int q4 = c.cols >> 2;  // 4-wide chunks per row that hold data
    if (j < N) {
        T* row = A + (size_t)j * ld;
        double acc = 0.0;
        if (c.LT) {
            for (int k = 0; k < c.cols; k++) row[k] = k < N ? (T)c.LT[k * N + j] : (T)0;
            for (int k = 0; k < N; k++) acc = fma((double)c.LT[k * N + j], c.v[k], acc);
        } else {
            const T z4[4] = {(T)0, (T)0, (T)0, (T)0};
            for (int q = 0; q < q4; q++) st4(row + 4 * q, z4);
        }
        struct Op {
            double ks, ya, yb;
            int a, b;
        };
        cta_incidences(
            cnt, [&](double ks, int a, int b) { return Op{ks, c.v[a], c.v[b], a, b}; },
            [&](const Op& o, bool in) {
                const double sum = fma(o.ks * o.ya, o.yb, acc);
                acc = in ? sum : acc;
                // (padding goes to column N, which is set last)
                row[o.a] = (T)((double)row[o.a] + o.ks * o.yb);
                row[o.b] = (T)((double)row[o.b] + o.ks * o.ya);
            });
        c.f[j] = acc;
        if (j < 3) c.best[j] = 0ull;  // pivot-vote slots of the next LU
        const int qn = N >> 2;  // whole chunks of matrix columns
#pragma unroll 4
        for (int q = 0; q < qn; q++) {
            T a[4];
            ld4(row + 4 * q, a);
#pragma unroll
            for (int t = 0; t < 4; t++) a[t] = (T)((4 * q + t == j ? 1.0 : 0.0) - h * (double)a[t]);
            st4(row + 4 * q, a);
        }
        for (int cc = 4 * qn; cc < N; cc++) row[cc] = (T)((cc == j ? 1.0 : 0.0) - h * (double)row[cc]);
        row[N] = (T)acc;
    }
    __syncthreads();
}

// f_j for j = tid at the state in c.v, FP64 with fused multiply-adds (the
// mixed solver's right-hand side; the bit-exact evaluation is cta_rhs).
__device__ __forceinline__ void cta_rhs_fast(int cnt) {
    const CtaCtx& c = cta_ctx;
    const int N = c.N, j = (int)threadIdx.x;
    if (j < N) {
        double acc = 0.0;
        if (c.LT)
            for (int k = 0; k < N; k++) acc = fma((double)c.LT[k * N + j], c.v[k], acc);
        struct Op {
            double kya, yb;
        };
        cta_incidences(
            cnt, [&](double ks, int a, int b) { return Op{ks * c.v[a], c.v[b]}; },
            [&](const Op& o, bool in) {
                const double sum = fma(o.kya, o.yb, acc);
                acc = in ? sum : acc;
            });
        c.f[j] = acc;
    }
    __syncthreads();
}

// (J x)_j from the reactions (and L), FP64, for the refinement residual.
__device__ __forceinline__ double cta_jx(int j, const double* xv, int cnt) {
    const CtaCtx& c = cta_ctx;
    const int N = c.N;
    double acc = 0.0;
    if (c.LT)
        for (int k = 0; k < N; k++) acc = fma((double)c.LT[k * N + j], xv[k], acc);
    struct Op {
        double ks, d;
    };
    cta_incidences(
        cnt, [&](double ks, int a, int b) { return Op{ks, fma(c.v[b], xv[a], c.v[a] * xv[b])}; },
        [&](const Op& o, bool in) {
            const double sum = fma(o.ks, o.d, acc);
            acc = in ? sum : acc;
        });
    return acc;
}

// U12 = L11^-1 A12 for the 16 pivot rows of the panel at k0 (row offsets
// prow[]), one thread per column c0..N.
template <typename T>
__device__ __forceinline__ void cta_u12(T* A, int k0, const int (&prow)[CTA_NB]) {
    const CtaCtx& c = cta_ctx;
    const int N = c.N;
    for (int col = k0 + CTA_NB + (int)threadIdx.x; col <= N; col += cta_threads()) {
        T u[CTA_NB];
#pragma unroll
        for (int j = 0; j < CTA_NB; j++) u[j] = A[prow[j] + col];
#pragma unroll
        for (int i = 0; i < CTA_NB; i++) {
#pragma unroll
            for (int j = i + 1; j < CTA_NB; j++) u[j] = fma(-A[prow[j] + k0 + i], u[i], u[j]);
        }
#pragma unroll
        for (int j = 1; j < CTA_NB; j++) A[prow[j] + col] = u[j];
    }
}

// Trailing update A22 -= L21 U12 of the panel at k0: the active rows act[0..m)
// times columns c0..N, 4x4 register tiles with 16-byte vectors.
template <typename T>
__device__ __forceinline__ void cta_trailing(T* A, int k0, const int (&prow)[CTA_NB]) {
    const CtaCtx& c = cta_ctx;
    constexpr int TR = 4;
    const int N = c.N, ld = c.ld, c0 = k0 + CTA_NB;
    const int m = N - c0, n = N + 1 - c0;
    const int tr = (m + TR - 1) / TR, tc = (n + 3) >> 2;
    for (int t = (int)threadIdx.x; t < tr * tc; t += cta_threads()) {
        const int ti = t / tc, col = c0 + 4 * (t - ti * tc);
        int rows[TR];
#pragma unroll
        for (int r = 0; r < TR; r++) {
            const int rr = TR * ti + r;
            rows[r] = rr < m ? c.act[rr] * ld : -1;
        }
        T acc[TR][4];
#pragma unroll
        for (int r = 0; r < TR; r++) {
            if (rows[r] >= 0) ld4(A + rows[r] + col, acc[r]);
            else {
#pragma unroll
                for (int q = 0; q < 4; q++) acc[r][q] = (T)0;
            }
        }
#pragma unroll 1  // (full unrolling hoists every load and spills)
        for (int jc = 0; jc < CTA_NB / 4; jc++) {
            T u[4][4];
#pragma unroll
            for (int q = 0; q < 4; q++) ld4(A + prow[4 * jc + q] + col, u[q]);
#pragma unroll
            for (int r = 0; r < TR; r++) {
                T l[4] = {(T)0, (T)0, (T)0, (T)0};
                if (rows[r] >= 0) ld4(A + rows[r] + k0 + 4 * jc, l);
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int cc = 0; cc < 4; cc++) acc[r][cc] = fma(-l[q], u[q][cc], acc[r][cc]);
            }
        }
#pragma unroll
        for (int r = 0; r < TR; r++)
            if (rows[r] >= 0) st4(A + rows[r] + col, acc[r]);
    }
}

// Blocked right-looking LU with partial pivoting of [A | b] in place (see
// the file comment).  On return: c.piv[i] = physical row of logical row i,
// c.rinv[i] = 1/U_ii, the multipliers below the pivots, U above, and
// column N holds the forward-eliminated right-hand side.
template <typename T>
__device__ void cta_lu(T* A) {
    const CtaCtx& c = cta_ctx;
    const int N = c.N, tid = (int)threadIdx.x, ld = c.ld;
    const int warp = tid >> 5, lane = tid & 31;
    CtaCand<T>* cand = static_cast<CtaCand<T>*>(c.cand);
    T* myrow = A + (size_t)(tid < N ? tid : 0) * ld;
    bool done = tid >= N;  // row is a pivot row already (or no row)
    for (int k0 = 0; k0 < N; k0 += CTA_NB) {
        const int kb = min(CTA_NB, N - k0);
        const bool act0 = !done;
        T a[CTA_NB];
        if (act0) {
#pragma unroll
            for (int q = 0; q < CTA_NB / 4; q++) ld4at(myrow + k0 + 4 * q, a + 4 * q);
        } else {
#pragma unroll
            for (int q = 0; q < CTA_NB; q++) a[q] = (T)0;
        }
        // 1. panel factorisation, one barrier per column
#pragma unroll
        for (int j = 0; j < CTA_NB; j++) {
            if (j < kb) {
                // vote: each warp's best row publishes its panel entries and
                // its packed (key, row) into the step's 64-bit max slot
                const int g = k0 + j;  // global step: slots rotate mod 3
                const uint32_t key = done ? 0u : mag_key(a[j]) + 1u;
                const T myr = nr_rcp(a[j]);  // off the post-vote path
                const uint32_t wmax = __reduce_max_sync(0xffffffffu, key);
                const int wl = __ffs(__ballot_sync(0xffffffffu, key == wmax)) - 1;
                CtaCand<T>* slot = cand + (j & 1) * CTA_WARPS;
                if (lane == wl && wmax) {
                    slot[warp].rcp = myr;
#pragma unroll
                    for (int q = 0; q < CTA_NB / 4; q++)
                        st4at(slot[warp].vals + 4 * q, a + 4 * q);
                    atomicMax(c.best + g % 3, ((unsigned long long)wmax << 32) | (unsigned)(0xffff - tid));
                }
                __syncthreads();
                // the slot read two steps from now is cleared here: its last
                // readers passed this barrier, its writers have not started
                if (tid == 0) c.best[(g + 2) % 3] = 0ull;
                const int pr = 0xffff - (int)(c.best[g % 3] & 0xffffu);
                const CtaCand<T>& win = slot[pr >> 5];
                const T ri = win.rcp;
                if (tid == pr) {
                    done = true;
                    c.piv[k0 + j] = pr;
                    c.rinv[k0 + j] = (double)ri;
                } else if (!done) {
                    const T l = a[j] * ri;
                    a[j] = l;
#pragma unroll
                    for (int jj = j + 1; jj < CTA_NB; jj++) a[jj] = fma(-l, win.vals[jj], a[jj]);
                }
            }
        }
        if (act0) {
#pragma unroll
            for (int q = 0; q < CTA_NB / 4; q++) st4at(myrow + k0 + 4 * q, a + 4 * q);
        }
        // 2. compaction of the active rows (physical order)
        const unsigned am = __ballot_sync(0xffffffffu, !done);
        if (lane == 0) c.misc[warp] = __popc(am);
        __syncthreads();
        const int c0 = k0 + CTA_NB;  // first trailing column
        if (c0 > N) break;           // last panel: b was eliminated in registers
        if (!done) {
            int rank = __popc(am & ((1u << lane) - 1u));
            for (int w = 0; w < warp; w++) rank += c.misc[w];
            c.act[rank] = tid;
        }
        // 3. U12 = L11^-1 A12, one thread per column c0..N
        int prow[CTA_NB];
#pragma unroll
        for (int j = 0; j < CTA_NB; j++) prow[j] = c.piv[k0 + j] * ld;
        cta_u12<T>(A, k0, prow);
        __syncthreads();
        // 4. trailing update over act[0..m) x [c0, N]
        cta_trailing<T>(A, k0, prow);
        __syncthreads();
    }
}

// Triangular solves with the factors of cta_lu, on warp 0 alone: lane l
// owns logical rows l, l+32, ... (z in registers), column sweeps broadcast
// each finished value by shuffle -- no CTA barrier inside, one at the end.
//  REFINE = false: z_i = A[piv[i]][N] (already forward-eliminated), solve
//                  U x = z, write c.x;
//  REFINE = true:  z_i = c.r[piv[i]], solve L U dx = z, c.x += dx.
template <typename T, bool REFINE>
__device__ void cta_solve(const T* A) {
    const CtaCtx& c = cta_ctx;
    if ((int)threadIdx.x < 32) {
        const int N = c.N, lane = (int)threadIdx.x, ld = c.ld;
        constexpr int M = CTA_MAXN / 32;
        double z[M], xr[M];
        int rp[M];  // row offsets
#pragma unroll
        for (int m = 0; m < M; m++) {
            const int i = lane + 32 * m;
            const bool in = i < N;
            const int pr = c.piv[in ? i : 0];
            rp[m] = pr * ld;
            z[m] = in ? (REFINE ? c.r[pr] : (double)A[rp[m] + N]) : 0.0;
            xr[m] = 0.0;
        }
        if (REFINE) {
            // L z = z, unit lower: k = 0 .. N-2
#pragma unroll
            for (int b = 0; b < M; b++) {
                if (32 * b < N) {
                    const int kend = min(N - 1, 32 * b + 32);
                    T u[M];  // column k of my rows, loaded one step ahead
#pragma unroll
                    for (int m = b; m < M; m++) u[m] = A[rp[m] + 32 * b];
                    for (int k = 32 * b; k < kend; k++) {
                        T un[M];
                        const int kn = k + 1 < kend ? k + 1 : k;
#pragma unroll
                        for (int m = b; m < M; m++) un[m] = A[rp[m] + kn];
                        const double zk = __shfl_sync(0xffffffffu, z[b], k - 32 * b);
#pragma unroll
                        for (int m = b; m < M; m++) {
                            const int i = lane + 32 * m;
                            if (i > k && i < N) z[m] = fma(-(double)u[m], zk, z[m]);
                            u[m] = un[m];
                        }
                    }
                }
            }
        }
        // U x = z: k = N-1 .. 0
#pragma unroll
        for (int b = M - 1; b >= 0; b--) {
            if (32 * b < N) {
                const int ktop = min(N, 32 * b + 32) - 1;
                T u[M];  // column k of my rows, loaded one step ahead
#pragma unroll
                for (int m = 0; m <= b; m++) u[m] = A[rp[m] + ktop];
                for (int k = ktop; k >= 32 * b; k--) {
                    T un[M];
                    const int kn = k > 32 * b ? k - 1 : k;
#pragma unroll
                    for (int m = 0; m <= b; m++) un[m] = A[rp[m] + kn];
                    const double xk = __shfl_sync(0xffffffffu, z[b] * c.rinv[k], k - 32 * b);
                    xr[b] = (lane == k - 32 * b) ? xk : xr[b];  // kept by its owner, no branch
#pragma unroll
                    for (int m = 0; m <= b; m++) {
                        const int i = lane + 32 * m;
                        if (i < k) z[m] = fma(-(double)u[m], xk, z[m]);
                        u[m] = un[m];
                    }
                }
            }
        }
        double dxm = 0.0, xm = 0.0;
        bool finite = true;
#pragma unroll
        for (int m = 0; m < M; m++) {
            const int i = lane + 32 * m;
            if (i < N) {
                const double xn = REFINE ? c.x[i] + xr[m] : xr[m];
                c.x[i] = xn;
                dxm = fmax(dxm, fabs(xr[m]));
                xm = fmax(xm, fabs(xn));
                finite = finite && isfinite(xr[m]) && isfinite(xn);  // (fmax drops NaN)
            }
        }
        if (REFINE) {
            // converged: on every lane the last correction is finite and below
            // 1e-6 of the largest |x| among the lane's rows (l, l+32, ...) --
            // at least as strict as the same test over all rows
            int ok = finite && dxm <= 1e-6 * xm;
            ok = __all_sync(0xffffffffu, ok);
            if (lane == 0) c.misc[CTA_CONV] = ok;
        }
    }
    __syncthreads();
}

// ---- MIXED: FP32 Gauss-Jordan inverse reused across an attempt ----------
// CTA-wide max of |v| (one barrier).  `phase` rotates over three slots; the
// slot of the next call is cleared here -- its last readers read it two
// calls ago, before the barrier of the previous call.
__device__ __forceinline__ double cta_max_abs(double v, int& phase) {
    unsigned* slot = cta_ctx.maxima;
    const unsigned w = __reduce_max_sync(0xffffffffu, fmax_bits(v));
    if (((int)threadIdx.x & 31) == 0) atomicMax(slot + phase, w);
    if ((int)threadIdx.x == 0) slot[(phase + 1) % 3] = 0u;
    __syncthreads();
    const unsigned m = slot[phase];
    phase = (phase + 1) % 3;
    return (double)__uint_as_float(m);
}

// A[R][R] -= A[R][P] A[P][R] (P = panel [k0, k0+kb), R the other indices)
// over TR x 4 register tiles of the TR-row and 4-column chunks that miss P (k0 is
// a multiple of 16), for the chunks from row TR * rc0 on (0: every row; 128 / TR:
// the rows below those the tensor cores update).  Eight rows to a tile move 3
// bytes of shared memory per multiply-add where four moved 4; small matrices
// take two, so that every thread has a tile.
// FULL: kb = 16; otherwise the operands beyond kb are read as zeros (selected,
// not branched around: branches between the loads serialise their latencies).
template <bool FULL, int TR>
static __device__ __forceinline__ void cta_rank_update(float* A, int k0, int kb, int rc0) {
    const CtaCtx& c = cta_ctx;
    const int N = c.N, tid = (int)threadIdx.x, ld = c.ld;
    const int nch = (N + 3) >> 2, nrow = (N + TR - 1) / TR;
    const int pc0 = k0 >> 2, pc1 = (k0 + kb + 3) >> 2;             // column chunks touching P
    const int p0 = k0 / TR, p1 = (k0 + kb + TR - 1) / TR;          // row chunks touching P
    const int r_lo = p0 > rc0 ? p0 : rc0, r_hi = p1 > rc0 ? p1 : rc0;
    const int mr = (nrow - rc0) - (r_hi - r_lo);  // row chunks to update
    const int m4 = nch - (pc1 - pc0);             // column chunks outside P
    for (int t = tid; t < mr * m4; t += cta_threads()) {
        const int ti = t / m4, tj = t - ti * m4;
        const int ri = rc0 + ti < r_lo ? rc0 + ti : rc0 + ti + (r_hi - r_lo);
        const int col = 4 * (tj < pc0 ? tj : tj + (pc1 - pc0));
        const int i0 = TR * ri;
        int off[TR];  // rows past the last read that one again and are not stored
        float acc[TR][4];
#pragma unroll
        for (int r = 0; r < TR; r++) {
            off[r] = min(i0 + r, N - 1) * ld;
            ld4(A + off[r] + col, acc[r]);
        }
#pragma unroll 1
        for (int q0 = 0; q0 < CTA_NB; q0 += 4) {
            float u[4][4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const bool in = FULL || q0 + q < kb;
                ld4(A + (k0 + (in ? q0 + q : 0)) * ld + col, u[q]);
#pragma unroll
                for (int cc = 0; cc < 4; cc++) u[q][cc] = in ? u[q][cc] : 0.0f;
            }
#pragma unroll
            for (int r = 0; r < TR; r++) {
                float l[4];
                ld4(A + off[r] + k0 + q0, l);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float lq = FULL || q0 + q < kb ? l[q] : 0.0f;
#pragma unroll
                    for (int cc = 0; cc < 4; cc++) acc[r][cc] = fmaf(-lq, u[q][cc], acc[r][cc]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < TR; r++)
            if (i0 + r < N) st4(A + off[r] + col, acc[r]);
    }
}

// Step 3 of the blocked inverse on the tensor cores.  The rows [0, M) of
// A, M = min(N, 128), go into the tensor-memory accumulator (row i = lane i),
// one kind::tf32 MMA chain adds (-A[R][P]) (A[P][R]) with both operands split
// into TF32 high and low parts (hi*hi + hi*lo + lo*hi: FP32-level products,
// the 3xTF32 scheme), and the accumulator is copied back.  Rows of P and
// columns of P are zero in the operands, so they come back unchanged.  Rows
// [128, N) are updated on the CUDA cores while the MMAs run.  `par` is the
// mbarrier's phase parity, flipped once per panel.  A wait that runs out
// (it never should) leaves those rows un-updated: the inverse is then wrong,
// the refinement that uses it does not converge, and the substep goes to the
// pivoted recovery path (flagged WIND_SYS_REFINE_FALLBACK).
static __device__ __forceinline__ void cta_rank_update_tc(float* A, int k0, int kb,
                                                           uint32_t& par) {
    const CtaCtx& c = cta_ctx;
    const int N = c.N, tid = (int)threadIdx.x, ld = c.ld;
    const int M = N < 128 ? N : 128;
    const int cols16 = c.tc_cols16;
    const int w = tid >> 5, lane = tid & 31;
    const int sub = w & 3, half = w >> 2;          // two warps per lane quarter
    const int row = sub * 32 + lane;
    const uint32_t trow = c.tmem + ((uint32_t)(sub * 32) << 16);
    unsigned char* xs = c.tcs;                     // [hi s0 | hi s1 | lo s0 | lo s1], 4 KB each
    unsigned char* gs = c.tcs + 4 * 4096;          // same, cols16 * 32 B each
    const int gsl = cols16 * 32;
    // (a) rows [0, M) into the accumulator, 16 columns per store
    for (int c0 = half * 16; c0 < cols16; c0 += 32) {
        float v[16];
        const float* src = A + (size_t)(row < M ? row : 0) * ld + c0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            float a4[4];
            ld4(src + 4 * q, a4);
#pragma unroll
            for (int e = 0; e < 4; e++) v[4 * q + e] = row < M ? a4[e] : 0.0f;
        }
        tc::tmem_st16(trow + c0, v);
    }
    // (b) operands: X = -A[R][P] (rows < M), G = A[P][R] stored by output column
    for (int t = tid; t < 128 * CTA_NB; t += cta_threads()) {
        const int i = t >> 4, q = t & 15;
        float x = 0.0f;
        if (i < M && (i < k0 || i >= k0 + kb) && q < kb) x = -A[(size_t)i * ld + k0 + q];
        const float hi = tc::to_tf32(x), lo = tc::to_tf32(x - hi);
        const int off = (q >> 3) * 4096 + tc::slab_off(i, q & 7);
        *reinterpret_cast<float*>(xs + off) = hi;
        *reinterpret_cast<float*>(xs + 2 * 4096 + off) = lo;
    }
    for (int t = tid; t < cols16 * CTA_NB; t += cta_threads()) {
        const int j = t >> 4, q = t & 15;
        float g = 0.0f;
        if (j < N && (j < k0 || j >= k0 + kb) && q < kb) g = A[(size_t)(k0 + q) * ld + j];
        const float hi = tc::to_tf32(g), lo = tc::to_tf32(g - hi);
        const int off = (q >> 3) * gsl + tc::slab_off(j, q & 7);
        *reinterpret_cast<float*>(gs + off) = hi;
        *reinterpret_cast<float*>(gs + 2 * gsl + off) = lo;
    }
    tc::fence_smem_to_async();
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0) {
        tc::fence_after_sync();
        const uint32_t id = tc::idesc_tf32(128, cols16);
        for (int sl = 0; sl < 2 && 8 * sl < kb; sl++) {
            const uint64_t xh = tc::smem_desc(tc::smem_u32(xs + sl * 4096));
            const uint64_t xl = tc::smem_desc(tc::smem_u32(xs + (2 + sl) * 4096));
            const uint64_t gh = tc::smem_desc(tc::smem_u32(gs + sl * gsl));
            const uint64_t gl = tc::smem_desc(tc::smem_u32(gs + (2 + sl) * gsl));
            tc::mma_tf32(c.tmem, xh, gh, id, true);
            tc::mma_tf32(c.tmem, xh, gl, id, true);
            tc::mma_tf32(c.tmem, xl, gh, id, true);
        }
        tc::mma_commit(c.mbar);
    }
    // (c) rows [128, N) on the CUDA cores meanwhile
    if (N > 128) {
        if (kb == CTA_NB) cta_rank_update<true, 8>(A, k0, kb, 16);
        else cta_rank_update<false, 8>(A, k0, kb, 16);
    }
    // (d) the accumulator back into rows [0, M)
    bool ok = tc::mbar_wait(c.mbar, par, 1u << 24);
    ok = __all_sync(0xffffffffu, ok);
    par ^= 1u;
    tc::fence_after_sync();
    if (ok) {
        for (int c0 = half * 16; c0 < cols16; c0 += 32) {
            float v[16];
            tc::tmem_ld16(trow + c0, v);
            if (row < M) {
                float* dst = A + (size_t)row * ld + c0;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    float a4[4] = {v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]};
                    st4(dst + 4 * q, a4);
                }
            }
        }
    }
    tc::fence_before_sync();
}

// Unpivoted blocked Gauss-Jordan inversion of A (N x N, FP32, row stride
// c.ld, shared memory) in place.  Per panel P = [k0, k0+kb) with the other
// indices R = [0, N) \ P:
//  1. warp 0 inverts D = A[P][P] in registers (cta_gj_diag);
//  2. A[P][R] <- D^-1 A[P][R];
//  3. A[R][R] <- A[R][R] - A[R][P] A[P][R]   register tiles over the aligned
//     row and column chunks that miss P (the rank-kb update);
//  4. A[R][P] <- -A[R][P] D^-1, beside step 1 of the next panel on warp 0.
// Three CTA barriers per panel.  Steps 2 and 4 put four threads on a column
// (row), each with four of its 16 results.  Without pivoting the diagonal blocks
// must be invertible; a bad inverse shows up as a refinement that does not
// converge.  (FULL: a whole panel, kb = 16.  The SMEM variant's matrix is in
// shared memory, and its accesses are compiled as such.)
//
// With run-time panel widths tested around every load, steps 2 and 4 on one
// thread per column and four barriers this took 402,000 cycles at N = 157 (two
// blocks per SM) and 91,000 at N = 64.
//
// TC = true (the MIXED_TC solver) runs step 3 for the first 128 rows on the
// tensor cores (cta_rank_update_tc) and for the rows below them on the CUDA
// cores at the same time.

// D^-1 of the panel at k0, on one warp: element Gauss-Jordan, lanes 2i and
// 2i + 1 hold columns 0-7 and 8-15 of row i.
template <bool FULL>
static __device__ __forceinline__ void cta_gj_diag(float* A, int k0, int kb) {
    constexpr unsigned ALL = 0xffffffffu;
    const int ld = cta_ctx.ld, lane = (int)threadIdx.x & 31;
    const int row = lane >> 1, half = lane & 1;
    const bool mine = FULL || row < kb;
    float* src = A + (k0 + (mine ? row : 0)) * ld + k0 + 8 * half;
    float d[8];
    ld4at(src, d);
    ld4at(src + 4, d + 4);
#pragma unroll
    for (int q = 0; q < 8; q++)
        if (!mine || (!FULL && 8 * half + q >= kb)) d[q] = 0.0f;
#pragma unroll
    for (int k = 0; k < CTA_NB; k++) {
        if (FULL || k < kb) {
            const int kh = k >> 3, kq = k & 7;               // half and slot of column k
            const float r = nr_rcp(__shfl_sync(ALL, d[kq], 2 * k + kh));
            const float dk = __shfl_sync(ALL, d[kq], (lane & ~1) + kh);  // this row's entry
            const bool prow = row == k;
            const float f = prow ? 0.0f : dk * r;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const float pq = __shfl_sync(ALL, d[q], 2 * k + half);
                const float e = prow ? d[q] * r : fmaf(-f, pq, d[q]);
                d[q] = (q == kq && half == kh) ? (prow ? r : -f) : e;
            }
        }
    }
    if (mine) {
        if (FULL) {
            st4at(src, d);
            st4at(src + 4, d + 4);
        } else {
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (8 * half + q < kb) src[q] = d[q];
        }
    }
}

// Steps 2 to 4 of the panel at k0, and step 1 of the next one.
template <bool TC, bool FULL>
static __device__ __forceinline__ void cta_gj_panel(float* A, int k0, int kb, uint32_t& tc_par) {
    const CtaCtx& c = cta_ctx;
    const int N = c.N, tid = (int)threadIdx.x, ld = c.ld, warp = tid >> 5, lane = tid & 31;
    const int sub = lane & 7, q0 = 4 * (lane >> 3);
    // 2. row panel: a warp takes eight columns of R, eight lanes each result group
    for (int t0 = 8 * warp; t0 < N - kb; t0 += 8 * cta_warps()) {
        const int t = min(t0 + sub, N - kb - 1);
        const int j = t < k0 ? t : t + kb;
        float u[CTA_NB], acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int q = 0; q < CTA_NB; q++) {
            const bool in = FULL || q < kb;
            u[q] = A[(k0 + (in ? q : 0)) * ld + j];
            if (!in) u[q] = 0.0f;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float* drow = A + (k0 + (FULL || q0 + q < kb ? q0 + q : 0)) * ld + k0;
#pragma unroll
            for (int pp = 0; pp < CTA_NB; pp += 4) {
                float d[4];
                ld4(drow + pp, d);
#pragma unroll
                for (int e = 0; e < 4; e++) acc[q] = fmaf(FULL || pp + e < kb ? d[e] : 0.0f, u[pp + e], acc[q]);
            }
        }
        __syncwarp();  // the column is read by its four threads before it is replaced
#pragma unroll
        for (int q = 0; q < 4; q++)
            if ((FULL || q0 + q < kb) && t0 + sub < N - kb) A[(k0 + q0 + q) * ld + j] = acc[q];
    }
    __syncthreads();
    // 3. rank-kb update of R x R: on the tensor cores for the first 128
    //    rows (TC), on the CUDA cores for the rest
    if constexpr (TC) cta_rank_update_tc(A, k0, kb, tc_par);
    else if (N <= 96) cta_rank_update<FULL, 2>(A, k0, kb, 0);
    else cta_rank_update<FULL, 8>(A, k0, kb, 0);
    __syncthreads();
    // 1 of the next panel, and 4: column panel, a warp takes eight rows of R
    if (warp == 0 && k0 + CTA_NB < N) {
        if (N - k0 - CTA_NB >= CTA_NB) cta_gj_diag<true>(A, k0 + CTA_NB, CTA_NB);
        else cta_gj_diag<false>(A, k0 + CTA_NB, N - k0 - CTA_NB);
    }
    for (int t0 = 8 * (warp - 1); warp > 0 && t0 < N - kb; t0 += 8 * (cta_warps() - 1)) {
        const int t = min(t0 + sub, N - kb - 1);
        float* row = A + (t < k0 ? t : t + kb) * ld + k0;
        float l[CTA_NB], acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int q = 0; q < CTA_NB / 4; q++) ld4at(row + 4 * q, l + 4 * q);
#pragma unroll
        for (int q = 0; q < CTA_NB; q++)
            if (!FULL && q >= kb) l[q] = 0.0f;
#pragma unroll
        for (int q = 0; q < CTA_NB; q++) {
            float d[4];
            ld4(A + (k0 + (FULL || q < kb ? q : 0)) * ld + k0 + q0, d);
#pragma unroll
            for (int e = 0; e < 4; e++) acc[e] = fmaf(l[q], FULL || q < kb ? d[e] : 0.0f, acc[e]);
        }
        __syncwarp();  // the row is read by its four threads before it is replaced
        if (t0 + sub < N - kb) {
            if (FULL) {
                const float o[4] = {-acc[0], -acc[1], -acc[2], -acc[3]};
                st4(row + q0, o);
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (q0 + e < kb) row[q0 + e] = -acc[e];
            }
        }
    }
    __syncthreads();
}

template <bool TC, bool SMEM>
static __device__ __noinline__ void cta_gj_invert(float* A) {
    const CtaCtx& c = cta_ctx;
    if (SMEM) __builtin_assume(__isShared(A));
    const int N = c.N, tid = (int)threadIdx.x;
    if (tid < N) c.act[tid] = tid;   // row i expresses unknown i (no pivoting)
    uint32_t tc_par = TC ? (uint32_t)c.misc[CTA_TCPAR] : 0u;  // mbarrier phase parity
    int k0 = 0;
    if (tid < 32) cta_gj_diag<true>(A, 0, CTA_NB);  // (N > 32)
    __syncthreads();
    for (; k0 + CTA_NB <= N; k0 += CTA_NB) cta_gj_panel<TC, true>(A, k0, CTA_NB, tc_par);
    if (k0 < N) cta_gj_panel<TC, false>(A, k0, N - k0, tc_par);
    if (TC && tid == 0) c.misc[CTA_TCPAR] = (int)tc_par;
}

// A[i][j] += sum_k alpha_i^k w_j^k in step order over the rows i that are not
// pivots of the panel at k0 and the columns j outside it: the factors stand in
// A[i][k0..], the pivot-row values in rows c.piv[k0..].  8x4 register tiles over
// 4-aligned column chunks; a chunk or row that touches the panel is masked
// when it is stored.
static __device__ __forceinline__ void cta_gj_rows(float* A, int k0, int kb) {
    const CtaCtx& c = cta_ctx;
    constexpr int TR = 8;
    const int N = c.N, ld = c.ld;
    const int nch = (N + 3) >> 2, pc0 = k0 >> 2, pc1 = (k0 + kb + 3) >> 2;
    const int m4 = nch - (pc1 - pc0), tr = (N + TR - 1) / TR;
    for (int t = (int)threadIdx.x; t < tr * m4; t += cta_threads()) {
        const int ti = t / m4, tj = t - ti * m4;
        const int col = 4 * (tj < pc0 ? tj : tj + (pc1 - pc0));
        const int i0 = TR * ti;
        const float* rows = A + (size_t)i0 * ld;
        float acc[TR][4];
        unsigned skip = 0u;
#pragma unroll
        for (int r = 0; r < TR; r++) {
            const bool in = i0 + r < N;
            // pivots of the panel: steps k0 .. k0 + kb - 1
            if (!in || (unsigned)(c.act[i0 + r] - k0) < (unsigned)kb) skip |= 1u << r;
            if (in) ld4(rows + r * ld + col, acc[r]);
            else acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.0f;
        }
        if (skip == (1u << TR) - 1u) continue;
#pragma unroll 1
        for (int q0 = 0; q0 < kb; q0 += 4) {
            float u[4][4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (q0 + q < kb) ld4(A + (size_t)c.piv[k0 + q0 + q] * ld + col, u[q]);
                else u[q][0] = u[q][1] = u[q][2] = u[q][3] = 0.0f;
            }
#pragma unroll
            for (int r = 0; r < TR; r++) {
                float l[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (i0 + r < N) ld4(rows + r * ld + k0 + q0, l);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float lq = (q0 + q < kb) ? l[q] : 0.0f;
#pragma unroll
                    for (int cc = 0; cc < 4; cc++) acc[r][cc] = fmaf(lq, u[q][cc], acc[r][cc]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < TR; r++)
            if (!(skip >> r & 1u)) st4(A + (size_t)(i0 + r) * ld + col, acc[r]);
    }
}

// Gauss-Jordan inversion of A in place with partial pivoting and no row
// exchanges, for systems whose matrices the unpivoted elimination cannot
// handle (mass-action Jacobians are not diagonally dominant: a reaction
// A + B -> C + D puts +h k y_B in row B of column A).  Column k's pivot is
// the largest |a_ik| over the rows not yet chosen, voted CTA-wide as in
// cta_lu (warp reduce, packed 64-bit atomicMax, rotating slots).  Step k gives
// every row a factor alpha (r - 1 for the pivot row, r = 1/pivot, and -a_ik r
// for the others) and adds alpha times the pivot row to it, the chosen rows
// included.  On return row i expresses unknown c.act[i]: x_{act[i]} = sum_j
// M[i][j] b_{p_j} with p_j the row chosen at step j.
//
// Sixteen steps at a time:
//  1. panel: thread i holds row i's 16 panel entries in registers, one barrier
//     per step (the pivot candidates publish their entries); it keeps the
//     finished entries and leaves its 16 factors in their place;
//  2. every other column's 16 pivot-row values, each as it stands at its own
//     step, one thread per column, stored over the pivot rows;
//  3. the other rows: 16 multiply-adds per element over 8x4 register tiles;
//  4. the pivot rows, one thread per column, and the panel's finished entries.
// Every element gets the multiply-adds of the step-by-step elimination in its
// order, so the bits are the same; that one (two barriers per step, every
// thread updating its own row through shared memory) is what bounded systems
// at large step sizes.
template <bool SMEM>
static __device__ __noinline__ void cta_gj_invert_pivoted(float* A) {
    const CtaCtx& c = cta_ctx;
    if (SMEM) __builtin_assume(__isShared(A));
    const int N = c.N, tid = (int)threadIdx.x, ld = c.ld;
    const int warp = tid >> 5, lane = tid & 31;
    CtaCand<float>* cand = static_cast<CtaCand<float>*>(c.cand);
    float* myrow = A + (size_t)(tid < N ? tid : 0) * ld;
    const bool own = tid < N;
    bool done = !own;
    if (tid < 3) c.best[tid] = 0ull;
    if (own) c.act[tid] = -1;  // not chosen yet
    __syncthreads();
    for (int k0 = 0; k0 < N; k0 += CTA_NB) {
        const int kb = min(CTA_NB, N - k0);
        // 1. panel
        float a[CTA_NB];
        if (own) {
#pragma unroll
            for (int q = 0; q < CTA_NB / 4; q++) ld4at(myrow + k0 + 4 * q, a + 4 * q);
        } else {
#pragma unroll
            for (int q = 0; q < CTA_NB; q++) a[q] = 0.0f;
        }
#pragma unroll
        for (int j = 0; j < CTA_NB; j++) {
            if (j < kb) {
                const int g = k0 + j;
                const uint32_t key = done ? 0u : mag_key(a[j]) + 1u;
                const float myr = nr_rcp(a[j]);
                const uint32_t wmax = __reduce_max_sync(0xffffffffu, key);
                const int wl = __ffs(__ballot_sync(0xffffffffu, key == wmax)) - 1;
                CtaCand<float>* slot = cand + (j & 1) * CTA_WARPS;
                if (lane == wl && wmax) {
                    slot[warp].rcp = myr;
#pragma unroll
                    for (int q = 0; q < CTA_NB / 4; q++) st4at(slot[warp].vals + 4 * q, a + 4 * q);
                    atomicMax(c.best + g % 3, ((unsigned long long)wmax << 32) | (unsigned)(0xffff - tid));
                }
                __syncthreads();
                if (tid == 0) c.best[(g + 2) % 3] = 0ull;
                const int pr = 0xffff - (int)(c.best[g % 3] & 0xffffu);
                const CtaCand<float>& win = slot[pr >> 5];
                const float r = win.rcp;
                const bool mine = tid == pr;
                const float alpha = mine ? r - 1.0f : -a[j] * r;
#pragma unroll
                for (int q = 0; q < CTA_NB; q++)
                    if (q != j) a[q] = fmaf(alpha, win.vals[q], a[q]);
                a[j] = mine ? r : alpha;
                if (own) myrow[k0 + j] = alpha;
                if (mine) {
                    done = true;
                    c.act[tid] = g;
                    c.piv[g] = tid;
                }
            }
        }
        __syncthreads();
        // 2. pivot-row values of every other column at their own steps
        const int col = tid < k0 ? tid : tid + kb;
        if (tid < N - kb) {
            float w[CTA_NB];
#pragma unroll
            for (int j = 0; j < CTA_NB; j++) w[j] = j < kb ? A[(size_t)c.piv[k0 + j] * ld + col] : 0.0f;
#pragma unroll
            for (int j = 1; j < CTA_NB; j++) {
                if (j < kb) {
                    float* prow = A + (size_t)c.piv[k0 + j] * ld;
                    float al[CTA_NB];
#pragma unroll
                    for (int q = 0; q < j; q += 4) ld4at(prow + k0 + q, al + q);
#pragma unroll
                    for (int k = 0; k < j; k++) w[j] = fmaf(al[k], w[k], w[j]);
                    prow[col] = w[j];
                }
            }
        }
        __syncthreads();
        // 3. the rows that are not this panel's pivots
        cta_gj_rows(A, k0, kb);
        __syncthreads();
        // 4. the pivot rows' other columns, then the panel itself
        if (tid < N - kb) {
            float w[CTA_NB];
#pragma unroll
            for (int j = 0; j < CTA_NB; j++) w[j] = j < kb ? A[(size_t)c.piv[k0 + j] * ld + col] : 0.0f;
#pragma unroll
            for (int j = 0; j < CTA_NB; j++) {
                if (j < kb) {
                    float* prow = A + (size_t)c.piv[k0 + j] * ld;
                    float al[CTA_NB], acc = w[j];
#pragma unroll
                    for (int q = j & ~3; q < CTA_NB; q += 4) ld4at(prow + k0 + q, al + q);
#pragma unroll
                    for (int k = j; k < CTA_NB; k++)
                        if (k < kb) acc = fmaf(al[k], w[k], acc);
                    prow[col] = acc;
                }
            }
        }
        __syncthreads();
        if (own) {
#pragma unroll
            for (int q = 0; q < CTA_NB; q++)
                if (q < kb) myrow[k0 + q] = a[q];
        }
        // (the next panel's entries of a row are the thread's own, its columns
        // step 4's: the barrier above orders them)
    }
    __syncthreads();
}

// Row j of M times the FP32 vector qb (shared memory), four accumulators.
__device__ __forceinline__ double cta_apply_row(const float* mrow, const float* qb, int N) {
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
    const int n4 = N & ~3;
    for (int k = 0; k < n4; k += 4) {
        float a[4];
        ld4(mrow + k, a);
        const float4 b = *reinterpret_cast<const float4*>(qb + k);
        s0 = fmaf(a[0], b.x, s0);
        s1 = fmaf(a[1], b.y, s1);
        s2 = fmaf(a[2], b.z, s2);
        s3 = fmaf(a[3], b.w, s3);
    }
    for (int k = n4; k < N; k++) s0 = fmaf(mrow[k], qb[k], s0);
    return (double)((s0 + s1) + (s2 + s3));
}

enum { CTA_REFINE_OK = 0, CTA_REFINE_GAVE_UP = 1 };

// FP64 iterative refinement of (I - h J(v)) x = f (v in c.v, f in c.f)
// around the approximate inverse A: x = M f, then r = f - (x - h J x),
// x += M r.  Stop and give-up rules as the team kernel's (predicted error
// below 2^-33 max|x|; contraction worse than `abort0` on the first sweep or
// 1/2 later).  The result is left in c.x (natural order).  Uniform across
// the CTA.
template <bool SMEM>
static __device__ __noinline__ int cta_refine(const float* A, double h, int maxit, double abort0, int& phase,
                                              int cnt) {
    const CtaCtx& c = cta_ctx;
    if (SMEM) __builtin_assume(__isShared(A));
    const int N = c.N, j = (int)threadIdx.x, ld = c.ld;
    const bool own = j < N;
    // FP32 broadcast vector in the residual slot (c.r starts 32N bytes into
    // the 16-byte aligned vector block, so float4 reads of it are aligned).
    // Row j of the inverse gives unknown act[j]: right-hand sides are
    // scattered to qb[act[j]], results gathered through c.x[act[j]].
    float* qb = reinterpret_cast<float*>(c.r);
    const int sj = own ? c.act[j] : 0;
    if (own) qb[sj] = (float)c.f[j];
    __syncthreads();
    double xt = own ? cta_apply_row(A + (size_t)j * ld, qb, N) : 0.0;  // x_{act[j]}
    const double xmax = cta_max_abs(xt, phase);
    double dprev = 0.0;
    int outcome = CTA_REFINE_GAVE_UP;
    for (int it = 0; it < maxit; it++) {
        if (own) c.x[sj] = xt;
        __syncthreads();
        const double r = own ? c.f[j] - fma(-h, cta_jx(j, c.x, cnt), c.x[j]) : 0.0;
        if (own) qb[sj] = (float)r;
        __syncthreads();
        const double d = own ? cta_apply_row(A + (size_t)j * ld, qb, N) : 0.0;
        xt += d;
        const double dmax = cta_max_abs(d, phase);
        const double rho = (it == 0) ? dmax / fmax(xmax, 1e-300) : dmax / fmax(dprev, 1e-300);
        if (dmax * rho <= 0x1p-33 * xmax || dmax == 0.0) { outcome = CTA_REFINE_OK; break; }
        if (rho > (it == 0 ? abort0 : 0.5)) break;
        dprev = dmax;
    }
    if (own) c.x[sj] = xt;
    __syncthreads();
    return outcome;
}

// The substep solve with pivoting (FP32 LU with partial pivoting and up to
// two FP64 refinement sweeps): the recovery path when the Gauss-Jordan
// inverse does not refine.  Builds [I - hJ(v) | f] itself; result in c.x.
static __device__ __noinline__ void cta_mixed_pivoted_solve(double h, float* A, int cnt) {
    const CtaCtx& c = cta_ctx;
    const int tid = (int)threadIdx.x;
    const bool own = tid < c.N;
    cta_build<float, false>(h, A, cnt);
    cta_lu<float>(A);
    cta_solve<float, false>(A);
    for (int it = 0; it < 2; it++) {
        if (own) c.r[tid] = c.f[tid] - (c.x[tid] - h * cta_jx(tid, c.x, cnt));
        __syncthreads();
        cta_solve<float, true>(A);
        if (c.misc[CTA_CONV]) break;
    }
}

// The reference Gauss-Jordan inverse, CTA-parallel, on global scratch.
// M = I - hJt in the reference orientation (rows of Jt), Inv starts as I.
template <int CTRL>
__device__ void cta_gje_exact(double h, double* M, double* Inv) {
    const CtaCtx& c = cta_ctx;
    const int N = c.N, tid = (int)threadIdx.x;
    // build M; thread j owns column j (Jt[.][j] = d f_j / d y_.)
    for (int j = tid; j < N; j += cta_threads()) {
        for (int i = 0; i < N; i++) M[(size_t)i * N + j] = c.LT ? (double)c.LT[i * N + j] : 0.0;
        const int e0 = c.inc_off[j], e1 = c.inc_off[j + 1];
        for (int e = e0; e < e1; e++) {
            const int rr = c.inc[e];
            const uint2 q = *reinterpret_cast<const uint2*>(c.sp + 4 * rr);
            const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
            const xd k = c.rates[rr];
            const xd da = k * xd(c.v[b]), db = k * xd(c.v[a]);
            double* ra = M + (size_t)a * N + j;
            double* rb = M + (size_t)b * N + j;
            if (a == j) *ra = xd(*ra) - da;
            if (b == j) *ra = xd(*ra) - da;
            if (cc == j) *ra = xd(*ra) + da;
            if (d == j) *ra = xd(*ra) + da;
            if (a == j) *rb = xd(*rb) - db;
            if (b == j) *rb = xd(*rb) - db;
            if (cc == j) *rb = xd(*rb) + db;
            if (d == j) *rb = xd(*rb) + db;
        }
        for (int i = 0; i < N; i++) {
            double* m = M + (size_t)i * N + j;
            if (CTRL == WIND_CTRL_GOLD) {
                xd v = -xd(h) * xd(*m);
                if (i == j) v += 1.0;
                *m = v.v;
            } else {
                *m = (xd(i == j ? 1.0 : 0.0) - xd(*m) * xd(h)).v;
            }
            Inv[(size_t)i * N + j] = (i == j) ? 1.0 : 0.0;
        }
    }
    __syncthreads();
    // U phase (gje_gold.c:56-100)
    for (int i = 0; i < N; i++) {
        for (int k = i + 1 + tid; k < N; k += cta_threads()) c.scr[k] = M[(size_t)k * N + i];
        if (tid == 0) c.scr[i] = M[(size_t)i * N + i];
        __syncthreads();
        const xd s = c.scr[i];
        for (int t = tid; t < N; t += cta_threads()) {
            M[(size_t)i * N + t] = (xd(M[(size_t)i * N + t]) / s).v;
            Inv[(size_t)i * N + t] = (xd(Inv[(size_t)i * N + t]) / s).v;
        }
        __syncthreads();
        const int rows = N - 1 - i;
        for (int idx = tid; idx < rows * N; idx += cta_threads()) {
            const int k = i + 1 + idx / N, t = idx % N;
            const xd fct = c.scr[k];
            M[(size_t)k * N + t] = (xd(M[(size_t)k * N + t]) - fct * xd(M[(size_t)i * N + t])).v;
            Inv[(size_t)k * N + t] = (xd(Inv[(size_t)k * N + t]) - fct * xd(Inv[(size_t)i * N + t])).v;
        }
        __syncthreads();
    }
    // L phase, pivot rows bottom-up (gje_gold.c:102-134)
    for (int b = N - 1; b >= 0; b--) {
        for (int k = tid; k < b; k += cta_threads()) c.scr[k] = M[(size_t)k * N + b];
        __syncthreads();
        for (int idx = tid; idx < b * N; idx += cta_threads()) {
            const int k = idx / N, t = idx % N;
            const xd fct = c.scr[k];
            M[(size_t)k * N + t] = (xd(M[(size_t)k * N + t]) - fct * xd(M[(size_t)b * N + t])).v;
            Inv[(size_t)k * N + t] = (xd(Inv[(size_t)k * N + t]) - fct * xd(Inv[(size_t)b * N + t])).v;
        }
        __syncthreads();
    }
    for (int l = tid; l < N; l += cta_threads()) {
        if (CTRL == WIND_CTRL_GOLD) {
            // matrix_ops.c:6-27 then sie_gold.c:72-74
            xd out = 0.0;
            for (int k = 0; k < N; k++) out += xd(Inv[(size_t)k * N + l]) * xd(c.f[k]);
            c.v[l] = (xd(c.v[l]) + xd(h) * out).v;
        } else {
            // kernel.cu:121-125
            xd yl = c.v[l];
            for (int k = 0; k < N; k++) yl += xd(Inv[(size_t)k * N + l]) * xd(c.f[k]) * xd(h);
            c.v[l] = yl.v;
        }
    }
    __syncthreads();
}

// One substep of size h on c.v (in place): RK2, or SIE with an FP64 solve (MIXED
// works attempt by attempt, in cta_run).
template <int METHOD, int CTRL, int SOLVER>
__device__ void cta_substep(double h, void* mat, double* gM, int cnt) {
    static_assert(METHOD == WIND_METHOD_RK2 || SOLVER != WIND_SOLVER_MIXED, "MIXED has its own attempt");
    const CtaCtx& c = cta_ctx;
    const int N = c.N, tid = (int)threadIdx.x;
    const bool own = tid < N;
    if (METHOD == WIND_METHOD_RK2) {
        cta_rhs();
        if (own) c.v[tid] = (xd(c.v[tid]) + xd(h) * xd(c.f[tid])).v;
        __syncthreads();
        return;
    }
    if (SOLVER == WIND_SOLVER_GJE_F64) {
        cta_rhs();
        cta_gje_exact<CTRL>(h, gM, gM + (size_t)N * N);
        return;
    }
    double* A = static_cast<double*>(mat);
    cta_build<double, false>(h, A, cnt);
    cta_lu<double>(A);
    cta_solve<double, false>(A);
    if (own) c.v[tid] = c.v[tid] + h * c.x[tid];
    __syncthreads();
}

// The persistent CTA loop over one group's systems (blockDim.x a multiple of
// 32, at least N and at least 64; CTA_THREADS with TC).  `gscratch` holds one slot
// of `gstride` >= CtaLayout::g_doubles doubles per block (null when the layout
// needs none).
template <int METHOD, int CTRL, int SOLVER, bool TC>
__device__ __forceinline__ void cta_run(const KParams& p, unsigned char* smem_raw, double* gscratch,
                                        size_t gstride, int smem_cap) {
    constexpr int CAP = Cap<METHOD, CTRL>::value;
    const int N = p.n_eq, R = p.n_react, tid = threadIdx.x;
    const bool own = tid < N;
    const bool lin = p.linear != nullptr;
    const CtaLayout lay(N, R, lin, SOLVER, smem_cap, TC, METHOD == WIND_METHOD_SIE);
    CtaCtx& c = cta_ctx;
    double* gslot = gscratch ? gscratch + (size_t)blockIdx.x * gstride : nullptr;
    unsigned char* incbase = lay.inc_in_smem ? smem_raw + lay.inc_off
                                             : reinterpret_cast<unsigned char*>(gslot + lay.g_inc);
    int* inc_off = reinterpret_cast<int*>(incbase);
    uint16_t* inc = reinterpret_cast<uint16_t*>(incbase + CtaLayout::a16((N + 1) * 4));
    float* LT = lin ? reinterpret_cast<float*>(smem_raw + lay.lt) : nullptr;
    __syncthreads();  // (a block's previous group is done with the context)
    if (tid == 0) {
        double* vec = reinterpret_cast<double*>(smem_raw + lay.vec);
        c.N = N;
        c.R = R;
        c.ld = lay.ld;
        c.cols = lay.cols;
        c.v = vec;
        c.f = vec + N;
        c.x = c.r = c.rinv = c.scr = nullptr;
        if (SOLVER == WIND_SOLVER_GJE_F64) {
            c.scr = vec + 2 * N;
        } else {
            c.x = vec + 2 * N;
            c.rinv = vec + 3 * N;
            if (SOLVER == WIND_SOLVER_MIXED) c.r = vec + 4 * N;
        }
        c.piv = reinterpret_cast<int*>(smem_raw + lay.piv);
        c.act = reinterpret_cast<int*>(smem_raw + lay.act);
        c.misc = reinterpret_cast<int*>(smem_raw + lay.misc);
        c.best = reinterpret_cast<unsigned long long*>(smem_raw + lay.misc + 4 * CTA_WARPS);
        c.cand = smem_raw + lay.cand;
        c.inc_off = inc_off;
        c.inc = inc;
        c.LT = LT;
        c.tmem = 0;
        c.mbar = TC ? reinterpret_cast<uint64_t*>(smem_raw + lay.tcs) : nullptr;
        c.tcs = TC ? smem_raw + lay.tcs + 64 : nullptr;
        c.tc_cols16 = (N + 15) & ~15;
    }
    __syncthreads();
    double* gM = gslot;
    void* mat = lay.mat_in_smem ? (void*)(smem_raw + lay.mat) : (void*)(gslot + lay.g_mat);
    const uint64_t t_start = p.timeout_ns ? global_ns() : 0;
    __shared__ unsigned long long s_ticket;
    __shared__ int s_flag;
    // MIXED_TC: the accumulator's tensor-memory columns (a power of two
    // >= 32 covering the columns rounded to 16), held for the whole launch
    uint32_t tc_ncols = 32;
    if constexpr (TC) {
        while ((int)tc_ncols < c.tc_cols16) tc_ncols <<= 1;
        uint32_t* taddr = reinterpret_cast<uint32_t*>(smem_raw + lay.tcs + 8);
        if (tid < 32) tc::tmem_alloc(taddr, tc_ncols);
        if (tid == 0) {
            tc::mbar_init(c.mbar, 1);
            c.misc[CTA_TCPAR] = 0;
        }
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        if (tid == 0) c.tmem = *taddr;
        __syncthreads();
    }

    while (true) {
        if (tid == 0) s_ticket = atomicAdd(&p.counters[CNT_QUEUE], 1ull);
        __syncthreads();
        const int64_t s = (int64_t)s_ticket;
        if (s >= p.nsys) break;
        const double* rates = p.rates + s * R;
        const uint16_t* sp = p.species + (s * R) * 4;
        if (lay.data_in_smem) {
            double* srt = reinterpret_cast<double*>(smem_raw + lay.rt);
            uint2* ssp = reinterpret_cast<uint2*>(smem_raw + lay.spc);
            for (int r = tid; r < R; r += cta_threads()) {
                srt[r] = rates[r];
                ssp[r] = *reinterpret_cast<const uint2*>(sp + 4 * r);
            }
            rates = srt;
            sp = reinterpret_cast<const uint16_t*>(ssp);
        }
        if (tid == 0) {
            c.rates = rates;
            c.sp = sp;
        }
        // validate species indices, then build the per-species incidence lists
        if (tid == 0) s_flag = 0;
        __syncthreads();
        for (int r = tid; r < R; r += cta_threads()) {
            const uint2 q = *reinterpret_cast<const uint2*>(c.sp + 4 * r);
            const unsigned nn = (unsigned)N;
            if ((q.x & 0xffffu) >= nn || (q.x >> 16) >= nn || (q.y & 0xffffu) >= nn || (q.y >> 16) >= nn)
                s_flag = 1;
        }
        __syncthreads();
        const bool bad = s_flag != 0;
        if (!bad) {
            if (own) {
                int cnt = 0;
                for (int r = 0; r < R; r++) {
                    const uint2 q = *reinterpret_cast<const uint2*>(c.sp + 4 * r);
                    const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
                    cnt += (a == tid || b == tid || cc == tid || d == tid);
                }
                inc_off[tid + 1] = cnt;
            }
            __syncthreads();
            if (tid == 0) {
                inc_off[0] = 0;
                for (int j = 0; j < N; j++) inc_off[j + 1] += inc_off[j];
            }
            __syncthreads();
            if (own) {
                int o = inc_off[tid];
                for (int r = 0; r < R; r++) {
                    const uint2 q = *reinterpret_cast<const uint2*>(c.sp + 4 * r);
                    const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
                    if (a == tid || b == tid || cc == tid || d == tid) inc[o++] = (uint16_t)r;
                }
            }
            if (lin) {
                const float* Lg = p.linear + s * (int64_t)N * N;
                for (int idx = tid; idx < N * N; idx += cta_threads()) {
                    const int j = idx / N, k = idx % N;
                    LT[k * N + j] = Lg[idx];
                }
            }
        }
        // reaction records from the lists, where the launch has room for them
        int rec_cnt = 0;
        if constexpr (METHOD == WIND_METHOD_SIE && SOLVER != WIND_SOLVER_GJE_F64) {
            double* rk = nullptr;
            if (lay.rec_in_smem) rk = reinterpret_cast<double*>(smem_raw + lay.rec);
            else if (lay.rec_doubles && gslot && gstride >= lay.slot_doubles()) rk = gslot + lay.g_rec;
            auto each = [&](auto&& fn) {
                if (!own || bad) return;
                const int e1 = inc_off[tid + 1];
                for (int e = inc_off[tid]; e < e1; e++) {
                    const int rr = inc[e];
                    const uint2 q = *reinterpret_cast<const uint2*>(c.sp + 4 * rr);
                    const int a = q.x & 0xffff, b = q.x >> 16, cc = q.y & 0xffff, d = q.y >> 16;
                    const int sg = (cc == tid) + (d == tid) - (a == tid) - (b == tid);
                    if (sg) fn((double)sg * c.rates[rr], a, b);
                }
            };
            if (rk) {
                each([&](double, int, int) { rec_cnt++; });
                const int width = ((int)__reduce_max_sync(0xffffffffu, (unsigned)rec_cnt) + 3) & ~3;
                if ((tid & 31) == 0) c.rec_off[tid / 32 + 1] = width;
                __syncthreads();
                if (tid == 0) {
                    c.rec_off[0] = 0;
                    for (int w = 0; w < cta_warps(); w++) c.rec_off[w + 1] += c.rec_off[w];
                    const bool fits = c.rec_off[cta_warps()] * 32 <= lay.rec_cap;
                    c.rec_k = fits ? rk : nullptr;
                    c.rec_ab = reinterpret_cast<const uint32_t*>(rk + lay.rec_cap);
                }
                __syncthreads();
                if (c.rec_k) {
                    uint32_t* rab = reinterpret_cast<uint32_t*>(rk + lay.rec_cap);
                    size_t at = (size_t)c.rec_off[tid / 32] * 32 + (tid & 31);
                    each([&](double ks, int a, int b) {
                        rk[at] = ks;
                        rab[at] = (uint32_t)a | ((uint32_t)b << 16);
                        at += 32;
                    });
                    for (int e = rec_cnt; e < width; e++, at += 32) {
                        rk[at] = 0.0;
                        rab[at] = (uint32_t)N | ((uint32_t)N << 16);
                    }
                }
            } else if (tid == 0) {
                c.rec_k = nullptr;
            }
        }
        double yl = own ? p.y[s * N + tid] : 0.0, y1l = 0.0, y2l = 0.0;
        if (tid < 3) c.maxima[tid] = 0u;
        __syncthreads();

        double tnow = p.tnow;
        const double tend = p.tend;
        double h = p.h0;
        int unsolved = 0;
        int64_t attempts = 0;
        int32_t st = bad ? WIND_SYS_BAD_INPUT : WIND_SYS_OK;
        // MIXED: f(y) cached while y is unchanged; the matrix area holds the
        // inverse for the next full step; rotating max-slot phase
        bool fy_ok = false, inv_ok = false;
        double h_pivot = INFINITY;  // MIXED: fresh inverses at this step size and above pivot
        double fyl = 0.0;
        int phase = 0;
        // The first half step of a refined attempt, kept: it is the next
        // attempt's full step, bit for bit, when the two sizes are the same
        // number (same state, matrix and solve -- and, for MIXED, the same kind
        // of inverse: an unpivoted one must still be allowed at that size).
        double vh_keep = 0.0, h_vh = 0.0;
        bool vh_ok = false, vh_unpiv = false;
        while (!bad && tnow < tend) {
            if (attempts >= p.max_attempts) { st |= WIND_SYS_MAX_ATTEMPTS; break; }
            if (p.timeout_ns) {
                // thread 0's clock decides for the whole CTA
                if (__syncthreads_or(tid == 0 && global_ns() - t_start > p.timeout_ns)) {
                    st |= WIND_SYS_TIMEOUT;
                    break;
                }
            }
            attempts++;
            h = fmin(tend - tnow, h);
            const double t1 = tnow + h;
            if constexpr (METHOD == WIND_METHOD_SIE && SOLVER == WIND_SOLVER_MIXED) {
                // One FP32 Gauss-Jordan inverse serves the attempt: the
                // previous attempt's half-step inverse (same y, same size)
                // for the full step, a fresh one for the first half step,
                // reused for the second half step while it still contracts.
                // Fresh inverses are unpivoted (blocked, fast) below the
                // smallest step size at which an unpivoted one failed to
                // refine for this system, pivoted (column vote) at and above
                // it: the growth of the unpivoted elimination rises with h.
                // A fresh pivoted inverse that does not refine either (I - hJ
                // too ill-conditioned for FP32) leaves the substep to the FP32
                // LU recovery.  Any recovery flags the system
                // WIND_SYS_REFINE_FALLBACK.
                const double hf = t1 - tnow, h1 = (t1 - tnow) * 0.5;
                const double h2 = (CTRL == WIND_CTRL_DEVICE) ? fmin(t1 - (tnow + h1), h1) : h1;
                float* A = static_cast<float*>(mat);
                const bool smat = TC || lay.mat_in_smem;
                auto build = [&](double hh) {
                    if (smat) cta_build<float, true>(hh, A, rec_cnt);
                    else cta_build<float, false>(hh, A, rec_cnt);
                };
                auto refine = [&](double hh, int maxit, double abort0) {
                    return smat ? cta_refine<true>(A, hh, maxit, abort0, phase, rec_cnt)
                                : cta_refine<false>(A, hh, maxit, abort0, phase, rec_cnt);
                };
                // a fresh inverse of this substep's own matrix, and its solve
                auto fresh_solve = [&](double hh) {
                    build(hh);
                    if (hh < h_pivot) {
                        if (smat) cta_gj_invert<TC, true>(A);
                        else cta_gj_invert<false, false>(A);
                        if (refine(hh, 24, 1.0) == CTA_REFINE_OK) return true;
                        h_pivot = hh;
                        build(hh);
                    }
                    st |= WIND_SYS_REFINE_FALLBACK;
                    if (smat) cta_gj_invert_pivoted<true>(A);
                    else cta_gj_invert_pivoted<false>(A);
                    if (refine(hh, 24, 1.0) == CTA_REFINE_OK) return true;
                    cta_mixed_pivoted_solve(hh, A, rec_cnt);
                    return false;
                };
                if (own) c.v[tid] = yl;
                __syncthreads();
                if (!fy_ok) {
                    cta_rhs_fast(rec_cnt);
                    fyl = own ? c.f[tid] : 0.0;
                    fy_ok = true;
                } else {
                    if (own) c.f[tid] = fyl;
                    __syncthreads();
                }
                if (vh_ok && hf == h_vh && (!vh_unpiv || hf < h_pivot)) {
                    y1l = vh_keep;
                } else {
                    if (!inv_ok || refine(hf, 8, 0.5) != CTA_REFINE_OK) fresh_solve(hf);
                    y1l = own ? yl + hf * c.x[tid] : 0.0;
                }
                inv_ok = fresh_solve(h1);  // the inverse stays for the next full step
                const double vhl = own ? yl + h1 * c.x[tid] : 0.0;
                vh_keep = vhl;
                h_vh = h1;
                vh_unpiv = h1 < h_pivot;
                if (own) c.v[tid] = vhl;
                __syncthreads();
                cta_rhs_fast(rec_cnt);
                if (!inv_ok || refine(h2, 8, 0.0625) != CTA_REFINE_OK) {
                    fresh_solve(h2);
                    inv_ok = false;
                }
                y2l = own ? vhl + h2 * c.x[tid] : 0.0;
            } else
            for (int pass = 0; pass < 2; pass++) {
                const int nsub = pass + 1;
                if (own) c.v[tid] = yl;
                __syncthreads();
                // (t1-t0)/nsub, nsub in {1,2}: exact as a multiplication
                double hs = (t1 - tnow) * (nsub == 1 ? 1.0 : 0.5);
                double t = tnow;
                if (pass == 0 && vh_ok && (CTRL == WIND_CTRL_DEVICE ? fmin(t1 - t, hs) : hs) == h_vh) {
                    y1l = vh_keep;
                    continue;
                }
                for (int k = 0; k < nsub; k++) {
                    if (CTRL == WIND_CTRL_DEVICE) hs = fmin(t1 - t, hs);
                    cta_substep<METHOD, CTRL, SOLVER>(hs, mat, gM, rec_cnt);
                    t += hs;
                    if (pass == 1 && k == 0) {
                        vh_keep = own ? c.v[tid] : 0.0;
                        h_vh = hs;
                    }
                }
                if (own) {
                    if (pass == 0) y1l = c.v[tid];
                    else y2l = c.v[tid];
                }
            }
            const int e = own && elem_error<METHOD, CTRL>(xd(y1l), xd(y2l), p.atol, p.rtol) ? 1 : 0;
            const bool err = __syncthreads_or(e) != 0;
            if (err && unsolved < CAP) {
                unsolved++;
                h /= 2.0;
                vh_ok = true;
            } else {
                unsolved = 0;
                fy_ok = inv_ok = vh_ok = false;
                if (own) yl = (METHOD == WIND_METHOD_RK2) ? (xd(2.0) * xd(y2l) - xd(y1l)).v : y2l;
                if (tnow + h == tnow) { st |= WIND_SYS_STALLED; break; }
                tnow += h;
                h = (METHOD == WIND_METHOD_RK2) ? h * 2 : tend - tnow;
            }
        }
        int nonfinite = 0;
        if (own) {
            if (!finite64(yl)) nonfinite = 1;
            p.y[s * N + tid] = yl;
        }
        if (__syncthreads_or(nonfinite)) st |= WIND_SYS_NONFINITE;
        if (tid == 0) {
            if (p.sys_status) p.sys_status[s] = st;
            if (p.sys_nsteps) p.sys_nsteps[s] = 3 * attempts;
            atomicAdd(&p.counters[CNT_STEPS], (unsigned long long)(3 * attempts));
        }
        __syncthreads();
    }
    if constexpr (TC) {
        // every MMA was waited for; the columns go back before the CTA exits
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        if (tid < 32) tc::tmem_dealloc(c.tmem, tc_ncols);
    }
}

// Two CTAs per SM for the FP32 factors (the 157-species matrix is ~100 KB) and
// for RK2, whose registers would pass 128 otherwise (600 systems of 200 species:
// 8.3 ms with one, 4.7 ms with two).
#ifndef WIND_CTA_MIXED_BLOCKS
#define WIND_CTA_MIXED_BLOCKS 2
#endif
template <int METHOD, int SOLVER>
struct CtaMinBlocks {
    static constexpr int value = METHOD == WIND_METHOD_RK2          ? 2
                                 : SOLVER == WIND_SOLVER_MIXED ? WIND_CTA_MIXED_BLOCKS
                                                               : 1;
};

// TC = true: MIXED with the inverse's rank updates on the tensor cores
// (the MIXED_TC solver).
template <int METHOD, int CTRL, int SOLVER, bool TC = false>
__global__ void __launch_bounds__(CTA_THREADS, CtaMinBlocks<METHOD, SOLVER>::value)
    k_cta(const KParams p, double* gscratch, size_t gstride, int smem_cap) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cta_run<METHOD, CTRL, SOLVER, TC>(p, smem_raw, gscratch, gstride, smem_cap);
}

}  // namespace wind
