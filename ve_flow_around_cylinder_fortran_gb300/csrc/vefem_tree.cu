// Multifrontal elimination of the bordered Newton Jacobian over a nested
// dissection of the mesh: the Newton and continuation drivers' linear solver,
// in place of the MUMPS factorisation and solve behind KSPSolve
// (Petsc_mod.F90:850).
//
// The fronts are those of a complete binary tree of element sets (the
// package's dissection.py); front t is an n x n matrix with leading dimension
// ld (n rounded up to 4), its p pivots first.  All fronts of one depth are
// factorised together, deepest first:
//
//   k_assemble  M += the children's Schur complements (pulled entry by entry,
//               first child before second: no atomics, the same bits every run);
//   k_invert    per 32 pivots K: D^-1, D = M[K,K];
//   k_pivot     T = D^-1 M[K,:], and a copy of the columns C = M[P,K];
//   k_update    M[i,:] -= C_i T for the other pivot rows i (M[i,K] = -C_i D^-1),
//               M[K,:] = T: blocked Gauss-Jordan without pivoting on the pivot
//               rows only, which leaves M[P,P] = A^-1 and M[P,F] = X = A^-1 B;
//   k_schur     M[F,F] -= C X, for which k_split_inner and k_split_outer find
//               the exponents.
//
// What bounds it on GB300: on the FP64 pipe (2 multiply-adds per clock and SM,
// 0.63 T/s) the 50 G multiply-adds of 20,000 quads are 80 ms, so every product
// goes to the tensor cores in bf16 digits (vefem_split.cuh) and only the
// inversion of the 32 x 32 pivot blocks stays on that pipe.  What is left is the
// fixed cost of a tile in the deep levels and the chain of 133 steps near the
// root.  A sweep of element columns (vefem_frontal.cu) does 270 G multiply-adds
// in 30,600 dependent steps.  Eliminating the pivot rows only and leaving the
// Schur complement to one product is 18% fewer operations than Gauss-Jordan
// over the whole front.  Measured, factorise and solve, 20,000 and 2,000 quads:
// panels 1,185 and 89.9 ms; the tree on the FP64 pipe, 16 pivots a step, 127 and
// 10.6; Schur complements in digits 76 and 8.1; all products in digits, 32
// pivots a step, 55.8 and 7.0; with two short tiles to an SM and the pivot
// blocks inverted in registers 38.9 and 5.2; the kernels of a step started
// before the last one's end 38.0 and 4.7 (36.0 and 4.2 without the solve).  A
// sweep went from 21 to 1.31 ms at 20,000 (2,500 panels are 5,000 dependent
// launches, the tree 41).
//
// What one sweep leaves, 32 bordered Jacobians of 2,000 to 20,000 quads (Wi 0.1 to
// 0.6, two states each), eight right-hand sides each, geometric means against a
// solution refined in twice the precision: with the same elimination on the FP64
// pipe a residual of 3e-16 to 1e-13; with all products in digits 0.96 times that
// and 0.79 times its error in x; with the pivot blocks inverted in registers (one
// elimination of 32 pivots instead of two of 16) 1.06 and 1.11 times (at 20,000
// quads 0.82 and 1.95, single matrices up to 7 and 3.5 times).  Dividing by the
// pivots in full there gives 0.90 and 1.00 times for 4% to 11% more time, a step
// of Newton's iteration on the inverse 0.88 and 5 times.  The panels leave a
// residual of 3e-15 to 2e-11 and errors 0.6 to 35,000 times as large.
//
// Solve: per depth, deepest first, y_P = A^-1 b_P and the update -C y_P a
// front hands to its parent; then, root first, x_P = y_P - X x_F.  A row's dot
// product is spread over 8 lanes: with 32, the five shuffle additions per row
// cost more of the FP64 pipe than the products of a small front.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <numeric>
#include <string>
#include <vector>

#include "vefem.h"
#include "vefem_early.cuh"
#include "vefem_gj.cuh"
#include "vefem_split.cuh"

namespace {

struct Front {
    int64_t off;       // first entry of the matrix in the factor buffer
    int64_t cpan;      // first entry of the pivot-column copy (32 per pivot row)
    int64_t tpan;      // first entry of T (32 rows of ld)
    int32_t base;      // first entry of the front's unknowns, maps and vectors
    int32_t n, p, ld;
    int32_t child[2];  // front index, or -1
};

// ---------------------------------------------------------------- factorisation

// original entries into their fronts (every entry has a place of its own)
__global__ void k_scatter(int64_t nnz, const int64_t *__restrict__ dest, const double *__restrict__ vals,
                          double *__restrict__ buf)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nnz) buf[dest[i]] = vals[i];
}

constexpr int AS_ROWS = 8;
// M[i,j] += S_child0[src0[i], src0[j]], then the same for the second child
__global__ void __launch_bounds__(32 * AS_ROWS)
k_assemble(const Front *__restrict__ fr, const int32_t *__restrict__ perm, const int32_t *__restrict__ src0,
           const int32_t *__restrict__ src1, double *__restrict__ buf)
{
    const Front f = fr[perm[blockIdx.x]];
    const int i = blockIdx.y * AS_ROWS + threadIdx.y;
    if (i >= f.n) return;
    const int a0 = src0[f.base + i], a1 = src1[f.base + i];
    if (a0 < 0 && a1 < 0) return;
    const double *r0 = nullptr, *r1 = nullptr;
    if (a0 >= 0) r0 = buf + fr[f.child[0]].off + (int64_t)a0 * fr[f.child[0]].ld;
    if (a1 >= 0) r1 = buf + fr[f.child[1]].off + (int64_t)a1 * fr[f.child[1]].ld;
    double *m = buf + f.off + (int64_t)i * f.ld;
    for (int j = threadIdx.x; j < f.n; j += 32) {
        const int b0 = r0 ? src0[f.base + j] : -1, b1 = r1 ? src1[f.base + j] : -1;
        if (b0 < 0 && b1 < 0) continue;
        double v = m[j];
        if (b0 >= 0) v += r0[b0];
        if (b1 >= 0) v += r1[b1];
        m[j] = v;
    }
}

constexpr int KB = 2 * NB;   // pivots per step
constexpr int BATCH = 6;    // entries a thread of a product reads before it writes them back

// The inverse of D = M[K,K], K = [k0, k0 + kb), transposed to dinv: in-place
// Gauss-Jordan without pivoting, a CTA per front, thread = (column, four rows)
// with its entries in registers; the warp that holds the next pivot's row
// updates and divides it first and passes it on, with the pivot's column,
// through shared memory.  A pivot is measured against the largest entry of its
// 16 x 16 block as the block is reached.  Bound by the chain of 32 pivots, each
// four dependent FP64 instructions and a barrier (0.8 us), and where the fronts
// are many by the FP64 pipe (32^3 multiply-adds, 8.6 us on an SM); comparisons
// are made on the bit patterns, which order like the numbers, to keep them off
// that pipe.  In two blocked steps of 16 pivots with the division at each
// pivot: 8.2 ms of a factorisation of 20,000 quads, so 4.1.
constexpr int IV_THREADS = 8 * KB;
__global__ void __launch_bounds__(IV_THREADS)
k_invert(const Front *__restrict__ fr, const int32_t *__restrict__ perm, int k0, const double *buf, double *dinv,
         int *err, unsigned long long *minpiv, double tol)
{
    __shared__ double s_row[2][KB], s_col[2][KB], s_out[KB][KB + 1];
    __shared__ unsigned long long s_max[2];
    const Front f = fr[perm[blockIdx.x]];
    split::wait_previous();
    split::launch_next();
    const int kb = min(KB, f.p - k0), t = threadIdx.x, j = t & 31, g = t >> 5;
    const double *M = buf + f.off + (int64_t)k0 * f.ld + k0;
    constexpr unsigned long long MAGN = 0x7fffffffffffffffull, INF = 0x7ff0000000000000ull;
    auto magn = [](double x) { return (unsigned long long)__double_as_longlong(x) & MAGN; };
    double a[4];
#pragma unroll
    for (int u = 0; u < 4; u++) a[u] = (g * 4 + u < kb && j < kb) ? M[(int64_t)(g * 4 + u) * f.ld + j] : 0.0;
    if (t < 2) s_max[t] = 0;
    unsigned long long largest[2] = {INF, INF}, smallest[2] = {INF, INF}, floor_ = 0;
    bool bad = false;
    // row q (the warp's row u) divided by its pivot, and the pivot.  v / piv from
    // the hardware's reciprocal r (20 bits, e = 1 - piv r): v r (1 + e + e^2), the
    // next term is 2^-60; three dependent FP64 instructions.
    auto publish = [&](int q, int u) {
        const double piv = __shfl_sync(0xffffffffu, a[u], q), v = j == q ? 1.0 : a[u];
        if (plain_exponent(piv)) {
            const double r = approximate_reciprocal(piv), e = fma(-piv, r, 1.0), y = v * r;
            s_row[q & 1][j] = fma(y, fma(e, e, e), y);
        } else {
            s_row[q & 1][j] = v * (1.0 / piv);
        }
        if (j == q) s_col[q & 1][q] = piv;
    };
    if (g == 0) publish(0, 0);
    if (j == 0)
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (g * 4 + u != 0) s_col[0][g * 4 + u] = a[u];
    for (int p0 = 0; p0 < kb; p0 += 4) {
        if (p0 % NB == 0) {                            // a 16 x 16 block begins
            unsigned long long m = 0;
            if (g * 4 / NB == p0 / NB && j / NB == p0 / NB)
#pragma unroll
                for (int u = 0; u < 4; u++) m = max(m, magn(a[u]));
#pragma unroll
            for (int o = NB / 2; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
            __syncthreads();
            if (m && j % NB == 0) atomicMax(&s_max[p0 / NB], m);
            __syncthreads();
            m = s_max[p0 / NB];
            largest[p0 / NB] = m;
            floor_ = magn(tol * __longlong_as_double((long long)m));
            bad = bad || m == 0 || m >= INF;
        }
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const int p = p0 + w, q = p + 1;
            if (p >= kb) break;
            const int b = w & 1, un = (w + 1) & 3;     // row q is its warp's row un
            __syncthreads();
            const double v = s_row[b][j];
            // the next pivot's row first, so that its reciprocal's chain runs
            // beside the other rows' updates
            const bool next = q < kb && g == q / 4;
            if (next) {
                a[un] = fma(-s_col[b][q], v, j == p ? 0.0 : a[un]);
                publish(q, un);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int r = g * 4 + u;
                if (!(next && u == un)) a[u] = r == p ? v : fma(-s_col[b][r], v, j == p ? 0.0 : a[u]);
            }
            if (j == q)
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (g * 4 + u != q) s_col[b ^ 1][g * 4 + u] = a[u];
            const unsigned long long piv = magn(s_col[b][p]);
            smallest[p0 / NB] = min(smallest[p0 / NB], piv);
            bad = bad || piv <= floor_ || piv >= INF;
        }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) s_out[g * 4 + u][j] = a[u];
    __syncthreads();
    double *D = dinv + (int64_t)blockIdx.x * KB * KB;
#pragma unroll
    for (int k = g; k < KB; k += 8) D[k * KB + j] = (k < kb && j < kb) ? s_out[j][k] : 0.0;
    if (t == 0) {
        if (bad) atomicCAS(err, 0, 1);
        for (int h = 0; h * NB < kb && !bad; h++)
            atomic_min_pos(minpiv, __longlong_as_double((long long)smallest[h]) / __longlong_as_double((long long)largest[h]));
    }
}

// T = D^-1 M[K,:] for 128 columns, as the product of M[K,:]^T and D^-T; columns
// K of T hold D^-1.  And 128 rows of the copy C = M[P,K].  Starts while k_invert
// runs, whose blocks have all waited for the kernel before it: M is as that one
// left it, and is read with load_early (vefem_early.cuh), which costs no more
// than plain loads (4.18 and 35.9 ms per factorisation of 2,000 and 20,000 quads
// with either; 4.37 and 36.4 with all loads after the wait).  D^-1 is read after
// the wait.
__global__ void __launch_bounds__(split::THREADS, 2)
k_pivot(const Front *__restrict__ fr, const int32_t *__restrict__ perm, int k0, const double *buf,
        const double *dinv, double *__restrict__ cpan, double *__restrict__ tpan, int *err)
{
    extern __shared__ __align__(1024) char s_stage[];
    split::launch_next();
    const Front f = fr[perm[blockIdx.x]];
    const int j0 = blockIdx.y * split::TM;
    if (j0 >= f.n) return;
    const int kb = min(KB, f.p - k0), t = threadIdx.x;
    const double *M = buf + f.off, *D = dinv + (int64_t)blockIdx.x * KB * KB;
#pragma unroll 8
    for (int u = t; u < split::TM * KB; u += split::THREADS) {
        const int r = j0 + u / KB, l = u % KB;
        if (r < f.p) cpan[f.cpan + (int64_t)r * KB + l] = l < kb ? load_early(M + (int64_t)r * f.ld + k0 + l) : 0.0;
    }
    const int m = min(split::TM, f.n - j0);
    const bool ok = split::short_product<KB, true>(
        s_stage, m, kb,
        [&](int j, int k, double (&x)[8]) {
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (k + u < kb) x[u] = load_early(M + (int64_t)(k0 + k + u) * f.ld + j0 + j);
        },
        [&](int r, int k, double (&y)[8]) {
#pragma unroll
            for (int u = 0; u < 8; u++) y[u] = D[(k + u) * KB + r];
        },
        [] { split::wait_previous(); });
    if (!ok) {
        if (t == 0) atomicExch(err, 2);
        return;
    }
    const double *out = reinterpret_cast<const double *>(s_stage);
    for (int u = t; u < KB * split::TM; u += split::THREADS) {
        const int r = u / split::TM, c = u % split::TM, j = j0 + c;
        if (r < kb && c < m)
            tpan[f.tpan + (int64_t)r * f.ld + j] = j >= k0 && j < k0 + kb ? D[(j - k0) * KB + r] : out[c * (KB + 1) + r];
    }
}

// M[i,:] -= C_i T for the pivot rows outside K, M[K,:] = T (in place: C and T
// are copies, an entry is read and written by its own thread)
__global__ void __launch_bounds__(split::THREADS, 2)
k_update(const Front *__restrict__ fr, const int32_t *__restrict__ perm, int k0, int ntc,
         const double *cpan, const double *tpan, double *buf, int *err)
{
    extern __shared__ __align__(1024) char s_stage[];
    split::launch_next();
    const Front f = fr[perm[blockIdx.x]];
    const int i0 = (blockIdx.y / ntc) * split::TM, j0 = (blockIdx.y % ntc) * split::TN;
    if (i0 >= f.p || j0 >= f.n) return;
    split::wait_previous();
    const int kb = min(KB, f.p - k0), t = threadIdx.x;
    const int m = min(split::TM, f.p - i0), n = min(split::TN, f.n - j0);
    const double *C = cpan + f.cpan + (int64_t)i0 * KB, *T = tpan + f.tpan + j0;
    const bool copy = i0 >= k0 && i0 + m <= k0 + kb;  // only rows K
    if (!copy && !split::short_product<split::TN, false>(
                     s_stage, m, n,
                     [&](int r, int k, double (&x)[8]) {
                         if (i0 + r >= k0 && i0 + r < k0 + kb) return;
#pragma unroll
                         for (int u = 0; u < 8; u += 2) {
                             const double2 v = *reinterpret_cast<const double2 *>(C + r * KB + k + u);
                             x[u] = v.x;
                             x[u + 1] = v.y;
                         }
                     },
                     [&](int c, int k, double (&y)[8]) {
#pragma unroll
                         for (int u = 0; u < 8; u++)
                             if (k + u < kb) y[u] = T[(int64_t)(k + u) * f.ld + c];
                     },
                     [] {})) {
        if (t == 0) atomicExch(err, 2);
        return;
    }
    const double *out = reinterpret_cast<const double *>(s_stage);
    double *A = buf + f.off + (int64_t)i0 * f.ld + j0;
    for (int u0 = t; u0 < m * split::TN; u0 += BATCH * split::THREADS) {
        double v[BATCH];
#pragma unroll
        for (int h = 0; h < BATCH; h++) {
            const int u = u0 + h * split::THREADS, r = u / split::TN, c = u % split::TN, i = i0 + r, j = j0 + c;
            v[h] = 0.0;
            if (r >= m || c >= n) continue;
            if (i >= k0 && i < k0 + kb)
                v[h] = T[(int64_t)(i - k0) * f.ld + c];
            else if (j < k0 || j >= k0 + kb)
                v[h] = A[(int64_t)r * f.ld + c];
        }
#pragma unroll
        for (int h = 0; h < BATCH; h++) {
            const int u = u0 + h * split::THREADS, r = u / split::TN, c = u % split::TN, i = i0 + r;
            if (r >= m || c >= n) continue;
            A[(int64_t)r * f.ld + c] = i >= k0 && i < k0 + kb ? v[h] : v[h] - out[r * split::OUT_LD + c];
        }
    }
}

// Scaling of the split product: the power of two that evens row k of X (e0 at
// the pivots' places); then, per 32 boundary unknowns, the largest exponent of
// their row of C (e0) and column of X (e1).
__global__ void __launch_bounds__(256)
k_split_inner(const Front *__restrict__ fr, const int32_t *__restrict__ perm, const double *__restrict__ buf,
              int32_t *__restrict__ e0)
{
    const Front f = fr[perm[blockIdx.x]];
    const int k0 = blockIdx.y * 32, x = threadIdx.x & 31;
    for (int r = k0 + (threadIdx.x >> 5); r < min(k0 + 32, f.p); r += 8) {
        const double *row = buf + f.off + (int64_t)r * f.ld;
        int b = 0;
        for (int j = f.p + x; j < f.n; j += 32) b = max(b, split::finite_high(row[j]));
        b = __reduce_max_sync(0xffffffffu, b);
        if (x == 0) e0[f.base + r] = split::inner_exponent(b);
    }
}

__global__ void __launch_bounds__(256)
k_split_outer(const Front *__restrict__ fr, const int32_t *__restrict__ perm, const double *__restrict__ buf, int32_t *e0,
              int32_t *__restrict__ e1)
{
    __shared__ int s_b[8][32];
    const Front f = fr[perm[blockIdx.x]];
    const int i0 = blockIdx.y * 32, q = f.n - f.p;
    if (i0 >= q) return;
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const double *M = buf + f.off;
    const int32_t *sk = e0 + f.base;
    for (int r = y; r < 32 && i0 + r < q; r += 8) {
        const double *row = M + (int64_t)(f.p + i0 + r) * f.ld;
        int a = split::EMPTY;
        for (int k = x; k < f.p; k += 32) a = max(a, split::scaled_exponent(row[k], sk[k]));
        a = __reduce_max_sync(0xffffffffu, a);
        if (x == 0) e0[f.base + f.p + i0 + r] = a;
    }
    int b = split::EMPTY;
    if (i0 + x < q)
        for (int k = y; k < f.p; k += 8) b = max(b, split::scaled_exponent(M[(int64_t)k * f.ld + f.p + i0 + x], -sk[k]));
    s_b[y][x] = b;
    __syncthreads();
    if (y == 0 && i0 + x < q) {
#pragma unroll
        for (int r = 1; r < 8; r++) b = max(b, s_b[r][x]);
        e1[f.base + f.p + i0 + x] = b;
    }
}

// M[F,F] -= M[F,P] M[P,F], for every p: fronts with fewer than 16, 32 or 64
// pivots left to a tiled FP64 product made 20,000 quads 0.2, 2.1 and 9.4 ms
// slower.  Two stages for fronts of more than EXACT_K pivots, whose sums are
// emptied into registers; one for the others: 43.5 ms with two stages for all,
// 40.6 with the line at 64, 40.0 at 128.
template <int BUFFERS>
__global__ void __launch_bounds__(split::THREADS, 3 - BUFFERS)
k_schur(const Front *__restrict__ fr, const int32_t *__restrict__ perm, int ntc, const int32_t *__restrict__ e0,
        const int32_t *__restrict__ e1, double *__restrict__ buf, int *err)
{
    extern __shared__ __align__(1024) char s_stage[];
    const Front f = fr[perm[blockIdx.x]];
    const int q = f.n - f.p;
    const int i0 = (blockIdx.y / ntc) * split::TM, j0 = (blockIdx.y % ntc) * split::TN;
    if (i0 >= q || j0 >= q || f.p == 0) return;
    double *M = buf + f.off;
    split::Operands o;
    o.a = M + (int64_t)(f.p + i0) * f.ld;
    o.b = M + f.p + j0;
    o.lda = o.ldb = f.ld;
    o.m = min(q - i0, split::TM);
    o.n = min(q - j0, split::TN);
    o.k = f.p;
    o.s = e0 + f.base;
    o.ta = e0 + f.base + f.p + i0;
    o.tb = e1 + f.base + f.p + j0;
    if (!split::product<BUFFERS>(s_stage, o)) {
        if (threadIdx.x == 0) atomicExch(err, 2);
        return;
    }
    const double *out = reinterpret_cast<const double *>(s_stage);
    double *S = M + (int64_t)(f.p + i0) * f.ld + f.p + j0;
    for (int u0 = threadIdx.x; u0 < o.m * split::TN; u0 += BATCH * split::THREADS) {
        double v[BATCH];
#pragma unroll
        for (int h = 0; h < BATCH; h++) {
            const int u = u0 + h * split::THREADS, r = u / split::TN, c = u % split::TN;
            v[h] = r < o.m && c < o.n ? S[(int64_t)r * f.ld + c] : 0.0;
        }
#pragma unroll
        for (int h = 0; h < BATCH; h++) {
            const int u = u0 + h * split::THREADS, r = u / split::TN, c = u % split::TN;
            if (r < o.m && c < o.n) S[(int64_t)r * f.ld + c] = v[h] - out[r * split::OUT_LD + c];
        }
    }
}

// ---------------------------------------------------------------- solve

constexpr int SV_THREADS = 256;
constexpr int SV_LANES = 8;                            // lanes per row
constexpr int SV_ROWS = SV_THREADS / SV_LANES;         // rows per pass of a CTA

// dot product of a row with the staged vector over 8 lanes (fixed order)
__device__ __forceinline__ double row_dot(const double *__restrict__ row, const double *s_vec, int m, int lane)
{
    double s = 0.0;
#pragma unroll 4
    for (int k = lane; k < m; k += SV_LANES) s = fma(row[k], s_vec[k], s);
#pragma unroll
    for (int o = SV_LANES / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// what the children hand to position j of front f
__device__ __forceinline__ double handed(const Front &f, const Front *__restrict__ fr, int j,
                                         const int32_t *__restrict__ src0, const int32_t *__restrict__ src1,
                                         const double *__restrict__ y)
{
    double v = 0.0;
    const int a0 = src0[f.base + j], a1 = src1[f.base + j];
    if (a0 >= 0) v += y[fr[f.child[0]].base + a0];
    if (a1 >= 0) v += y[fr[f.child[1]].base + a1];
    return v;
}

// y_P = A^-1 (b_P + handed)
__global__ void __launch_bounds__(SV_THREADS)
k_tree_fwd(const Front *__restrict__ fr, const int32_t *__restrict__ perm, int rows, const int32_t *__restrict__ ids,
           const int32_t *__restrict__ src0, const int32_t *__restrict__ src1, const double *__restrict__ buf,
           const double *__restrict__ b, double *__restrict__ y)
{
    extern __shared__ double s_vec[];
    const Front f = fr[perm[blockIdx.x]];
    const int r0 = blockIdx.y * rows, r1 = min(r0 + rows, f.p);
    if (r0 >= f.p) return;
    for (int j = threadIdx.x; j < f.p; j += SV_THREADS)
        s_vec[j] = b[ids[f.base + j]] + handed(f, fr, j, src0, src1, y);
    __syncthreads();
    const int lane = threadIdx.x % SV_LANES;
    for (int rr = r0; rr < r1; rr += SV_ROWS) {
        const int r = rr + threadIdx.x / SV_LANES;
        const double s = row_dot(buf + f.off + (int64_t)min(r, f.p - 1) * f.ld, s_vec, f.p, lane);
        if (r < r1 && lane == 0) y[f.base + r] = s;
    }
}

// the update for the parent: handed - C y_P
__global__ void __launch_bounds__(SV_THREADS)
k_tree_up(const Front *__restrict__ fr, const int32_t *__restrict__ perm, int rows, const int32_t *__restrict__ src0,
          const int32_t *__restrict__ src1, const double *__restrict__ buf, double *__restrict__ y)
{
    extern __shared__ double s_vec[];
    const Front f = fr[perm[blockIdx.x]];
    const int r0 = f.p + blockIdx.y * rows, r1 = min(r0 + rows, f.n);
    if (r0 >= f.n) return;
    for (int j = threadIdx.x; j < f.p; j += SV_THREADS) s_vec[j] = y[f.base + j];
    __syncthreads();
    const int lane = threadIdx.x % SV_LANES;
    for (int rr = r0; rr < r1; rr += SV_ROWS) {
        const int r = rr + threadIdx.x / SV_LANES;
        const double s = row_dot(buf + f.off + (int64_t)min(r, f.n - 1) * f.ld, s_vec, f.p, lane);
        if (r < r1 && lane == 0) y[f.base + r] = handed(f, fr, r, src0, src1, y) - s;
    }
}

// x_P = y_P - X x_F
__global__ void __launch_bounds__(SV_THREADS)
k_tree_bwd(const Front *__restrict__ fr, const int32_t *__restrict__ perm, int rows, const int32_t *__restrict__ ids,
           const double *__restrict__ buf, const double *__restrict__ y, double *__restrict__ x)
{
    extern __shared__ double s_vec[];
    const Front f = fr[perm[blockIdx.x]];
    const int r0 = blockIdx.y * rows, r1 = min(r0 + rows, f.p);
    if (r0 >= f.p) return;
    const int q = f.n - f.p;
    for (int j = threadIdx.x; j < q; j += SV_THREADS) s_vec[j] = x[ids[f.base + f.p + j]];
    __syncthreads();
    const int lane = threadIdx.x % SV_LANES;
    for (int rr = r0; rr < r1; rr += SV_ROWS) {
        const int r = rr + threadIdx.x / SV_LANES;
        const double s = row_dot(buf + f.off + (int64_t)min(r, f.p - 1) * f.ld + f.p, s_vec, q, lane);
        if (r < r1 && lane == 0) x[ids[f.base + r]] = y[f.base + r] - s;
    }
}

struct Guard {
    int prev = -1;
    explicit Guard(int d)
    {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        cudaSetDevice(d);
    }
    ~Guard()
    {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

struct Level {
    int first, count;           // fronts, and their places in perm (most pivots first)
    int nmax, pmax, qmax, ldmax;
    std::vector<int> active;    // fronts with more than 32 s pivots, per step s
    std::vector<int> ld_active; // largest leading dimension among them
    int many;                   // fronts whose Schur product is a long one
};

}  // namespace

struct vefem_tree {
    int device = 0, nfront = 0, sms = 0;
    int64_t N = 0, total = 0, buf_len = 0;  // buf_len: doubles that the fronts take
    std::vector<Level> levels;
    int pmax = 0, qmax = 0;
    Front *fr = nullptr;
    int32_t *perm = nullptr, *ids = nullptr, *src0 = nullptr, *src1 = nullptr;
    int32_t *e0 = nullptr, *e1 = nullptr;   // exponents of the split products
    double *cpan = nullptr, *tpan = nullptr, *dinv = nullptr;
    double *y = nullptr, *b = nullptr, *x = nullptr;
    int *err = nullptr;
    unsigned long long *minpiv = nullptr;
    unsigned long long h_one = 0;      // staging of the initial minimum (outlives the async copy)
    cudaStream_t cs = nullptr;
    cudaGraphExec_t graph = nullptr;   // the sweeps of a solve, captured per factor buffer
    const double *graph_buf = nullptr;
    std::string msg;
};

namespace {

int tfail(vefem_tree *f, int code, const std::string &m)
{
    if (f) f->msg = m;
    return code;
}

#define TCK(call)                                                                        \
    do {                                                                                 \
        cudaError_t _e = (call);                                                         \
        if (_e != cudaSuccess)                                                           \
            return tfail(f, VEFEM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(_e)); \
    } while (0)

unsigned up(int a, int b) { return (unsigned)((a + b - 1) / b); }

// programmatic launch: the kernel starts when every block of the one before it
// has let it, and waits itself for what it reads
template <class... P, class... A>
cudaError_t launch_early(void (*kernel)(P...), dim3 grid, int threads, int smem, cudaStream_t s, A... args)
{
    cudaLaunchAttribute early[1];
    early[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cfg.attrs = early;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Rows per CTA of a sweep launch: one pass of its 32 groups of lanes, unless
// that makes more than 32 CTAs an SM.  A pass is mostly the latency of its rows'
// loads: with passes in turn wherever the fronts fill the GPU twice a sweep of
// 20,000 quads took 1.49 ms, of 2,000 0.33, now 1.31 and 0.27.
int rows_per_cta(const vefem_tree *f, int fronts, int rmax)
{
    const int parts = std::max(1, 32 * f->sms / fronts);
    return std::max(SV_ROWS, (int)up((int)up(rmax, parts), SV_ROWS) * SV_ROWS);
}

cudaError_t launch_sweeps(vefem_tree *f, const double *buf, cudaStream_t s)
{
    for (const Level &l : f->levels) {
        const int32_t *perm = f->perm + l.first;
        const size_t sm = (size_t)std::max(1, l.pmax) * sizeof(double);
        if (l.pmax > 0) {
            const int r = rows_per_cta(f, l.count, l.pmax);
            k_tree_fwd<<<dim3(l.count, up(l.pmax, r)), SV_THREADS, sm, s>>>(f->fr, perm, r, f->ids, f->src0, f->src1,
                                                                           buf, f->b, f->y);
        }
        if (l.qmax > 0) {
            const int r = rows_per_cta(f, l.count, l.qmax);
            k_tree_up<<<dim3(l.count, up(l.qmax, r)), SV_THREADS, sm, s>>>(f->fr, perm, r, f->src0, f->src1, buf, f->y);
        }
    }
    for (auto it = f->levels.rbegin(); it != f->levels.rend(); ++it) {
        const Level &l = *it;
        if (l.pmax == 0) continue;
        const int r = rows_per_cta(f, l.count, l.pmax);
        k_tree_bwd<<<dim3(l.count, up(l.pmax, r)), SV_THREADS, (size_t)std::max(1, l.qmax) * sizeof(double), s>>>(
            f->fr, f->perm + l.first, r, f->ids, buf, f->y, f->x);
    }
    return cudaGetLastError();
}

}  // namespace

extern "C" int vefem_tree_create(int device, int nfront, int nlevel, const int32_t *level_ptr, const int64_t *off,
                                 const int32_t *n, const int32_t *p, const int32_t *ld, const int32_t *child,
                                 const int64_t *ids, const int64_t *idx_off, const int32_t *src, int64_t N,
                                 vefem_tree **out)
{
    if (!out || nfront <= 0 || nlevel <= 0 || !level_ptr || !off || !n || !p || !ld || !child || !ids || !idx_off ||
        !src || N <= 0 || N >= INT32_MAX || idx_off[nfront] >= INT32_MAX)
        return VEFEM_ERR_ARG;
    *out = nullptr;
    if (level_ptr[0] != 0 || level_ptr[nlevel] != nfront || off[0] < 0) return VEFEM_ERR_ARG;
    const int64_t tot = idx_off[nfront];
    // every unknown a pivot once; every map inside its child's boundary; children one level below
    std::vector<int> level(nfront);
    for (int l = 0; l < nlevel; l++) {
        if (level_ptr[l + 1] <= level_ptr[l]) return VEFEM_ERR_ARG;
        for (int t = level_ptr[l]; t < level_ptr[l + 1]; t++) level[t] = l;
    }
    std::vector<char> seen((size_t)N, 0);
    int64_t pivots = 0;
    for (int t = 0; t < nfront; t++) {
        if (n[t] < 0 || p[t] < 0 || p[t] > n[t] || ld[t] < n[t] || ld[t] % 4 || off[t] % 4 ||
            off[t + 1] - off[t] < (int64_t)n[t] * ld[t] || idx_off[t + 1] - idx_off[t] != n[t])
            return VEFEM_ERR_ARG;
        for (int j = 0; j < n[t]; j++) {
            const int64_t u = ids[idx_off[t] + j];
            if (u < 0 || u >= N || (j < p[t] && seen[(size_t)u])) return VEFEM_ERR_ARG;
            if (j < p[t]) seen[(size_t)u] = 1;
        }
        pivots += p[t];
        for (int s = 0; s < 2; s++) {
            const int c = child[2 * t + s];
            if (c >= nfront || (c >= 0 && level[c] != level[t] - 1)) return VEFEM_ERR_ARG;
            for (int j = 0; j < n[t]; j++) {
                const int a = src[s * tot + idx_off[t] + j];
                if (a >= 0 && (c < 0 || a < p[c] || a >= n[c])) return VEFEM_ERR_ARG;
            }
        }
    }
    if (pivots != N) return VEFEM_ERR_ARG;

    vefem_tree *f = new vefem_tree();
    f->device = device;
    f->nfront = nfront;
    f->N = N;
    f->total = tot;
    f->buf_len = off[nfront];
    std::vector<Front> fr(nfront);
    std::vector<int32_t> perm(nfront);
    std::iota(perm.begin(), perm.end(), 0);
    int64_t cmax = 0, tmax = 0, dmax = 0;
    for (int l = 0; l < nlevel; l++) {
        Level v{level_ptr[l], level_ptr[l + 1] - level_ptr[l], 0, 0, 0, 0, {}, {}, 0};
        std::stable_sort(perm.begin() + v.first, perm.begin() + v.first + v.count,
                         [&](int a, int c) { return p[a] > p[c]; });
        int64_t cp = 0, tp = 0;
        for (int k = v.first; k < v.first + v.count; k++) {
            const int t = perm[k];
            fr[t] = Front{off[t], cp, tp, (int32_t)idx_off[t], n[t], p[t], ld[t], {child[2 * t], child[2 * t + 1]}};
            cp += (int64_t)p[t] * KB;
            tp += (int64_t)ld[t] * KB;
            v.nmax = std::max(v.nmax, n[t]);
            v.pmax = std::max(v.pmax, p[t]);
            v.qmax = std::max(v.qmax, n[t] - p[t]);
            v.ldmax = std::max(v.ldmax, ld[t]);
        }
        for (int k0 = 0; k0 < v.pmax; k0 += KB) {
            int a = 0, m = 0;
            while (a < v.count && p[perm[v.first + a]] > k0) m = std::max(m, (int)ld[perm[v.first + a++]]);
            v.active.push_back(a);
            v.ld_active.push_back(m);
        }
        while (v.many < v.count && p[perm[v.first + v.many]] > split::EXACT_K) v.many++;
        dmax = std::max<int64_t>(dmax, (int64_t)v.count * KB * KB);
        cmax = std::max(cmax, cp);
        tmax = std::max(tmax, tp);
        f->pmax = std::max(f->pmax, v.pmax);
        f->qmax = std::max(f->qmax, v.qmax);
        f->levels.push_back(std::move(v));
    }
    std::vector<int32_t> ids32(ids, ids + tot);
    Guard g(device);
    auto put = [](auto **dst, const auto *from, size_t count) {
        return cudaMalloc((void **)dst, std::max<size_t>(1, count) * sizeof(**dst)) == cudaSuccess &&
               (!from || cudaMemcpy(*dst, from, count * sizeof(**dst), cudaMemcpyHostToDevice) == cudaSuccess);
    };
    const double *none = nullptr;
    const bool ok =
        cudaDeviceGetAttribute(&f->sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess &&
        cudaStreamCreateWithFlags(&f->cs, cudaStreamNonBlocking) == cudaSuccess && put(&f->fr, fr.data(), fr.size()) &&
        put(&f->perm, perm.data(), perm.size()) && put(&f->ids, ids32.data(), ids32.size()) &&
        put(&f->src0, src, (size_t)tot) && put(&f->src1, src + tot, (size_t)tot) &&
        put(&f->e0, (const int32_t *)nullptr, (size_t)tot) && put(&f->e1, (const int32_t *)nullptr, (size_t)tot) && put(&f->cpan, none, (size_t)cmax) &&
        put(&f->tpan, none, (size_t)tmax) && put(&f->dinv, none, (size_t)dmax) && put(&f->y, none, (size_t)tot) && put(&f->b, none, (size_t)N) &&
        put(&f->x, none, (size_t)N) && put(&f->err, (const int *)nullptr, 1) &&
        put(&f->minpiv, (const unsigned long long *)nullptr, 1);
    // The sweeps stage a vector of pivots or boundary unknowns.  The limit of a
    // kernel's dynamic shared memory is the device's, not this handle's: beyond
    // the default it is set to all there is, so that no handle lowers another's.
    const int64_t staged = (int64_t)std::max(f->pmax, f->qmax) * (int64_t)sizeof(double);
    int most = 0;
    bool fits = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) == cudaSuccess &&
                staged <= most;
    if (fits && staged > 48 * 1024)
        fits = cudaFuncSetAttribute(k_tree_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, most) == cudaSuccess &&
               cudaFuncSetAttribute(k_tree_up, cudaFuncAttributeMaxDynamicSharedMemorySize, most) == cudaSuccess &&
               cudaFuncSetAttribute(k_tree_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, most) == cudaSuccess;
    if (!ok || !fits ||
        cudaFuncSetAttribute(k_pivot, cudaFuncAttributeMaxDynamicSharedMemorySize, split::SHORT_SMEM<KB>) != cudaSuccess ||
        cudaFuncSetAttribute(k_update, cudaFuncAttributeMaxDynamicSharedMemorySize, split::SHORT_SMEM<split::TN>) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_schur<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             2 * split::STAGE) != cudaSuccess ||
        cudaFuncSetAttribute(k_schur<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, split::STAGE) != cudaSuccess) {
        cudaGetLastError();
        vefem_tree_destroy(f);
        return VEFEM_ERR_NOMEM;
    }
    *out = f;
    return VEFEM_OK;
}

extern "C" int vefem_tree_factor(vefem_tree *f, const double *vals, const int64_t *dest, int64_t nnz, double *buf,
                                 int64_t buf_len, void *stream, double tol, double *min_pivot)
{
    if (!f || !vals || !dest || nnz <= 0 || !buf || reinterpret_cast<uintptr_t>(buf) % 16 || buf_len < f->buf_len)
        return VEFEM_ERR_ARG;
    Guard g(f->device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const double one = 1.0;
    std::memcpy(&f->h_one, &one, sizeof(one));
    TCK(cudaMemsetAsync(f->err, 0, sizeof(int), s));
    TCK(cudaMemcpyAsync(f->minpiv, &f->h_one, sizeof(f->h_one), cudaMemcpyHostToDevice, s));
    TCK(cudaMemsetAsync(buf, 0, (size_t)buf_len * sizeof(double), s));
    k_scatter<<<(unsigned)((nnz + 255) / 256), 256, 0, s>>>(nnz, dest, vals, buf);
    for (size_t li = 0; li < f->levels.size(); li++) {
        const Level &l = f->levels[li];
        const int32_t *perm = f->perm + l.first;
        if (li > 0 && l.nmax > 0)
            k_assemble<<<dim3(l.count, up(l.nmax, AS_ROWS)), dim3(32, AS_ROWS), 0, s>>>(f->fr, perm, f->src0, f->src1,
                                                                                       buf);
        for (size_t st = 0; st < l.active.size(); st++) {
            const int k0 = (int)st * KB, a = l.active[st], ld = l.ld_active[st];
            const int ntc = (int)up(ld, split::TN);
            TCK(launch_early(k_invert, dim3(a), IV_THREADS, 0, s, f->fr, perm, k0, buf, f->dinv, f->err, f->minpiv, tol));
            TCK(launch_early(k_pivot, dim3(a, up(ld, split::TM)), split::THREADS, split::SHORT_SMEM<KB>, s, f->fr, perm, k0,
                             buf, f->dinv, f->cpan, f->tpan, f->err));
            TCK(launch_early(k_update, dim3(a, ntc * up(l.pmax, split::TM)), split::THREADS, split::SHORT_SMEM<split::TN>, s,
                             f->fr, perm, k0, ntc, f->cpan, f->tpan, buf, f->err));
        }
        if (l.qmax > 0 && l.pmax > 0) {
            const int ntc = (int)up(l.qmax, split::TN);
            k_split_inner<<<dim3(l.count, up(l.pmax, 32)), 256, 0, s>>>(f->fr, perm, buf, f->e0);
            k_split_outer<<<dim3(l.count, up(l.qmax, 32)), 256, 0, s>>>(f->fr, perm, buf, f->e0, f->e1);
            const unsigned tiles = ntc * up(l.qmax, split::TM);
            if (l.many > 0)
                k_schur<2><<<dim3(l.many, tiles), split::THREADS, 2 * split::STAGE, s>>>(
                    f->fr, perm, ntc, f->e0, f->e1, buf, f->err);
            if (l.many < l.count)
                k_schur<1><<<dim3(l.count - l.many, tiles), split::THREADS, split::STAGE, s>>>(
                    f->fr, perm + l.many, ntc, f->e0, f->e1, buf, f->err);
        }
    }
    TCK(cudaGetLastError());
    int herr = 0;
    unsigned long long hmin = 0;
    TCK(cudaMemcpyAsync(&herr, f->err, sizeof(int), cudaMemcpyDeviceToHost, s));
    TCK(cudaMemcpyAsync(&hmin, f->minpiv, sizeof(hmin), cudaMemcpyDeviceToHost, s));
    TCK(cudaStreamSynchronize(s));
    if (min_pivot) std::memcpy(min_pivot, &hmin, sizeof(double));
    if (herr == 2) return tfail(f, VEFEM_ERR_CUDA, "a wait for the tensor core ran out");
    if (herr) return tfail(f, VEFEM_ERR_SINGULAR, "a pivot below the tolerance (unpivoted elimination)");
    return VEFEM_OK;
}

extern "C" int vefem_tree_solve(vefem_tree *f, const double *buf, const double *b, double *x, void *stream)
{
    if (!f || !buf || !b || !x) return VEFEM_ERR_ARG;
    Guard g(f->device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (!f->graph || f->graph_buf != buf) {
        if (f->graph) cudaGraphExecDestroy(f->graph);
        f->graph = nullptr;
        cudaGraph_t gr = nullptr;
        TCK(cudaStreamBeginCapture(f->cs, cudaStreamCaptureModeThreadLocal));
        const cudaError_t le = launch_sweeps(f, buf, f->cs);
        const cudaError_t ce = cudaStreamEndCapture(f->cs, &gr);
        cudaError_t e = le != cudaSuccess ? le : ce;
        if (e == cudaSuccess) e = cudaGraphInstantiate(&f->graph, gr, 0);
        if (gr) cudaGraphDestroy(gr);
        if (e != cudaSuccess) {
            f->graph = nullptr;
            cudaGetLastError();
            return tfail(f, VEFEM_ERR_CUDA, std::string("solve graph: ") + cudaGetErrorString(e));
        }
        f->graph_buf = buf;
    }
    TCK(cudaMemcpyAsync(f->b, b, (size_t)f->N * sizeof(double), cudaMemcpyDeviceToDevice, s));
    TCK(cudaGraphLaunch(f->graph, s));
    TCK(cudaMemcpyAsync(x, f->x, (size_t)f->N * sizeof(double), cudaMemcpyDeviceToDevice, s));
    return VEFEM_OK;
}

extern "C" int vefem_tree_launches(const vefem_tree *f)
{
    if (!f) return -1;
    int n = 0;
    for (const Level &l : f->levels) n += 2 * (l.pmax > 0) + (l.qmax > 0);
    return n;
}

extern "C" void vefem_tree_destroy(vefem_tree *f)
{
    if (!f) return;
    {
        Guard g(f->device);
        if (f->graph) cudaGraphExecDestroy(f->graph);
        if (f->cs) cudaStreamDestroy(f->cs);
        void *p[] = {f->fr, f->perm, f->ids, f->src0, f->src1, f->e0, f->e1, f->cpan, f->tpan, f->dinv, f->y, f->b, f->x, f->err, f->minpiv};
        for (void *q : p) cudaFree(q);
    }
    delete f;
}

extern "C" const char *vefem_tree_last_error(const vefem_tree *f) { return f ? f->msg.c_str() : "null tree handle"; }
