// Inversion of one pivot block of the blocked Gauss-Jordan eliminations
// (vefem_frontal.cu, vefem_tree.cu).
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace {

constexpr int NB = 16;   // pivots per Gauss-Jordan step

// Positive doubles order like their bit patterns: atomicMin on the bits.
__device__ void atomic_min_pos(unsigned long long *addr, double v)
{
    atomicMin(addr, (unsigned long long)__double_as_longlong(v));
}

// 1/x: the hardware's approximation (20 bits) refined by two steps of Newton's
// iteration for the reciprocal, r <- r + r (1 - x r) (quadratic convergence: 20
// -> 40 -> rounding level).  Four FP64 instructions instead of a full IEEE
// division, which matters on the critical path of a pivot block's inversion (a
// warp issues an FP64 instruction every few tens of clocks on this GPU, and a
// conversion to and from a single-precision seed counts as two).  Values whose
// reciprocal comes near the ends of the range take the IEEE division.
__device__ __forceinline__ bool plain_exponent(double x)
{
    const int ex = (__double2hiint(x) >> 20) & 0x7ff;
    return ex >= 64 && ex <= 1982;
}

__device__ __forceinline__ double approximate_reciprocal(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}

__device__ __forceinline__ double recip(double x)
{
    if (!plain_exponent(x)) return 1.0 / x;
    double r = approximate_reciprocal(x);
    double e = fma(-x, r, 1.0);
    r = fma(r, e, r);
    e = fma(-x, r, 1.0);
    return fma(r, e, r);
}

// In-place Gauss-Jordan inversion without pivoting of the NB x NB block held
// in A (shared, column-major: A[column][row]; columns 0..NB-1 the block padded
// with the identity, columns NB..2NB-1 the identity on entry and the inverse on
// exit), by threads 0..127 of the block (named barrier 1), so that other warps
// of the block can work meanwhile: thread = (column, quarter of the rows), the
// FP64 work of a pivot step spread over four warps.  Returns (to the 128
// threads) the smallest |pivot| over the largest |entry| of the kb x kb block,
// or -1 when a pivot is at most tol times that largest entry or not finite.
__device__ __forceinline__ void bar128() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

__device__ double block_invert(double (*A)[NB + 1], int kb, double tol, double *s_red)
{
    const int t = threadIdx.x;
    const int c = t & 31, q = (t >> 5) & 3;
    double amax = 0.0;
    if (c < kb) {
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (q * 4 + u < kb) amax = fmax(amax, fabs(A[c][q * 4 + u]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (c == 0) s_red[q] = amax;
    bar128();
    amax = fmax(fmax(s_red[0], s_red[1]), fmax(s_red[2], s_red[3]));
    bool bad = !(amax > 0.0) || !isfinite(amax);
    const double floor_ = tol * amax;
    double pmin = INFINITY;
#pragma unroll 1
    for (int p = 0; p < NB; p++) {
        const double piv = A[p][p];
        if (p < kb) {
            pmin = fmin(pmin, fabs(piv));
            if (!(fabs(piv) > floor_) || !isfinite(piv)) bad = true;
        }
        const double rp = A[c][p] * recip(piv);
        double f[4];
#pragma unroll
        for (int u = 0; u < 4; u++) f[u] = A[p][q * 4 + u];
        bar128();
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int r = q * 4 + u;
            A[c][r] = (r == p) ? rp : fma(-f[u], rp, A[c][r]);
        }
        bar128();
    }
    return bad ? -1.0 : pmin / amax;
}

}  // namespace
