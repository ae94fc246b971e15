// Panel-frontal elimination of the bordered Newton Jacobian on the device, in
// place of the MUMPS factorisation and solve behind KSPSolve (Petsc_mod.F90:850):
// the fronts of a caller's panel ordering, one after the other.  The drivers'
// default is the nested dissection of vefem_tree.cu.
//
// The symbolic phase (element panels, pivots and fronts, the map of every AIJ
// entry into a frontal matrix, the extend-add maps) is the caller's; this file
// runs the numeric phases on frontal matrices stored row-major, one after the
// other, in one device buffer.
//
// Factorisation.  Panel q's frontal matrix M (n x n) holds its P pivots first and
// its front F after them.  After the extend-add of the previous panel's Schur
// complement, the P pivot columns are eliminated by blocked Gauss-Jordan without
// pivoting, NB pivots per step:
//
//     D = M[K,K] (NB x NB),  T = D^-1 M[K,:],  C = M[:,K]
//     M[K,:] = T,   M[K,K] = D^-1,
//     M[i,K] = -C[i] D^-1,          i not in K
//     M[i,j] = M[i,j] - C[i] T[j],  i, j not in K
//
// After the P pivots M = [A^-1, A^-1 B; -C A^-1, S] with A = M[P,P], B = M[P,F],
// C = M[F,P] and S = M[F,F] - C A^-1 B the Schur complement passed on to the
// next panel.  Gauss-Jordan does about twice the work of a partial LU on these
// matrices, but every step is one parallel rank-NB update (no triangular solves,
// whose column-by-column latency dominates dense LU at these sizes), and it
// leaves exactly what the solve needs as dense blocks.  Without pivoting the
// elimination needs a nonzero pivot in every step: a pivot below tol times the
// largest entry of its NB x NB block sets an error flag and the caller
// factorises that matrix another way.
//
// Solve (two launches per panel, replayed from a CUDA graph): forward
// y_P = A^-1 b_P, b_F += (-C A^-1) b_P; backward x_P = y_P - (A^-1 B) x_F.  Sums
// run in a fixed order (warp-strided, then a fixed shuffle tree): results are
// reproducible run to run.  The sweeps are latency-bound (a panel's rows are a
// few hundred dot products of a few hundred entries), so the vectors are kept
// in elimination order (a panel's right-hand side is one contiguous slice,
// staged in shared memory) and consecutive launches overlap by programmatic
// dependent launch: each kernel loads its rows of the factors before it waits
// for the previous one.  (Measured slower: one launch of one 16-CTA cluster
// with cluster barriers between panels, bound by the FP64 rate of 16 SMs; and
// one cooperative launch of all SMs whose CTAs ordered the panels through
// per-panel counters in global memory, 29 ms against 21 ms per solve at
// 20,000 quads: a counter handoff between SMs costs more than the hardware's
// launch-to-launch dependency.)
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "vefem.h"
#include "vefem_gj.cuh"

namespace {

// First step of a panel: D^-1 of the first pivot block (every CTA) and
// T = D^-1 M[K,:] for the CTA's 32 columns.  128 threads.
__global__ void __launch_bounds__(128) k_gj_start(const double *__restrict__ M, int n, int kb,
                                                  double *__restrict__ Tbuf, double *__restrict__ invbuf,
                                                  int *err, unsigned long long *minpiv, double tol)
{
    __shared__ double sA[2 * NB][NB + 1];
    __shared__ double s_red[4];
    const int t = threadIdx.x;
    for (int u = t; u < 2 * NB * NB; u += blockDim.x) {
        const int c = u / NB, r = u % NB;
        double v;
        if (c < NB)
            v = (r < kb && c < kb) ? M[(int64_t)r * n + c] : (r == c ? 1.0 : 0.0);
        else
            v = (r == c - NB) ? 1.0 : 0.0;
        sA[c][r] = v;
    }
    __syncthreads();
    const double rel = block_invert(sA, kb, tol, s_red);
    if (blockIdx.x == 0) {
        for (int u = t; u < NB * NB; u += blockDim.x) invbuf[u] = sA[NB + u % NB][u / NB];
        if (t == 0) {
            if (rel < 0.0) atomicExch(err, 1);
            else atomic_min_pos(minpiv, rel);
        }
    }
    const int j = blockIdx.x * 32 + (t & 31);
    const int g = t >> 5;
    if (j < n) {
        double m[NB];
#pragma unroll
        for (int l = 0; l < NB; l++) m[l] = l < kb ? M[(int64_t)l * n + j] : 0.0;
#pragma unroll
        for (int kk = 0; kk < 4; kk++) {
            const int k = g * 4 + kk;
            double acc = 0.0;
#pragma unroll
            for (int l = 0; l < NB; l++) acc = fma(sA[NB + l][k], m[l], acc);
            Tbuf[(int64_t)k * n + j] = acc;
        }
    }
}

// The new value of entry (i, j) in a Gauss-Jordan step on pivots
// K = [k0, k0+kb): C the row's K entries (Min[i, K]), T = D^-1 Min[K,:],
// inv = D^-1.  One function for every caller, so that the look-ahead's
// recomputed pivot block equals the written entries bit for bit.
__device__ __forceinline__ double gj_entry(const double *__restrict__ Min, int n, int i, int j, int k0,
                                           int kb, const double *ci, const double (*sT)[32], int cc,
                                           const double (*sInv)[NB])
{
    const bool iK = i >= k0 && i < k0 + kb, jK = j >= k0 && j < k0 + kb;
    if (iK) return jK ? sInv[i - k0][j - k0] : sT[i - k0][cc];
    double acc = 0.0;
    if (jK) {
#pragma unroll
        for (int l = 0; l < NB; l++) acc = fma(ci[l], sInv[l][j - k0], acc);
        return -acc;
    }
#pragma unroll
    for (int l = 0; l < NB; l++) acc = fma(ci[l], sT[l][cc], acc);
    return Min[(int64_t)i * n + j] - acc;
}

// One Gauss-Jordan step on pivots K = [k0, k0+kb): reads Min (the matrix
// before the step), writes every entry of Mout; T = D^-1 Min[K,:] and D^-1
// come from the previous launch (Tcur, invcur).
//
// Blocks 0 .. nlook-1 are look-ahead blocks (when a next pivot block
// K' = [k1, k1+kb1) exists), one per 32 columns J: warps 0-3 form the next
// pivot block D' = Mout[K',K'] from the inputs and invert it while warps 4-7
// write the rows K' of Mout for the columns J; then all form
// T' = D'^-1 Mout[K', J] (Tnext), and block 0 writes D'^-1 (invnext): the
// next step needs no separate preparation launch, and the serial inversion
// overlaps the bulk update.  The other blocks update the 16-row x 32-column
// tiles of every other row band, taking tiles from a ticket counter (zero at
// launch) until none are left.  256 threads.
__global__ void __launch_bounds__(256) k_gj_step(const double *__restrict__ Min, double *__restrict__ Mout,
                                                 int n, int k0, int kb,
                                                 const double *__restrict__ Tcur,
                                                 const double *__restrict__ invcur, int k1, int kb1,
                                                 double *__restrict__ Tnext, double *__restrict__ invnext,
                                                 int *err, unsigned long long *minpiv, double tol,
                                                 int *__restrict__ ticket)
{
    __shared__ double sC[NB][NB + 1];
    __shared__ double sT[NB][32];
    __shared__ double sInv[NB][NB];
    __shared__ double sOut[NB][33];
    __shared__ double sA[2 * NB][NB + 1];
    __shared__ double s_red[4];
    const int t = threadIdx.x;
    const int ncol = (n + 31) / 32;
    const bool look = kb1 > 0;
    const int nlook = look ? ncol : 0;
    const int nband = (n + NB - 1) / NB;
    const int nbulk = (nband - (look ? 1 : 0)) * ncol;
    sInv[t >> 4][t & 15] = invcur[t];
    if ((int)blockIdx.x >= nlook) {
        // bulk: 16-row x 32-column tiles handed out by a ticket counter (every
        // SM keeps working until the tiles run out), 2 columns per thread
        __shared__ int s_tile;
        for (;;) {
            __syncthreads();
            if (t == 0) s_tile = atomicAdd(ticket, 1);
            __syncthreads();
            const int b = s_tile;
            if (b >= nbulk) return;
            const int rb = b / ncol;
            const int band = (look && rb >= k1 / NB) ? rb + 1 : rb;
            const int jc = b - rb * ncol;
            const int i0 = band * NB, j0 = jc * 32;
            {
                const int r = t >> 4, l = t & 15;
                sC[r][l] = (i0 + r < n && l < kb) ? Min[(int64_t)(i0 + r) * n + k0 + l] : 0.0;
                for (int u = t; u < NB * 32; u += 256) {
                    const int k = u >> 5, cc = u & 31;
                    sT[k][cc] = (j0 + cc < n) ? Tcur[(int64_t)k * n + j0 + cc] : 0.0;
                }
            }
            __syncthreads();
            const int r = t >> 4, c0 = (t & 15) * 2;
            const int i = i0 + r;
            if (i < n) {
                double ci[NB];
#pragma unroll
                for (int l = 0; l < NB; l++) ci[l] = sC[r][l];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int cc = c0 + u, j = j0 + cc;
                    if (j < n) Mout[(int64_t)i * n + j] = gj_entry(Min, n, i, j, k0, kb, ci, sT, cc, sInv);
                }
            }
        }
    }
    // look-ahead block: band K', column chunk blockIdx.x
    const int i0 = k1, j0 = blockIdx.x * 32;
    {
        const int r = t >> 4, l = t & 15;
        sC[r][l] = (i0 + r < n && l < kb) ? Min[(int64_t)(i0 + r) * n + k0 + l] : 0.0;
        for (int u = t; u < NB * 32; u += 256) {
            const int k = u >> 5, cc = u & 31;
            sT[k][cc] = (j0 + cc < n) ? Tcur[(int64_t)k * n + j0 + cc] : 0.0;
        }
    }
    __syncthreads();
    if (t < 128) {
        // D' from the inputs: rows K' = this band, columns K' (their C rows are
        // sC, their T columns read from Tcur)
        for (int u = t; u < 2 * NB * NB; u += 128) {
            const int cc = u / NB, rr = u % NB;
            double v;
            if (cc < NB) {
                if (rr < kb1 && cc < kb1) {
                    double ci[NB];
#pragma unroll
                    for (int l = 0; l < NB; l++) ci[l] = sC[rr][l];
                    const int j = k1 + cc;
                    double acc = 0.0;
                    const bool jK = j >= k0 && j < k0 + kb;
                    if (jK) {
#pragma unroll
                        for (int l = 0; l < NB; l++) acc = fma(ci[l], sInv[l][j - k0], acc);
                        v = -acc;
                    } else {
#pragma unroll
                        for (int l = 0; l < NB; l++) acc = fma(ci[l], Tcur[(int64_t)l * n + j], acc);
                        v = Min[(int64_t)(k1 + rr) * n + j] - acc;
                    }
                } else {
                    v = rr == cc ? 1.0 : 0.0;
                }
            } else {
                v = (rr == cc - NB) ? 1.0 : 0.0;
            }
            sA[cc][rr] = v;
        }
        bar128();
        const double rel = block_invert(sA, kb1, tol, s_red);
        if (blockIdx.x == 0 && t == 0) {
            if (rel < 0.0) atomicExch(err, 1);
            else atomic_min_pos(minpiv, rel);
        }
    } else {
        // rows K' of this chunk: 16 x 32 entries, 4 per thread
        const int tt = t - 128;
        const int r = tt >> 3, c0 = (tt & 7) * 4;
        const int i = i0 + r;
        double ci[NB];
#pragma unroll
        for (int l = 0; l < NB; l++) ci[l] = sC[r][l];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int cc = c0 + u, j = j0 + cc;
            double out = 0.0;
            if (i < n && j < n) {
                out = gj_entry(Min, n, i, j, k0, kb, ci, sT, cc, sInv);
                Mout[(int64_t)i * n + j] = out;
            }
            sOut[r][cc] = (r < kb1) ? out : 0.0;
        }
    }
    __syncthreads();
    if (blockIdx.x == 0)
        for (int u = t; u < NB * NB; u += 256) invnext[u] = sA[NB + u % NB][u / NB];
    // T' = D'^-1 rows K' for this chunk: 2 entries per thread
    {
        const int k = t >> 4, c0 = (t & 15) * 2;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int cc = c0 + u, j = j0 + cc;
            if (j < n) {
                double acc = 0.0;
#pragma unroll
                for (int l = 0; l < NB; l++) acc = fma(sA[NB + l][k], sOut[l][cc], acc);
                Tnext[(int64_t)k * n + j] = acc;
            }
        }
    }
}

// M_q[e[a], e[b]] += S_prev[a, b], S_prev = M_prev[p_prev:, p_prev:]
__global__ void k_extend_add(double *__restrict__ Mq, int nq, const double *__restrict__ Mp, int np,
                             int pp, const int32_t *__restrict__ e, int f)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)f * f) return;
    const int a = (int)(t / f), b = (int)(t - (int64_t)a * f);
    Mq[(int64_t)e[a] * nq + e[b]] += Mp[(int64_t)(pp + a) * np + pp + b];
}

__device__ double warp_sum(double s)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Programmatic dependent launch: a sweep kernel is launched while the previous
// one still runs; everything before pdl_wait() may read only what no kernel of
// the solve writes (the factors and the index arrays), everything after it
// sees the previous kernel's results.  Without a programmatic dependency the
// wait returns at once.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

constexpr int SV_WARPS = 8;   // rows per CTA of the sweep kernels (a warp per row)
constexpr int SV_PRE = 8;     // row entries per lane loaded before the wait

// The sweeps work in elimination order: position start[q] + r holds the
// unknown of panel q's pivot r, so a panel's right-hand side entries are one
// contiguous slice; pidx[r] is the position of the panel's row r (its pivots
// map to start + r, its front to the pivots of later panels).  Each row's sum
// runs lane-strided over the columns, then a fixed shuffle tree.
//
// forward, panel q: row r of M[:, :p] against b_P; r < p -> y, r >= p -> b_F +=
__global__ void __launch_bounds__(SV_WARPS * 32) k_solve_fwd(const double *__restrict__ M, int n, int p,
                                                             int start, const int32_t *__restrict__ pidx,
                                                             double *__restrict__ bp,
                                                             double *__restrict__ y)
{
    extern __shared__ double s_vec[];
    const int r = blockIdx.x * SV_WARPS + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    const double *row = M + (int64_t)(r < n ? r : 0) * n;
    double pre[SV_PRE];
#pragma unroll
    for (int k = 0; k < SV_PRE; k++) {
        const int c = lane + 32 * k;
        pre[k] = (r < n && c < p) ? row[c] : 0.0;
    }
    const int dst = (r < n && r >= p) ? pidx[r] : start + r;
    pdl_wait();
    for (int c = threadIdx.x; c < p; c += blockDim.x) s_vec[c] = bp[start + c];
    __syncthreads();
    pdl_launch_dependents();
    if (r >= n) return;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < SV_PRE; k++) {
        const int c = lane + 32 * k;
        if (c < p) s = fma(pre[k], s_vec[c], s);
    }
    for (int c = lane + 32 * SV_PRE; c < p; c += 32) s = fma(row[c], s_vec[c], s);
    s = warp_sum(s);
    if (lane == 0) {
        if (r < p)
            y[dst] = s;
        else
            bp[dst] += s;
    }
}

// backward, panel q: x_P = y_P - M[:p, p:] x_F
__global__ void __launch_bounds__(SV_WARPS * 32) k_solve_bwd(const double *__restrict__ M, int n, int p,
                                                             int start, const int32_t *__restrict__ pidx,
                                                             const double *__restrict__ y,
                                                             double *__restrict__ xp)
{
    extern __shared__ double s_vec[];
    const int r = blockIdx.x * SV_WARPS + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    const int f = n - p;
    const double *row = M + (int64_t)(r < p ? r : 0) * n + p;
    double pre[SV_PRE];
#pragma unroll
    for (int k = 0; k < SV_PRE; k++) {
        const int c = lane + 32 * k;
        pre[k] = (r < p && c < f) ? row[c] : 0.0;
    }
    int src[SV_PRE];
#pragma unroll
    for (int k = 0; k < SV_PRE; k++) {
        const int c = threadIdx.x + k * SV_WARPS * 32;
        src[k] = c < f ? pidx[p + c] : 0;
    }
    pdl_wait();
#pragma unroll
    for (int k = 0; k < SV_PRE; k++) {
        const int c = threadIdx.x + k * SV_WARPS * 32;
        if (c < f) s_vec[c] = xp[src[k]];
    }
    for (int c = threadIdx.x + SV_PRE * SV_WARPS * 32; c < f; c += blockDim.x) s_vec[c] = xp[pidx[p + c]];
    __syncthreads();
    pdl_launch_dependents();
    if (r >= p) return;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < SV_PRE; k++) {
        const int c = lane + 32 * k;
        if (c < f) s = fma(pre[k], s_vec[c], s);
    }
    for (int c = lane + 32 * SV_PRE; c < f; c += 32) s = fma(row[c], s_vec[c], s);
    s = warp_sum(s);
    if (lane == 0) xp[start + r] = y[start + r] - s;
}

// b in elimination order (bp[i] = b[elim[i]]), and back (x[elim[i]] = xp[i])
__global__ void k_to_elim(int64_t N, const int32_t *__restrict__ elim, const double *__restrict__ b,
                          double *__restrict__ bp)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) bp[i] = b[elim[i]];
}

__global__ void k_from_elim(int64_t N, const int32_t *__restrict__ elim, const double *__restrict__ xp,
                            double *__restrict__ x)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) x[elim[i]] = xp[i];
}

}  // namespace

struct vefem_frontal {
    int device = 0;
    int npan = 0;
    int64_t N = 0;
    int nmax = 0;
    std::vector<int64_t> off, ext_off, idx_off;
    std::vector<int> n, p;
    const int32_t *ext = nullptr;   // caller's device arrays
    const int64_t *idx = nullptr;
    double *Tbuf[2] = {nullptr, nullptr}, *inv[2] = {nullptr, nullptr};
    double *W = nullptr;                  // ping-pong partner of a panel's matrix
    int *tickets = nullptr;               // one tile counter per Gauss-Jordan step
    int64_t nsteps_total = 0;
    int bulk_ctas = 0;                    // resident CTAs of the step kernel on this GPU
    int *err = nullptr;
    unsigned long long *minpiv = nullptr;
    unsigned long long h_minpiv = 0;   // staging of the initial value (outlives the async copy)
    // solve: work vectors in elimination order and the CUDA graph of the two
    // sweeps (captured per buf)
    double *wb = nullptr, *wy = nullptr, *wx = nullptr;
    int32_t *elim = nullptr;              // global unknown at each elimination position
    int32_t *pidx = nullptr;              // elimination position of every panel row (idx layout)
    std::vector<int> start;               // first elimination position of each panel's pivots
    int max_p = 0, max_f = 0;
    bool pdl = true;                      // sweeps chained by programmatic dependent launch
    int last_path = -1;                   // 1 graph with PDL, 2 graph without
    cudaStream_t cs = nullptr;
    cudaGraphExec_t graph = nullptr;
    const double *graph_buf = nullptr;
    std::string msg;
};

namespace {

int ffail(vefem_frontal *f, int code, const std::string &m)
{
    if (f) f->msg = m;
    return code;
}

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int d)
    {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        cudaSetDevice(d);
    }
    ~DeviceGuard()
    {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

}  // namespace

#define FCK(call)                                                                        \
    do {                                                                                 \
        cudaError_t _e = (call);                                                         \
        if (_e != cudaSuccess)                                                           \
            return ffail(f, VEFEM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(_e)); \
    } while (0)

extern "C" int vefem_frontal_create(int device, int npan, const int64_t *off, const int32_t *n,
                                    const int32_t *p, const int32_t *ext, const int64_t *ext_off,
                                    const int64_t *idx, const int64_t *idx_off, int64_t N,
                                    vefem_frontal **out)
{
    if (!out || npan <= 0 || !off || !n || !p || !ext_off || !idx || !idx_off || N <= 0 ||
        (npan > 1 && !ext))
        return VEFEM_ERR_ARG;
    *out = nullptr;
    vefem_frontal *f = new vefem_frontal();
    f->device = device;
    f->npan = npan;
    f->N = N;
    f->off.assign(off, off + npan + 1);
    f->ext_off.assign(ext_off, ext_off + npan);
    f->idx_off.assign(idx_off, idx_off + npan + 1);
    f->n.assign(n, n + npan);
    f->p.assign(p, p + npan);
    f->ext = ext;
    f->idx = idx;
    int64_t tot = 0;
    for (int q = 0; q < npan; q++) {
        if (n[q] <= 0 || p[q] < 0 || p[q] > n[q] || f->off[q + 1] - f->off[q] != (int64_t)n[q] * n[q] ||
            f->idx_off[q + 1] - f->idx_off[q] != n[q]) {
            delete f;
            return VEFEM_ERR_ARG;
        }
        if (q + 1 < npan && n[q] - p[q] > n[q + 1]) {   // the front must fit in the next panel
            delete f;
            return VEFEM_ERR_ARG;
        }
        tot += p[q];
        f->nmax = std::max(f->nmax, n[q]);
    }
    if (tot != N) {            // every unknown is a pivot exactly once
        delete f;
        return VEFEM_ERR_ARG;
    }
    for (int q = 0; q < npan; q++) f->nsteps_total += (p[q] + NB - 1) / NB;
    DeviceGuard g(device);
    {
        int sms = 0, occ = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_gj_step, 256, 0) != cudaSuccess) {
            delete f;
            return VEFEM_ERR_CUDA;
        }
        f->bulk_ctas = sms * std::max(1, occ);
    }
    if (cudaMalloc(&f->wb, (size_t)N * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&f->wy, (size_t)N * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&f->wx, (size_t)N * sizeof(double)) != cudaSuccess ||
        cudaStreamCreateWithFlags(&f->cs, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMalloc(&f->Tbuf[0], (size_t)NB * f->nmax * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&f->Tbuf[1], (size_t)NB * f->nmax * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&f->inv[0], NB * NB * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&f->inv[1], NB * NB * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&f->W, (size_t)f->nmax * f->nmax * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&f->tickets, (size_t)std::max<int64_t>(1, f->nsteps_total) * sizeof(int)) != cudaSuccess ||
        cudaMalloc(&f->err, sizeof(int)) != cudaSuccess ||
        cudaMalloc(&f->minpiv, sizeof(unsigned long long)) != cudaSuccess) {
        vefem_frontal_destroy(f);
        return VEFEM_ERR_NOMEM;
    }
    // elimination order of the solve: panel q's pivots at start[q] .. start[q] + p[q]
    {
        if (N >= INT32_MAX || f->idx_off[npan] >= INT32_MAX) {
            vefem_frontal_destroy(f);
            return VEFEM_ERR_ARG;
        }
        std::vector<int64_t> hidx((size_t)f->idx_off[npan]);
        if (cudaMemcpy(hidx.data(), idx, hidx.size() * sizeof(int64_t), cudaMemcpyDeviceToHost) != cudaSuccess) {
            vefem_frontal_destroy(f);
            return VEFEM_ERR_CUDA;
        }
        std::vector<int32_t> elim((size_t)N, -1), pos((size_t)N, -1), pidx(hidx.size());
        f->start.resize(npan);
        int64_t at = 0;
        bool ok = true;
        for (int q = 0; q < npan && ok; q++) {
            f->start[q] = (int)at;
            f->max_p = std::max(f->max_p, p[q]);
            f->max_f = std::max(f->max_f, n[q] - p[q]);
            for (int r = 0; r < p[q]; r++, at++) {
                const int64_t g = hidx[(size_t)(f->idx_off[q] + r)];
                if (g < 0 || g >= N || pos[(size_t)g] >= 0) { ok = false; break; }
                pos[(size_t)g] = (int32_t)at;
                elim[(size_t)at] = (int32_t)g;
            }
        }
        for (size_t k = 0; ok && k < hidx.size(); k++) {
            const int64_t g = hidx[k];
            if (g < 0 || g >= N) { ok = false; break; }
            pidx[k] = pos[(size_t)g];
        }
        if (!ok) {             // an unknown outside [0, N) or a pivot of two panels
            vefem_frontal_destroy(f);
            return VEFEM_ERR_ARG;
        }
        if (cudaMalloc(&f->elim, elim.size() * sizeof(int32_t)) != cudaSuccess ||
            cudaMalloc(&f->pidx, pidx.size() * sizeof(int32_t)) != cudaSuccess) {
            vefem_frontal_destroy(f);
            return VEFEM_ERR_NOMEM;
        }
        if (cudaMemcpy(f->elim, elim.data(), elim.size() * sizeof(int32_t), cudaMemcpyHostToDevice) != cudaSuccess ||
            cudaMemcpy(f->pidx, pidx.data(), pidx.size() * sizeof(int32_t), cudaMemcpyHostToDevice) != cudaSuccess) {
            vefem_frontal_destroy(f);
            return VEFEM_ERR_CUDA;
        }
        const size_t smem = (size_t)std::max(f->max_p, f->max_f) * sizeof(double);
        if (smem > 48 * 1024 &&
            (cudaFuncSetAttribute(k_solve_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
             cudaFuncSetAttribute(k_solve_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)) {
            vefem_frontal_destroy(f);
            return VEFEM_ERR_ARG;
        }
    }
    *out = f;
    return VEFEM_OK;
}

extern "C" int vefem_frontal_factor(vefem_frontal *f, double *buf, void *stream, double tol,
                                    double *min_pivot)
{
    if (!f || !buf) return VEFEM_ERR_ARG;
    DeviceGuard g(f->device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    FCK(cudaMemsetAsync(f->err, 0, sizeof(int), s));
    FCK(cudaMemsetAsync(f->tickets, 0, (size_t)f->nsteps_total * sizeof(int), s));
    int64_t step_id = 0;
    const double d_one = 1.0;
    std::memcpy(&f->h_minpiv, &d_one, sizeof(d_one));
    FCK(cudaMemcpyAsync(f->minpiv, &f->h_minpiv, sizeof(f->h_minpiv), cudaMemcpyHostToDevice, s));
    for (int q = 0; q < f->npan; q++) {
        const int n = f->n[q], p = f->p[q];
        double *M = buf + f->off[q];
        if (q > 0) {
            const int np = f->n[q - 1], pp = f->p[q - 1], fr = np - pp;
            if (fr > 0) {
                const int64_t tot = (int64_t)fr * fr;
                k_extend_add<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(
                    M, n, buf + f->off[q - 1], np, pp, f->ext + f->ext_off[q - 1], fr);
            }
        }
        if (p == 0) continue;
        // Gauss-Jordan steps ping-pong between the panel's matrix and W
        const int ncol = (n + 31) / 32, nband = (n + NB - 1) / NB;
        const int nsteps = (p + NB - 1) / NB;
        k_gj_start<<<(unsigned)ncol, 128, 0, s>>>(M, n, std::min(NB, p), f->Tbuf[0], f->inv[0], f->err,
                                                  f->minpiv, tol);
        for (int st = 0; st < nsteps; st++) {
            const int k0 = st * NB, kb = std::min(NB, p - k0);
            const int k1 = k0 + NB, kb1 = k1 < p ? std::min(NB, p - k1) : 0;
            const double *Min = (st & 1) ? f->W : M;
            double *Mout = (st & 1) ? M : f->W;
            // look-ahead blocks (one per column chunk, when a next pivot block
            // exists) + bulk blocks for every other row band
            const int nlook = kb1 > 0 ? ncol : 0;
            const int nbulk = (nband - (kb1 > 0 ? 1 : 0)) * ncol;
            const int grid = nlook + std::max(1, std::min(nbulk, f->bulk_ctas - nlook));
            k_gj_step<<<(unsigned)grid, 256, 0, s>>>(Min, Mout, n, k0, kb, f->Tbuf[st & 1],
                                                     f->inv[st & 1], k1, kb1, f->Tbuf[(st + 1) & 1],
                                                     f->inv[(st + 1) & 1], f->err, f->minpiv, tol,
                                                     f->tickets + step_id);
            step_id++;
        }
        if (nsteps & 1) FCK(cudaMemcpyAsync(M, f->W, (size_t)n * n * sizeof(double), cudaMemcpyDeviceToDevice, s));
    }
    FCK(cudaGetLastError());
    int herr = 0;
    unsigned long long hmin = 0;
    FCK(cudaMemcpyAsync(&herr, f->err, sizeof(int), cudaMemcpyDeviceToHost, s));
    FCK(cudaMemcpyAsync(&hmin, f->minpiv, sizeof(hmin), cudaMemcpyDeviceToHost, s));
    FCK(cudaStreamSynchronize(s));
    if (min_pivot) std::memcpy(min_pivot, &hmin, sizeof(double));
    if (herr) return ffail(f, VEFEM_ERR_SINGULAR, "a pivot below the tolerance (unpivoted elimination)");
    return VEFEM_OK;
}

namespace {

// One sweep launch; with pdl, the launch may begin while the previous kernel
// on the stream still runs (programmatic stream serialisation).
template <typename... Args, typename... Act>
cudaError_t launch_sweep(bool pdl, void (*kern)(Args...), unsigned grid, size_t smem, cudaStream_t s,
                         Act... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(SV_WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

// the two sweeps of a solve in elimination order (wb -> wy -> wx), on stream s
cudaError_t launch_sweeps(vefem_frontal *f, const double *buf, cudaStream_t s, bool pdl)
{
    const size_t smem_f = (size_t)std::max(1, f->max_p) * sizeof(double);
    const size_t smem_b = (size_t)std::max(1, f->max_f) * sizeof(double);
    for (int q = 0; q < f->npan; q++) {
        const int n = f->n[q], p = f->p[q];
        if (p == 0) continue;
        const cudaError_t e = launch_sweep(pdl, k_solve_fwd, (unsigned)((n + SV_WARPS - 1) / SV_WARPS), smem_f,
                                           s, (const double *)(buf + f->off[q]), n, p, f->start[q],
                                           (const int32_t *)(f->pidx + f->idx_off[q]), f->wb, f->wy);
        if (e != cudaSuccess) return e;
    }
    for (int q = f->npan - 1; q >= 0; q--) {
        const int n = f->n[q], p = f->p[q];
        if (p == 0) continue;
        const cudaError_t e = launch_sweep(pdl, k_solve_bwd, (unsigned)((p + SV_WARPS - 1) / SV_WARPS), smem_b,
                                           s, (const double *)(buf + f->off[q]), n, p, f->start[q],
                                           (const int32_t *)(f->pidx + f->idx_off[q]),
                                           (const double *)f->wy, f->wx);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// capture the sweeps into f->graph; cudaSuccess or the first error
cudaError_t capture_sweeps(vefem_frontal *f, const double *buf, bool pdl)
{
    cudaError_t e = cudaStreamBeginCapture(f->cs, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
    const cudaError_t le = launch_sweeps(f, buf, f->cs, pdl);
    cudaGraph_t gr = nullptr;
    e = cudaStreamEndCapture(f->cs, &gr);
    if (le != cudaSuccess || e != cudaSuccess) {
        if (gr) cudaGraphDestroy(gr);
        cudaGetLastError();
        return le != cudaSuccess ? le : e;
    }
    e = cudaGraphInstantiate(&f->graph, gr, 0);
    cudaGraphDestroy(gr);
    if (e != cudaSuccess) {
        f->graph = nullptr;
        cudaGetLastError();
    }
    return e;
}

}  // namespace

extern "C" int vefem_frontal_solve(vefem_frontal *f, const double *buf, const double *b, double *x,
                                   void *stream)
{
    if (!f || !buf || !b || !x) return VEFEM_ERR_ARG;
    DeviceGuard g(f->device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const unsigned pg = (unsigned)((f->N + 255) / 256);
    if (!f->graph || f->graph_buf != buf) {
        // capture the 2 x npan launches once per factor buffer: a replay costs a
        // fraction of their launch overhead.  Chained by programmatic dependent
        // launch where the driver accepts it, plain stream order otherwise.
        if (f->graph) {
            cudaGraphExecDestroy(f->graph);
            f->graph = nullptr;
        }
        cudaError_t e = f->pdl ? capture_sweeps(f, buf, true) : cudaErrorNotSupported;
        if (e != cudaSuccess) {
            f->pdl = false;
            e = capture_sweeps(f, buf, false);
        }
        if (e != cudaSuccess)
            return ffail(f, VEFEM_ERR_CUDA, std::string("solve graph: ") + cudaGetErrorString(e));
        f->graph_buf = buf;
    }
    k_to_elim<<<pg, 256, 0, s>>>(f->N, f->elim, b, f->wb);
    FCK(cudaGetLastError());
    FCK(cudaGraphLaunch(f->graph, s));
    k_from_elim<<<pg, 256, 0, s>>>(f->N, f->elim, f->wx, x);
    FCK(cudaGetLastError());
    f->last_path = f->pdl ? 1 : 2;
    return VEFEM_OK;
}

extern "C" int vefem_frontal_solve_path(const vefem_frontal *f)
{
    return f ? f->last_path : -1;
}

extern "C" void vefem_frontal_destroy(vefem_frontal *f)
{
    if (!f) return;
    {
        DeviceGuard g(f->device);
        if (f->graph) cudaGraphExecDestroy(f->graph);
        if (f->cs) cudaStreamDestroy(f->cs);
        cudaFree(f->wb);
        cudaFree(f->wy);
        cudaFree(f->wx);
        cudaFree(f->Tbuf[0]);
        cudaFree(f->Tbuf[1]);
        cudaFree(f->inv[0]);
        cudaFree(f->inv[1]);
        cudaFree(f->W);
        cudaFree(f->tickets);
        cudaFree(f->err);
        cudaFree(f->minpiv);
        cudaFree(f->elim);
        cudaFree(f->pidx);
    }
    delete f;
}

extern "C" const char *vefem_frontal_last_error(const vefem_frontal *f)
{
    return f ? f->msg.c_str() : "null frontal handle";
}
