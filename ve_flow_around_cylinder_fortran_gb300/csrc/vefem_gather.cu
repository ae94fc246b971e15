// Deterministic scatter of element contributions into the global residual and
// the AIJ values, in element order, without atomics.
//
// The reference adds element after element with VecSetValues/MatSetValues
// (ADD_VALUES, Storage_mod.F90:10-115), so a global entry is the sequential
// sum  ((v + c_e1) + c_e2) + ...  over the elements that touch it, in element
// order.  Here each global entry is owned by one thread, which reads the
// contributions from the element scratch through a precomputed contributor
// list sorted by element and adds them in that order: the same sum, bit for
// bit, with no colouring and no atomics.  These kernels are bandwidth-bound
// (the lists and the scratch are streamed once).
#include <cuda_runtime.h>
#include <stdint.h>

#include "vefem_gather.cuh"
#include "vefem_internal.h"

namespace vefem {

// b[gnode*6 + jeq] += sum over contributors (e*9 + jnod) of rs[(e*9+jnod)*6 + jeq]
__global__ void k_gather_residual(const GatherArgs g, const double *__restrict__ rs,
                                  double *__restrict__ b)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)g.nnodes * 6) return;
    const int node = (int)(t / 6), jeq = (int)(t - (int64_t)node * 6);
    const double acc0 = g.store ? 0.0 : b[t];
    b[t] = ordered_sum(acc0, g.ncon, g.nptr[node], g.nptr[node + 1],
                       [&](int c) { return rs[(int64_t)c * 6 + jeq]; });
}

// two entries of a node-pair block per thread, then (CTAs from nblk on) the
// arclength column (vefem_gather.cuh)
template <class T>
__global__ void __launch_bounds__(GB_THREADS)
k_gather_rows(const GatherArgs g, const T *__restrict__ es, const T *__restrict__ as, T *__restrict__ vals,
              unsigned nblk)
{
    if (blockIdx.x >= nblk) {
        const int64_t t = (int64_t)(blockIdx.x - nblk) * GB_THREADS + threadIdx.x;
        if (t < (int64_t)g.nnodes * 6) gather_arclength(g, (int)(t / 6), (int)(t % 6), as, vals);
        return;
    }
    const int64_t t = (int64_t)blockIdx.x * GB_THREADS + threadIdx.x;
    if (t >= (int64_t)g.nblocks * GB_PAIRS) return;
    const int blk = (int)(t / GB_PAIRS);
    gather_pair(g, blk, (int)(t - (int64_t)blk * GB_PAIRS), es, vals);
}

__global__ void k_block_records(int nblocks, const int32_t *__restrict__ brow, const int32_t *__restrict__ boff,
                                const int32_t *__restrict__ bptr, const int32_t *__restrict__ bcon,
                                BlockRec *__restrict__ rec)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nblocks) return;
    BlockRec r;
    r.row = brow[i];
    r.off = boff[i];
    r.c0 = bptr[i];
    r.n = bptr[i + 1] - r.c0;
#pragma unroll
    for (int k = 0; k < ORDERED_PREFETCH; k++) r.id[k] = k < r.n ? bcon[r.c0 + k] : 0;
    rec[i] = r;
}

cudaError_t launch_block_records(int nblocks, const int32_t *brow, const int32_t *boff, const int32_t *bptr,
                                 const int32_t *bcon, BlockRec *rec, cudaStream_t s)
{
    if (nblocks <= 0) return cudaSuccess;
    k_block_records<<<(nblocks + 255) / 256, 256, 0, s>>>(nblocks, brow, boff, bptr, bcon, rec);
    return cudaGetLastError();
}

// Dirichlet rows: b = TL - value, and the AIJ row zeroed with 1 on the diagonal
template <class V>
__global__ void k_dirichlet(int nrows, int nnodes, const int64_t *__restrict__ rows,
                            const double *__restrict__ values, const double *__restrict__ TL,
                            double *b, const int64_t *__restrict__ rowptr,
                            const int32_t *__restrict__ colind, V *vals)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nrows) return;
    const int64_t row = rows[r];
    if (row < 0 || row >= (int64_t)nnodes * 6) return;   // rows outside the node unknowns are ignored
    if (b) {
        const int64_t node = row / 6, eq = row - 6 * (row / 6);
        b[row] = TL[eq * nnodes + node] - values[r];
    }
    if (vals) {
        for (int64_t s = rowptr[row]; s < rowptr[row + 1]; s++)
            vals[s] = colind[s] == row ? (V)1 : (V)0;
    }
}

cudaError_t launch_dirichlet(int nrows, int nnodes, const int64_t *rows, const double *values,
                             const double *TL, double *b, const int64_t *rowptr,
                             const int32_t *colind, void *vals, int vals_float, cudaStream_t s)
{
    if (nrows <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)((nrows + 127) / 128);
    if (vals_float)
        k_dirichlet<float><<<grid, 128, 0, s>>>(nrows, nnodes, rows, values, TL, b, rowptr, colind,
                                                 static_cast<float *>(vals));
    else
        k_dirichlet<double><<<grid, 128, 0, s>>>(nrows, nnodes, rows, values, TL, b, rowptr,
                                                  colind, static_cast<double *>(vals));
    return cudaGetLastError();
}

static inline unsigned grid_for(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

cudaError_t launch_gather_residual(const GatherArgs &g, const double *rs, double *b,
                                   cudaStream_t s)
{
    const int64_t n = (int64_t)g.nnodes * 6;
    if (n == 0) return cudaSuccess;
    k_gather_residual<<<grid_for(n, 256), 256, 0, s>>>(g, rs, b);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_gather_rows(const GatherArgs &g, const T *es, const T *as, T *vals, cudaStream_t s)
{
    const unsigned nblk = grid_for((int64_t)g.nblocks * GB_PAIRS, GB_THREADS);
    const unsigned narc = g.nex > 0 ? grid_for((int64_t)g.nnodes * 6, GB_THREADS) : 0;
    if (nblk + narc > 0) k_gather_rows<T><<<nblk + narc, GB_THREADS, 0, s>>>(g, es, as, vals, nblk);
    return cudaGetLastError();
}

template cudaError_t launch_gather_rows<double>(const GatherArgs &, const double *, const double *, double *,
                                                cudaStream_t);
template cudaError_t launch_gather_rows<float>(const GatherArgs &, const float *, const float *, float *, cudaStream_t);

}  // namespace vefem
