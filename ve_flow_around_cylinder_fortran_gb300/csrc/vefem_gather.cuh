// AIJ entries from the element scratch (single-mesh and batched scatter).
//
// A thread owns two neighbouring entries of a 6 x 6 node-pair block.  What it
// needs to find them is one 32-byte record per block (BlockRec: row, offset and
// the first four contributors), so a value is two dependent loads away from
// the thread's index; list bounds, contributor ids and values looked up one
// after the other were three, and these kernels are bound by that chain at full
// occupancy, not by the bytes (0.85 GB per 40,000 FP32 elements, 0.13 ms).
// Kernel alone: FP32, 40,000 elements 588 -> 309 us; FP64, 5,000 elements 103 -> 93;
// 16 meshes of 1,000 to 10,000 in a batch 1,204 -> 687.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "vefem_internal.h"

namespace vefem {

constexpr int GB_THREADS = 288;   // 16 blocks
constexpr int GB_PAIRS = 18;      // pairs of a block

template <class T> struct Pair;
template <> struct Pair<float> { typedef float2 type; };
template <> struct Pair<double> { typedef double2 type; };

template <class T>
__device__ __forceinline__ void gather_pair(const GatherArgs &g, const int blk, const int pair,
                                            const T *__restrict__ es, T *__restrict__ vals)
{
    typedef typename Pair<T>::type V;
    const int4 *rp = reinterpret_cast<const int4 *>(g.brec + blk);
    const int4 head = rp[0], ids = rp[1];                 // row, off, c0, n; id[0..3]
    const int jeq = pair / 3, ieq = 2 * (pair - 3 * jeq), n = head.w;
    T *dst = vals + (g.rowptr[(int64_t)head.x * 6 + jeq] + head.y + ieq);
    const V *src = reinterpret_cast<const V *>(es) + pair;
    V v[ORDERED_PREFETCH];
    v[0] = n > 0 ? src[(int64_t)ids.x * GB_PAIRS] : V{};
    v[1] = n > 1 ? src[(int64_t)ids.y * GB_PAIRS] : V{};
    v[2] = n > 2 ? src[(int64_t)ids.z * GB_PAIRS] : V{};
    v[3] = n > 3 ? src[(int64_t)ids.w * GB_PAIRS] : V{};
    T x = g.store ? (T)0 : dst[0], y = g.store ? (T)0 : dst[1];
#pragma unroll
    for (int k = 0; k < ORDERED_PREFETCH; k++)
        if (k < n) {
            x = x + v[k].x;
            y = y + v[k].y;
        }
    for (int k = ORDERED_PREFETCH; k < n; k++) {
        const V w = src[(int64_t)g.bcon[head.z + k] * GB_PAIRS];
        x = x + w.x;
        y = y + w.y;
    }
    dst[0] = x;
    dst[1] = y;
}

// arclength column: the last entry of a node row (column N - 1)
template <class T>
__device__ __forceinline__ void gather_arclength(const GatherArgs &g, int node, int jeq, const T *__restrict__ as,
                                                 T *__restrict__ vals)
{
    const int64_t slot = g.rowptr[(int64_t)node * 6 + jeq + 1] - 1;
    const T acc0 = g.store ? (T)0 : vals[slot];
    vals[slot] = ordered_sum(acc0, g.ncon, g.nptr[node], g.nptr[node + 1],
                             [&](int c) { return as[(int64_t)c * 6 + jeq]; });
}

}  // namespace vefem
