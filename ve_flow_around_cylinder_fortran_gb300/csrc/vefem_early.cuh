// Loads of a programmatically launched kernel before its own
// griddepcontrol.wait, of data that a kernel or copy before its predecessor wrote.
//
// What such a load relies on.  The predecessor has itself waited for all that
// came before: it was launched in plain stream order, or its threads pass their
// own wait before they let this kernel start.  Then those grids have completed
// and their writes are performed and visible to a grid whose blocks may run on
// any SM, that is, in L2.  What the programming model grants before the own wait
// is no more than that: an older copy in this SM's L1 or on its read-only path
// (where const __restrict__ sends a plain load) need not be gone.  A relaxed load
// at GPU scope is answered by neither.  Data that the predecessor itself writes
// is read after the wait only.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

__device__ __forceinline__ double load_early(const double *p)
{
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ __nv_bfloat16 load_early(const __nv_bfloat16 *p)
{
    unsigned short v;
    asm volatile("ld.relaxed.gpu.global.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
    return __ushort_as_bfloat16(v);
}
